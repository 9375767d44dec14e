// Lets the host compiler take the device headers: the intrinsics they use, as
// plain C++.  Include before dr_device.cuh.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>
#undef __device__
#undef __host__
#undef __forceinline__
#undef __noinline__
#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__
template <class T> inline T __ldg(const T *p) { return *p; }
inline uint32_t __popc(uint32_t x) { return (uint32_t)__builtin_popcount(x); }
inline int __ffs(int x) { return __builtin_ffs(x); }
inline uint32_t __float_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
inline float __uint_as_float(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
inline float __int_as_float(int u) { return __uint_as_float((uint32_t)u); }
inline uint32_t __umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    s &= 31u;
    return s ? (lo >> s) | (hi << (32u - s)) : lo;
}
inline float __fdiv_rn(float a, float b) { return a / b; }
inline unsigned long long atomicAdd(unsigned long long *p, unsigned long long v) { *p += v; return *p - v; }
using std::isfinite;
using std::max;
using std::min;
