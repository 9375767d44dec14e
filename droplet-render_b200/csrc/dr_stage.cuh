// Device helpers shared by the kernels: staging of the phase tables in shared
// memory, counter sums and small vector helpers.
#pragma once
#include "dr_device.cuh"

namespace dr {

// ---- shared-memory staging of the phase tables ------------------------------
// Layout in global and shared memory: pdf as float4 (r, g, b, 0) x n, then the
// red CDF x n (n % 4 == 0, so the block is a multiple of 16 bytes).  One thread
// issues a bulk copy (cp.async.bulk, completion counted on an mbarrier); the
// wait is bounded and reports a give-up instead of spinning forever.
// Exact mode appends its sampler table: (2n + 1) float4 after the CDF.
__device__ __forceinline__ uint32_t mie_bytes(const DevParams &P) {
    return P.mie_n * 20u + (P.phase_mode == 1u ? (2u * P.mie_n + 1u) * 16u : 0u);
}

__device__ __forceinline__ MieSmem mie_view(const DevParams &P, unsigned char *smem) {
    return MieSmem{reinterpret_cast<float4 *>(smem), reinterpret_cast<float *>(smem + 16u * P.mie_n), P.mie_n,
                   P.phase_mode == 1u ? reinterpret_cast<const float4 *>(smem + 20u * P.mie_n) : nullptr};
}

__device__ __forceinline__ bool stage_mie(const void *src, uint32_t bytes, unsigned char *smem, uint64_t *mbar) {
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(mbar);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
            "l"(src), "r"(bytes), "r"(bar)
            : "memory");
    }
    uint32_t done = 0;
    for (uint32_t it = 0; it < (1u << 22) && !done; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar)
            : "memory");
    }
    return done != 0;
}

__device__ __forceinline__ void warp_sum_counts(Count &c, DevCounters *C, uint32_t paths) {
    const uint32_t full = 0xffffffffu;
    uint32_t v = __reduce_add_sync(full, c.vertices);
    uint32_t nv = __reduce_add_sync(full, c.node_visits);
    uint32_t dl = __reduce_add_sync(full, c.density_lookups);
    uint32_t me = __reduce_add_sync(full, c.mie_evals);
    uint32_t gu = __reduce_add_sync(full, c.gave_up);
    uint32_t pa = __reduce_add_sync(full, paths);
    if ((threadIdx.x & 31) == 0 && (v | nv | dl | me | gu | pa)) {  // an idle warp adds nothing
        atomicAdd(&C->vertices, (unsigned long long)v);
        atomicAdd(&C->node_visits, (unsigned long long)nv);
        atomicAdd(&C->density_lookups, (unsigned long long)dl);
        atomicAdd(&C->mie_evals, (unsigned long long)me);
        if (gu) atomicAdd(&C->gave_up, (unsigned long long)gu);
        atomicAdd(&C->paths, (unsigned long long)pa);
    }
}

__device__ __forceinline__ float4 shfl_xor4(float4 v, int m) {
    v.x = __shfl_xor_sync(0xffffffffu, v.x, m);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, m);
    v.z = __shfl_xor_sync(0xffffffffu, v.z, m);
    v.w = __shfl_xor_sync(0xffffffffu, v.w, m);
    return v;
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

}  // namespace dr
