// The path pipeline: three kernels that render a tile (or every view of a
// batch) whose octree has a block grid (DevScene::gblock).
//
//   camera lists   one thread per pixel traverses the camera ray once and
//                  records its leaves; pixels whose ray meets no leaf are counted
//                  and finished here, the others go to a list of active pixels
//   camera paths   the camera segments of the active pixels' samples, 32 samples
//                  of a pixel side by side: a warp's lanes read the same leaf list
//                  and run the same steps.  The samples that collide become records
//   scatter        everything after a path's first collision, from the records
//
// Splitting the paths there is what the hardware asks for: a path is mostly a
// camera segment that hits nothing (of the 512^3 cumulus frame's 133 M samples
// 119 M meet no leaf at all and about 5 M collide), those are coherent, and the
// rest is not.  One kernel for all three (render_persistent_kernel, which
// serves the octrees without a block grid) was bound by instruction issue at 8
// of 32 lanes per instruction: 39.4 ms for that frame at 64 samples, 63.4 ms for a
// 1024^3 sparse slab at 1920 x 1080 x 256.  The pipeline takes 17.6 and 24.9 ms, the
// scatter kernel at 12.5 lanes per instruction.  (Times here are those of the timing
// cases in perf/cases.py, single passes by CUDA events, the mean of three seeds; the
// camera and the noise differ by seed, and with them these frames by up to 9%.  The benchmark's
// frame, another camera again, takes 16.2 ms: lists 0.21, camera 2.34, scatter 13.7.)
//
// Per path, the operations and random draws are those of path_sample(): a
// path's result does not depend on the kernel that computed it.
#include <cuda_runtime.h>
#include "dr_kernels.h"
#include "dr_stage.cuh"

namespace dr {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kTicketMost = 128;  // camera samples per ticket (W.ticket: 128 or, in small launches, 32)
constexpr int kListBlock = 128, kListTx = 16, kListTy = 8;  // camera lists: a block covers 16 x 8 pixels

// ---- camera lists -------------------------------------------------------------
// Leaf list of one camera ray: the ray's traversal run to its end, as every
// sample of the pixel would run it.  The leaves are counted first, then a
// contiguous range of the pool is taken and filled by a second traversal; a
// pixel whose range does not fit gets x = ~0 and its samples traverse.
// Rays with a zero direction component take the octree (node ids become slots).
__device__ __noinline__ uint4 octree_list(const DevScene &S, float ox, float oy, float oz, float dx, float dy, float dz,
                                          uint4 *pool, uint32_t cap, unsigned long long *used) {
    const float ro[3] = {ox, oy, oz}, rd[3] = {dx, dy, dz};
    const SlotStack stk{S};
    Trav T;
    Count c;
    c.zero();
    trav_init(T, S, ro, rd, c);
    uint4 h = make_uint4(0u, 0u, c.node_visits, 0u);
    uint32_t leaf, n = 0;
    float tra, trb;
    while (trav_next_s(T, S, stk, leaf, tra, trb, c, kNone) == kTravLeaf) ++n;
    const uint32_t off = n ? pool_range(used, n, cap) : 0u;
    h.x = off;
    if (off == kNone) return h;
    h.y = n;
    trav_init(T, S, ro, rd, c);
    c.zero();
    for (uint32_t k = 0; k < n; ++k) {
        trav_next_s(T, S, stk, leaf, tra, trb, c, kNone);
        pool[off + k] = make_uint4(__float_as_uint(__ldg(&S.leaf[2 * leaf + 1]).w), __float_as_uint(tra),
                                   __float_as_uint(trb), c.node_visits);
        c.zero();
    }
    trav_next_s(T, S, stk, leaf, tra, trb, c, kNone);  // kTravDone
    h.w = c.node_visits;
    return h;
}

// The whole warp calls (ray: the lane has one); its lanes share one addition to the counter.
__device__ __forceinline__ uint4 grid_list(const DevScene &S, bool ray, const float ro[3], const float rd[3], float *col,
                                           uint4 *pool, uint32_t cap, unsigned long long *used) {
    GridTrav G;
    Count c;
    c.zero();
    const uint32_t mode = ray ? grid_init<kListBlock>(G, S, col, ro, rd, c) : 0u;
    uint32_t leaf, n = 0;
    float tra, trb;
    if (mode == 1u)
        while (grid_next<kListBlock>(G, S, col, ro, rd, leaf, tra, trb, c, kNone) == kTravLeaf) ++n;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t end = n;  // of the lane's entries among the warp's
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t o = __shfl_up_sync(kFull, end, d);
        if (lane >= d) end += o;
    }
    unsigned long long first = 0;
    if (lane == 31u && end) first = atomicAdd(used, (unsigned long long)end);
    first = __shfl_sync(kFull, first, 31) + (end - n);
    if (mode == 2u) return octree_list(S, ro[0], ro[1], ro[2], rd[0], rd[1], rd[2], pool, cap, used);
    if (mode == 0u) return make_uint4(0u, 0u, 0u, 0u);
    if (n == 0) return make_uint4(0u, 0u, 1u, c.node_visits - 1u);
    const uint32_t off = pool_place(first, n, cap);
    if (off == kNone) return make_uint4(kNone, 0u, 0u, 0u);
    c.zero();
    grid_init<kListBlock>(G, S, col, ro, rd, c);
    c.node_visits -= 1u;  // the root (h.z)
    for (uint32_t k = 0; k < n; ++k) {
        grid_next<kListBlock>(G, S, col, ro, rd, leaf, tra, trb, c, kNone);
        pool[off + k] = make_uint4(leaf, __float_as_uint(tra), __float_as_uint(trb), c.node_visits);
        c.zero();
    }
    grid_next<kListBlock>(G, S, col, ro, rd, leaf, tra, trb, c, kNone);  // kTravDone
    return make_uint4(off, n, 1u, c.node_visits);
}

// Pixel (ix, iy) of a tile (valid lanes): its header, and its place among the
// active pixels or, without a leaf, its samples' counters.
__device__ __forceinline__ void list_pixel(const DevScene &S, const DevParams &P, const TileArgs &A, uint32_t ix,
                                           uint32_t iy, bool valid, float *col, uint4 *head, const PathWork &W,
                                           uint32_t *active, unsigned int *n_active, DevCounters *C) {
    uint4 h = make_uint4(0u, 0u, 0u, 0u);
    bool ray = false;
    const uint32_t pix = iy * A.cols + ix;
    float ro[3], rd[3];
    if (valid) ray = camera_ray(P, A.x0 + ix, A.y0 + iy, ro, rd);
    h = grid_list(S, ray, ro, rd, col, W.pool, W.pool_cap, W.pool_used);
    if (valid) {
        head[2 * (size_t)pix] = h;
        head[2 * (size_t)pix + 1] =
            make_uint4(__float_as_uint(rd[0]), __float_as_uint(rd[1]), __float_as_uint(rd[2]), ray ? 1u : 0u);
    }
    const uint32_t lane = threadIdx.x & 31u;
    const bool act = ray && (h.y > 0u || h.x == kNone);
    const uint32_t am = __ballot_sync(kFull, act), em = __ballot_sync(kFull, ray && !act);
    uint32_t at = 0;
    if (lane == 0 && am) at = atomicAdd(n_active, (unsigned int)__popc(am));
    at = __shfl_sync(kFull, at, 0);
    if (act) active[at + __popc(am & ((1u << lane) - 1u))] = pix;
    if (em && C) {  // (the adjoint does not count)
        const uint32_t v = __reduce_add_sync(kFull, (ray && !act) ? h.z + h.w : 0u);
        if (lane == 0) {
            const unsigned long long n = (unsigned long long)__popc(em) * A.spp;
            atomicAdd(&C->paths, n);
            atomicAdd(&C->vertices, n);
            atomicAdd(&C->node_visits, (unsigned long long)v * A.spp);
        }
    }
}

__global__ void __launch_bounds__(kListBlock) path_lists_kernel(const __grid_constant__ DevScene S,
                                                                const __grid_constant__ DevParams P,
                                                                const __grid_constant__ TileArgs A,
                                                                const __grid_constant__ PathWork W, DevCounters *C) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *const col = reinterpret_cast<float *>(smem) + threadIdx.x;
    const uint32_t bx = (A.cols + kListTx - 1) / kListTx, by = blockIdx.x / bx;
    const uint32_t ix = (blockIdx.x - by * bx) * kListTx + (threadIdx.x & (kListTx - 1));
    const uint32_t iy = by * kListTy + threadIdx.x / kListTx;
    list_pixel(S, P, A, ix, iy, ix < A.cols && iy < A.rows, col, W.head, W, W.active, W.n_active, C);
}

// The lists of every view of a batch: view v owns the blocks from
// block_begins[v] on, its pixels' headers start at its TileArgs::cam_head and its
// active pixels at active + pix_begins[v].
__device__ __forceinline__ uint32_t find_last(const uint32_t *begins, uint32_t n, uint32_t t) {
    uint32_t lo = 0, hi = n - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(&begins[mid]) <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(kListBlock) path_lists_batch_kernel(BatchArgs B, PathWork W, DevCounters *C) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *const col = reinterpret_cast<float *>(smem) + threadIdx.x;
    const uint32_t v = find_last(W.block_begins, B.n_views, blockIdx.x), blk = blockIdx.x - __ldg(&W.block_begins[v]);
    const BatchView &V = B.views[v];
    const uint32_t bx = (V.A.cols + kListTx - 1) / kListTx, by = blk / bx;
    const uint32_t ix = (blk - by * bx) * kListTx + (threadIdx.x & (kListTx - 1));
    const uint32_t iy = by * kListTy + threadIdx.x / kListTx;
    list_pixel(B.scenes[V.scene], V.P, V.A, ix, iy, ix < V.A.cols && iy < V.A.rows, col,
               const_cast<uint4 *>(V.A.cam_head), W, W.active + W.pix_begins[v], &W.view_active[v], C);
}

// First ticket of every view (and the number of tickets) from its active pixels: one warp.
__global__ void view_tickets_kernel(BatchArgs B, PathWork W) {
    const uint32_t lane = threadIdx.x;
    uint32_t run = 0;
    for (uint32_t v0 = 0; v0 < B.n_views; v0 += 32) {
        const uint32_t v = v0 + lane;
        uint32_t n = 0;
        if (v < B.n_views) n = (uint32_t)(((uint64_t)W.view_active[v] * B.views[v].A.spp + W.ticket - 1) / W.ticket);
        uint32_t sum = n;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(kFull, sum, d);
            if (lane >= (uint32_t)d) sum += o;
        }
        if (v < B.n_views) W.view_tickets[v] = run + sum - n;
        run += __shfl_sync(kFull, sum, 31);
    }
    if (lane == 0) W.view_tickets[B.n_views] = run;
}

// ---- free flight in a leaf ---------------------------------------------------------
// The adjoint's tape, as a warp writes it: space is taken 256 entries at a time
// (an entry at a time would be one atomic addition per pass of full flights on a
// single address); what a warp leaves unused is marked.  Nothing without the
// adjoint.  A path whose entries do not fit, with more than 64 shadow segments, or
// with a segment slow_segment traces is marked in its record and replayed.
// Tracing twice and scattering from the second trace was bound by the octree walk
// and one scalar atomic per brick sample: a 256 x 256 view at 32 samples of a 128^3
// cloud took 3.2 + 6.5 ms.  With the tape: 2.9 ms here, 0.16 ms in
// tape_scatter_kernel, 0.03 ms looking for paths to replay (an inverse step of
// eight views 95 -> 46 ms).
struct NoTape {
    static constexpr bool on = false;
};

struct Tape {
    static constexpr bool on = true;
    const AdjointArgs &J;
    uint32_t at, left;
    bool full;
    // the lane's decision, filled by leaf_flight
    bool has;
    uint32_t idx, corner;
    float d, nl[3];
    __device__ __forceinline__ void mark(uint32_t lane) {  // the unused rest of the space
        for (uint32_t i = lane; i < left; i += 32) J.tape[2 * (size_t)(at + i)].x = kNone;
        left = 0;
    }
    // All lanes: the lanes with a decision append it.  flags: see AdjointArgs.
    __device__ __forceinline__ void put(uint32_t path, uint32_t flags, float value, uint32_t lane) {
        const uint32_t m = __ballot_sync(kFull, has);
        if (!m) return;
        const uint32_t n = __popc(m);
        if (n > left && !full) {
            mark(lane);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(J.tape_used, 256u);
            base = __shfl_sync(kFull, base, 0);
            if (base <= J.tape_cap && J.tape_cap - base >= 256u) {
                at = base;
                left = 256u;
            } else {
                // no room: what was handed out but does not fit in whole is marked
                full = true;
                for (uint32_t i = base + lane; i < J.tape_cap && i - base < 256u; i += 32)
                    J.tape[2 * (size_t)i].x = kNone;
            }
        }
        if (n > left) {  // the tape is full: the paths are replayed
            if (has) J.rec[path].pad = kReplay;
        } else if (has) {
            uint4 *const t = J.tape + 2 * (size_t)(at + __popc(m & ((1u << lane) - 1u)));
            t[0] = make_uint4(path, idx, flags | corner, __float_as_uint(d));
            t[1] = make_uint4(__float_as_uint(nl[0]), __float_as_uint(nl[1]), __float_as_uint(nl[2]), __float_as_uint(value));
        }
        if (n <= left) {
            at += n;
            left -= n;
        }
        has = false;
    }
};

template <bool ADJ> __device__ __forceinline__ auto make_tape(const AdjointArgs &J) {
    if constexpr (ADJ) return Tape{J, 0u, 0u, false, false, 0u, 0u, 0.0f, {0.0f, 0.0f, 0.0f}};
    else return NoTape{};
}

// A flight leaves_at_once does not decide, in full (src/kernel.cpp:241-317): a flight in leaf `slot`
// with interval [tra, trb], entered at distance lo.  first: v is the uniform
// draw of the first flight, else the distance flown so far in the leaf.
// kLeft: the leaf is left; kReal: a real collision at td; kNull: a null one (v
// is the distance flown, call again).
enum : uint32_t { kLeft = 0, kReal = 1, kNull = 2 };
template <uint32_t FEAT, class TP>
__device__ __forceinline__ uint32_t leaf_flight(TP &tape, const DevScene &S, float sigma_e, const float ro[3], const float rd[3],
                                                uint32_t slot, float tra, float trb, float lo, bool first, float &v,
                                                float &td, Rng &g, Count &cnt) {
    const float4 meta = __ldg(&S.gleaf[2 * slot + 1]), ce = __ldg(&S.gleaf[2 * slot]);
    const float denom = sigma_e * meta.x;
    const float tr0 = tra - lo, tr1 = trb - lo;
    float s0 = tra > lo ? tr0 : __uint_as_float(__float_as_uint(tr0) & 1u);
    const float *sdf = nullptr;
    if constexpr ((FEAT & kFeatSdf) != 0) {
        const uint32_t sdfx = __float_as_uint(meta.z);
        if (sdfx != kNone) {
            sdf = S.sdf_bricks + (size_t)sdfx * kBrick;
            s0 = 0.0f;
            if (tra > lo) {  // src/kernel.cpp:253-263
                const float r0[3] = {ro[0] + rd[0] * tra, ro[1] + rd[1] * tra, ro[2] + rd[2] * tra};
                if (sample_voxel_space(r0, sdf, ce) > 0.0f) s0 = tr0;
                if (first) ++cnt.density_lookups;
            }
        }
    }
    const float u = first ? v : g.uniform();
    const float sr = (first ? 0.0f : v) - dlog_unit(u) / denom;
    v = sr;
    const float sc = s0 + sr;
    td = lo + sc;
    if (!(sc < tr1)) {
        td = trb;
        return kLeft;
    }
    bool rm = sc > tr0;
    float rho = -1.0f, dist = 1.0f;
    if (rm) {
        const float rc[3] = {ro[0] + rd[0] * td, ro[1] + rd[1] * td, ro[2] + rd[2] * td};
        const uint32_t fog = __float_as_uint(meta.y);
        bool look = true;
        if constexpr ((FEAT & kFeatSdf) != 0) {
            if (sdf) {  // src/kernel.cpp:287-300: inside the surface always collides
                dist = sample_voxel_space(rc, sdf, ce);
                ++cnt.density_lookups;
                look = dist > 0.0f && fog != kNone;
            }
        }
        if (look) {
            rho = sample_voxel_inv(rc, S.bricks + (size_t)fog * kBrick, ce, S.ginv);
            ++cnt.density_lookups;
        }
    }
    const float q = g.uniform();
    const bool null = rm && ratio_below(rho, meta.x, q) && (dist > 0.0f);
    if constexpr (TP::on) {  // what the fog density decided
        const uint32_t fog = __float_as_uint(meta.y);
        const float d = null ? meta.x - rho : rho;
        if (rm && fog != kNone && dist > 0.0f && d > 0.0f) {
            const float4 ce = __ldg(&S.gleaf[2 * slot]);
            const float rc[3] = {ro[0] + rd[0] * td, ro[1] + rd[1] * td, ro[2] + rd[2] * td};
            uint32_t ia[3], ib[3];
            if (!voxel_cell_inv(rc, ce, S.ginv, ia, ib, tape.nl)) voxel_cell(rc, ce, ia, ib, tape.nl);
            tape.has = true;
            tape.idx = fog * kBrick + ia[2] * 64u + ia[1] * 8u + ia[0];
            tape.corner = (ib[0] - ia[0]) | (ib[1] - ia[1]) << 1 | (ib[2] - ia[2]) << 2;
            tape.d = null ? 0.0f - d : d;
        }
    }
    return null ? kNull : kReal;
}

// Whether a leaf may be passed by leaves_at_once: not with a surface brick
// (its flight starts where the distance at the entry says).
template <uint32_t FEAT>
__device__ __forceinline__ bool fog_only(const DevScene &S, uint32_t slot) {
    if constexpr ((FEAT & kFeatSdf) != 0) return __float_as_uint(__ldg(&S.gleaf[2 * slot + 1]).z) == kNone;
    else return true;
}

// ---- camera paths ---------------------------------------------------------------
// A lane walks a sample's camera segment: it enters its next leaf and draws the
// first flight (kWalk), or waits with a flight to be computed in full (kHard,
// kHardAgain; these run when enough lanes wait, or all), or is done (kOut).
enum : uint32_t { kWalk = 0, kHard = 1, kHardAgain = 2, kOut = 3 };
constexpr uint32_t kHardBatch = 8;

struct SlowSeg {
    uint32_t res, visits, lookups, gave_up;
    float td;
    uint64_t state;
};
// A segment with a zero direction component, traced through the octree.
template <uint32_t FEAT>
__device__ __noinline__ SlowSeg slow_segment(const DevScene &S, SegMedium med, float ox, float oy, float oz, float dx,
                                             float dy, float dz, float depth, uint64_t state, uint64_t inc) {
    const float ro[3] = {ox, oy, oz}, rd[3] = {dx, dy, dz};
    const NoVisit nv;
    Count c;
    c.zero();
    Rng g;
    g.state = state;
    g.inc = inc;
    SlowSeg o;
    o.res = track_on<NoVisit, (FEAT & kFeatSdf) != 0>(S, med, ro, rd, g, depth, o.td, SlotStack{S}, c, nv);
    o.visits = c.node_visits;
    o.lookups = c.density_lookups;
    o.gave_up = c.gave_up;
    o.state = g.state;
    return o;
}

struct CamSeg {
    uint32_t res;
    float td;
    Rng g;
};

// Camera segments of a warp's 32 samples (alive lanes).  LISTED: along the
// pixel's leaf list h; else by traversing.
template <uint32_t FEAT, bool LISTED, class TP>
__device__ __forceinline__ CamSeg camera_segments(TP &tape, uint32_t path, const DevScene &S, SegMedium med, bool alive, const float ro[3],
                                                  const float rd[3], Rng g, float depth, uint4 h, const uint4 *pool,
                                                  float *col, Count &cnt) {
    uint32_t k = h.x, left = h.y, budget = med.budget, slot = 0;
    float td = 0.0f, lo = 0.0f, v = 0.0f, tra = 0.0f, trb = 0.0f;
    CamSeg o;
    o.res = kTrackEscaped;
    GridTrav G;
    uint32_t st = alive ? kWalk : kOut;
    if (alive) {
        if constexpr (LISTED) {
            cnt.node_visits += h.z;
        } else {
            const uint32_t m = grid_init<kListBlock>(G, S, col, ro, rd, cnt);
            if (m == 0u) st = kOut;
            if (m == 2u) {  // a zero direction component
                const SlowSeg q = slow_segment<FEAT>(S, med, ro[0], ro[1], ro[2], rd[0], rd[1], rd[2], depth, g.state,
                                                     g.inc);
                cnt.node_visits += q.visits;
                cnt.density_lookups += q.lookups;
                cnt.gave_up += q.gave_up;
                o.res = q.res;
                td = q.td;
                g.state = q.state;
                st = kOut;
                if constexpr (TP::on) tape.J.rec[path].pad = kReplay;  // its decisions are not on the tape
            }
        }
    }
    for (;;) {
        if (st == kWalk) {
            uint32_t r;
            if constexpr (LISTED) {
                if (left) {
                    const uint4 e = __ldg(&pool[k]);
                    ++k;
                    --left;
                    slot = e.x;
                    tra = __uint_as_float(e.y);
                    trb = __uint_as_float(e.z);
                    cnt.node_visits += e.w;
                    r = kTravLeaf;
                } else {
                    cnt.node_visits += h.w;
                    r = kTravDone;
                }
            } else {
                r = grid_next<kListBlock>(G, S, col, ro, rd, slot, tra, trb, cnt, 1u);
            }
            if (r == kTravDone || (r == kTravLeaf && !(td < depth))) {
                st = kOut;
            } else if (r == kTravLeaf) {
                const float denom = med.sigma_e * __ldg(&S.gmaj[slot]);
                v = g.uniform();
                if (leaves_at_once(v, denom, tra, trb, td) && fog_only<FEAT>(S, slot)) {
                    td = trb;
                } else {
                    lo = td;
                    st = kHard;
                }
            }
        }
        const bool hard = st == kHard || st == kHardAgain;
        const uint32_t nl = __ballot_sync(kFull, hard), nb = __ballot_sync(kFull, st == kWalk);
        if (!(nl | nb)) break;
        const bool pass = nl && ((uint32_t)__popc(nl) >= kHardBatch || !nb);
        if (pass && hard) {
            const uint32_t r = leaf_flight<FEAT>(tape, S, med.sigma_e, ro, rd, slot, tra, trb, lo, st == kHard, v, td, g, cnt);
            st = r == kLeft ? kWalk : kHardAgain;
            if (r == kReal) {
                o.res = td < depth ? kTrackCollided : kTrackCut;
                st = kOut;
            } else if (r == kNull && --budget == 0) {
                ++cnt.gave_up;
                st = kOut;
            }
        }
        if constexpr (TP::on) {
            if (pass) tape.put(path, 0u, 0.0f, threadIdx.x & 31u);
        }
    }
    o.td = td;
    o.g = g;
    return o;
}

// Sample q of a tile's active pixels: pixel and sample number.
__device__ __forceinline__ void active_sample(const TileArgs &A, const uint32_t *active, uint64_t q, uint32_t &pix,
                                              uint32_t &s) {
    uint32_t a;
    if (q <= 0xffffffffull) {
        a = fastdiv((uint32_t)q, A.spp_div);
        s = (uint32_t)q - a * A.spp;
    } else {
        const uint64_t l = q / A.spp;
        a = (uint32_t)l;
        s = (uint32_t)(q - l * A.spp);
    }
    pix = __ldg(&active[a]);
}

// Camera samples are handed out in tickets of W.ticket consecutive ones.  A warp
// takes a ticket only while the record buffer has room for every warp's
// (W.limit = capacity - warps * W.ticket), so the buffer never overflows and the
// tickets taken are exactly those done: the next round goes on from there.
// ADJ: the adjoint's first pass (the samples of pixels without a gradient are
// left out, nothing is counted or added to an image).  8 blocks per SM: 5 to 8 are
// within 1% of each other (512^3 frame 17.65 ms, with 5 or 6 17.80; slab 24.9 and 25.1).
template <uint32_t FEAT, bool BATCH, bool ADJ>
__global__ void __launch_bounds__(kListBlock, ADJ ? 6 : 8) camera_paths_kernel(const __grid_constant__ DevScene S0,
                                                                     const __grid_constant__ DevParams P0,
                                                                     const __grid_constant__ TileArgs A0,
                                                                     const __grid_constant__ PathWork W,
                                                                     float4 *sun0, float4 *sky0, DevCounters *C,
                                                                     BatchArgs B,
                                                                     const __grid_constant__ AdjointArgs J) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *const col = reinterpret_cast<float *>(smem) + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    Count cnt;
    cnt.zero();
    auto tape = make_tape<ADJ>(J);
    uint32_t paths = 0;
    uint64_t total = 0;
    uint64_t n_tickets;  // (a tile may have 2^32 and more)
    const uint64_t step = B.step ? *B.step : 0ull;
    if constexpr (BATCH) {
        n_tickets = W.view_tickets[B.n_views];
    } else {
        total = (uint64_t)*W.n_active * A0.spp;
        n_tickets = (total + W.ticket - 1) / W.ticket;
    }
    const unsigned long long base = W.ctl->base;
    for (;;) {
        unsigned long long t = ~0ull;
        if (lane == 0) {
            const uint32_t rec = *(volatile uint32_t *)&W.ctl->records;
            const unsigned long long tk = *(volatile unsigned long long *)&W.ctl->ticket;
            if (rec <= W.limit && tk < n_tickets && tk - base < kRoundTickets) t = atomicAdd(&W.ctl->ticket, 1ull);
        }
        t = __shfl_sync(kFull, t, 0);
        if (t >= n_tickets) break;
        uint32_t view = 0;
        uint64_t q0 = t * W.ticket;
        if constexpr (BATCH) {
            view = find_last(W.view_tickets, B.n_views, (uint32_t)t);
            q0 = (t - W.view_tickets[view]) * W.ticket;
            total = (uint64_t)W.view_active[view] * B.views[view].A.spp;
        }
        const BatchView *V = BATCH ? &B.views[view] : nullptr;
        const TileArgs &A = BATCH ? V->A : A0;
        const DevParams &P = BATCH ? V->P : P0;
        const DevScene &S = BATCH ? B.scenes[V->scene] : S0;
        const uint4 *head = BATCH ? A.cam_head : W.head;
        const uint32_t *active = BATCH ? W.active + W.pix_begins[view] : W.active;
        for (uint32_t c = 0; c < W.ticket; c += 32u) {
            const uint64_t q = q0 + c + lane;
            if (q - lane >= total) break;
            bool valid = q < total;
            uint32_t pix = kNone, s = 0;
            uint4 h = make_uint4(0u, 0u, 0u, 0u);
            float ro[3], rd[3] = {0.0f, 0.0f, 0.0f};
            for (int k = 0; k < 3; ++k) ro[k] = P.viewi[12 + k];
            float depth = 3.402823466e+38f;
            Rng g;
            g.state = g.inc = 0;
            if (valid) {
                active_sample(A, active, q, pix, s);
                h = __ldg(&head[2 * (size_t)pix]);
                const uint4 ray = __ldg(&head[2 * (size_t)pix + 1]);
                rd[0] = __uint_as_float(ray.x);
                rd[1] = __uint_as_float(ray.y);
                rd[2] = __uint_as_float(ray.z);
                const uint32_t iy = fastdiv(pix, A.cols_div), ix = pix - iy * A.cols;
                const uint64_t fp = (uint64_t)(A.y0 + iy) * P.w + (A.x0 + ix);
                if (P.depth && P.depthcomp) depth = __ldg(&P.depth[fp]);
                g = rng_seed(A.seed, fp, A.sample_base + step * A.spp + s);
                ++paths;
                ++cnt.vertices;
                if constexpr (ADJ) {
                    const size_t off = (size_t)iy * A.tw + ix;
                    const float4 ds = __ldg(&J.dsun[off]), dk = __ldg(&J.dsky[off]);
                    valid = (ds.x * ds.x + ds.y * ds.y + ds.z * ds.z) + (dk.x * dk.x + dk.y * dk.y + dk.z * dk.z) > 0.0f;
                }
            }
            const uint32_t path = ADJ ? pix * A.spp + s : 0u;
            CamSeg o;
            if (!__any_sync(kFull, valid && h.x == kNone))
                o = camera_segments<FEAT, true>(tape, path, S, seg_medium(P), valid, ro, rd, g, depth, h, W.pool, col, cnt);
            else  // a pixel whose list did not fit: the whole group traverses
                o = camera_segments<FEAT, false>(tape, path, S, seg_medium(P), valid, ro, rd, g, depth, h, W.pool, col, cnt);
            // alpha of the pixel's samples that collided (or were cut at the depth, src/kernel.cpp:370-384)
            const bool hit = !ADJ && valid && first_alpha(P, o.res) != 0.0f;
            const uint32_t hm = __ballot_sync(kFull, hit);
            if (hit) {
                const uint32_t same = __match_any_sync(hm, pix);
                if (lane == (uint32_t)__ffs((int)same) - 1u) {
                    const uint32_t iy = fastdiv(pix, A.cols_div);
                    const size_t off = (size_t)iy * A.tw + (pix - iy * A.cols);
                    const float a = (float)__popc(same);
                    atomicAdd(&(BATCH ? V->sun : sun0)[off].w, a);
                    atomicAdd(&(BATCH ? V->sky : sky0)[off].w, a);
                }
            }
            const bool go = valid && o.res == kTrackCollided && P.scattevs > 0u;
            const uint32_t gm = __ballot_sync(kFull, go);
            if (gm) {
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&W.ctl->records, (uint32_t)__popc(gm));
                at = __shfl_sync(kFull, at, 0) + __popc(gm & ((1u << lane) - 1u));
                if (go)
                    W.records[at] = make_uint4((uint32_t)o.g.state, (uint32_t)(o.g.state >> 32), __float_as_uint(o.td),
                                               (uint32_t)(t * W.ticket + c + lane));
            }
        }
    }
    if constexpr (ADJ) tape.mark(lane);
    else warp_sum_counts(cnt, C, paths);
}

// ---- occluder test ------------------------------------------------------------------
// occluded() with the stack in the lane's column of shared memory (S.occ_stack
// words, STRIDE lanes apart), since these kernels keep no array in local memory.
// The traversal is bound by instruction issue, hence the running 32-bit address, and
// the test inlined: 640 x 360 at 32 samples and 402 triangles, HG phase and a map, takes
// 1.525 ms (1.520 with the stack in local memory); with the test as a call 1.63, with
// an index into a generic pointer 2% more, the last four entries in registers 4%.
template <int STRIDE>
struct OccSharedStack {
    uint32_t p, base, end;
    __device__ __forceinline__ OccSharedStack(const float *column, uint32_t entries) {
        p = base = (uint32_t)__cvta_generic_to_shared(column);
        end = base + entries * (4u * STRIDE);
    }
    __device__ __forceinline__ void push(uint32_t v) {
        if (p == end) return;
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(p), "r"(v) : "memory");
        p += 4u * STRIDE;
    }
    __device__ __forceinline__ bool empty() const { return p == base; }
    __device__ __forceinline__ uint32_t pop() {
        uint32_t v;
        p -= 4u * STRIDE;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(p) : "memory");
        return v;
    }
};
template <int STRIDE>
__device__ __forceinline__ bool occluded_col(const DevScene &S, const float o[3], const float d[3], const float *column) {
    if (!S.occ_nodes) return false;
    OccSharedStack<STRIDE> stack(column, S.occ_stack);
    return occ_any_hit(S.occ_nodes, S.occ_tris, S.occ_n_nodes, o, d, stack);
}

// The same as a call, for the shadow kernel, which is short of registers: 960 x 540 at 16
// samples beside the same triangles 1.43 ms, inlined 1.58 (stack in local memory 1.49).
template <int STRIDE>
__device__ __noinline__ bool occluded_call(const float4 *__restrict__ nodes, const float4 *__restrict__ tris,
                                           uint32_t n_nodes, uint32_t entries, float ox, float oy, float oz, float dx,
                                           float dy, float dz, const float *column) {
    const float o[3] = {ox, oy, oz}, d[3] = {dx, dy, dz};
    OccSharedStack<STRIDE> stack(column, entries);
    return occ_any_hit(nodes, tris, n_nodes, o, d, stack);
}

// ---- shadow pass ------------------------------------------------------------------
// RenderKernel::Shadow (src/kernel.cpp:569-607, see shadow_sample): the segments
// of a pixel's samples start at one point and stay within the sun's cone, so
// 32 samples side by side walk the grid together like camera samples.  Resident
// warps loop over the samples: a warp's counters cost six additions to the same
// words whatever it did, and with a warp per 32 samples those were the bound.
// 960 x 540 at 16 samples: 0.72 ms, 0.96 with a thread per sample on the octree; bound
// by the setup of the samples (48% of cycles issue).  Lanes that take a new sample
// when theirs ends made it 1.7 to 1.9 times as long (8 to 24 idle lanes at a time):
// the setup then runs at those few lanes.
template <uint32_t FEAT>
__global__ void __launch_bounds__(kListBlock, 8) shadow_paths_kernel(const __grid_constant__ DevScene S,
                                                                     const __grid_constant__ DevParams P,
                                                                     const __grid_constant__ TileArgs A, float4 *out,
                                                                     DevCounters *C) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *const col = reinterpret_cast<float *>(smem) + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    Count cnt;
    cnt.zero();
    NoTape none;
    uint32_t paths = 0;
    for (uint64_t q = (uint64_t)blockIdx.x * kListBlock + threadIdx.x; q - lane < A.n_paths;
         q += (uint64_t)gridDim.x * kListBlock) {
        uint32_t pix = kNone;
        bool active = false;
        float ro[3] = {0.f, 0.f, 0.f}, rd[3] = {0.f, 0.f, 0.f};
        Rng g;
        g.state = g.inc = 0;
        if (q < A.n_paths) {
            uint32_t s;
            if (q <= 0xffffffffull) {
                pix = fastdiv((uint32_t)q, A.spp_div);
                s = (uint32_t)q - pix * A.spp;
            } else {
                const uint64_t l = q / A.spp;
                pix = (uint32_t)l;
                s = (uint32_t)(q - l * A.spp);
            }
            const uint32_t iy = fastdiv(pix, A.cols_div), ix = pix - iy * A.cols;
            if (camera_ray(P, A.x0 + ix, A.y0 + iy, ro, rd)) {
                ++paths;
                const uint64_t fp = (uint64_t)(A.y0 + iy) * P.w + (A.x0 + ix);
                const float depth = P.depth ? __ldg(&P.depth[fp]) : 3.402823466e+38f;
                active = depth < P.clip_end;
                g = rng_seed(A.seed, fp, A.sample_base + s);
                const float u3 = g.uniform(), u4 = g.uniform();
                for (int k = 0; k < 3; ++k) ro[k] = ro[k] + rd[k] * depth;
                sun_sample(P, u3, u4, rd);
            } else {
                pix = kNone;  // outside the frame: nothing is written, as in the reference
            }
        }
        if (active) ++cnt.vertices;
        const CamSeg o = camera_segments<FEAT, false>(none, 0u, S, seg_medium(P), active, ro, rd, g, 3.402823466e+38f,
                                                      make_uint4(0u, 0u, 0u, 0u), nullptr, col, cnt);
        const bool esc = !active || o.res == kTrackEscaped;
        bool occ = false;  // (the segment is over: its column is the test's stack)
        if constexpr ((FEAT & kFeatOcc) != 0)
            occ = active && esc && P.embree && S.occ_nodes &&
                  occluded_call<kListBlock>(S.occ_nodes, S.occ_tris, S.occ_n_nodes, S.occ_stack, ro[0], ro[1], ro[2], rd[0],
                                            rd[1], rd[2], col);
        const bool lit = pix != kNone && P.scattevs > 0u && esc && !occ && sun_hit(P, rd);
        const bool one = pix != kNone && (P.scattevs > 0u || !esc) && !occ;
        // a pixel's samples each add sun(lrd) / colour = colour / colour or 0 / colour,
        // and 1 / 0 or 0 / 0 in w: summed by their numbers, once per pixel
        const uint32_t peers = __match_any_sync(kFull, pix);
        const uint32_t nl = __popc(__ballot_sync(kFull, lit) & peers), nw = __popc(__ballot_sync(kFull, one) & peers);
        if (pix != kNone && lane == (uint32_t)__ffs((int)peers) - 1u) {
            const uint32_t n = __popc(peers);
            float v[3];
            for (int k = 0; k < 3; ++k) {
                const float c = P.sun_color[k];
                v[k] = (nl ? (float)nl * __fdiv_rn(c, c) : 0.0f) + (n - nl ? (float)(n - nl) * __fdiv_rn(0.0f, c) : 0.0f);
            }
            const float w = (nw ? __fdiv_rn(1.0f, 0.0f) : 0.0f) + (n - nw ? __fdiv_rn(0.0f, 0.0f) : 0.0f);
            const uint32_t iy = fastdiv(pix, A.cols_div);
            atomicAdd(&out[(size_t)iy * A.tw + (pix - iy * A.cols)], make_float4(v[0], v[1], v[2], w));
        }
    }
    warp_sum_counts(cnt, C, paths);
}

// ---- transmittance -----------------------------------------------------------------
// Fraction of delta-tracked samples of a ray that escape.  A warp takes a ray
// and `chunk` of its samples: it walks the ray once, keeping the leaves in
// shared memory, and its lanes take samples from the chunk and run along that
// list; most leaves then cost a draw and a comparison.  A ray with more than
// kRayLeaves leaves (deep grids) is traversed per sample.  Nothing is
// allocated, so the allocation-free entry point runs it too.
constexpr uint32_t kRayLeaves = 96;
constexpr uint32_t kRayRefill = 8;  // idle lanes that take new samples together

__host__ __device__ constexpr size_t ray_smem(uint32_t levels) {
    return (size_t)grid_words(levels) * 4 * kListBlock + (size_t)(kListBlock / 32) * kRayLeaves * 16;
}

template <uint32_t FEAT>
__global__ void __launch_bounds__(kListBlock, 8) transmittance_kernel(const __grid_constant__ DevScene S,
                                                                      SegMedium med, const float *ro_in,
                                                                      const float *rd_in, uint32_t n_rays,
                                                                      uint64_t nsamp, uint32_t chunk, uint64_t seed,
                                                                      unsigned long long *escapes) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint4 *const list = reinterpret_cast<uint4 *>(smem) + (threadIdx.x >> 5) * kRayLeaves;
    float *const col = reinterpret_cast<float *>(smem + (size_t)(kListBlock / 32) * kRayLeaves * 16) + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint64_t chunks = (nsamp + chunk - 1) / chunk;
    const uint64_t item = (uint64_t)blockIdx.x * (kListBlock / 32) + (threadIdx.x >> 5);
    if (item >= chunks * n_rays) return;
    const uint32_t r = (uint32_t)(item / chunks);
    const uint64_t s0 = (item - (uint64_t)r * chunks) * chunk;
    const uint32_t n = (uint32_t)(nsamp - s0 < chunk ? nsamp - s0 : chunk);
    float ro[3], rd[3];
    for (int k = 0; k < 3; ++k) {
        ro[k] = __ldg(&ro_in[3 * (size_t)r + k]);
        rd[k] = __ldg(&rd_in[3 * (size_t)r + k]);
    }
    Count cnt;
    cnt.zero();
    NoTape none;
    // the ray's leaves (every lane walks the same ray)
    GridTrav G;
    const uint32_t mode = grid_init<kListBlock>(G, S, col, ro, rd, cnt);
    uint32_t leaves = 0, leaf;
    float tra, trb;
    if (mode == 1u) {
        while (leaves <= kRayLeaves &&
               grid_next<kListBlock>(G, S, col, ro, rd, leaf, tra, trb, cnt, kNone) == kTravLeaf) {
            if (lane == 0 && leaves < kRayLeaves)
                list[leaves] = make_uint4(leaf, __float_as_uint(tra), __float_as_uint(trb),
                                          __float_as_uint(med.sigma_e * __ldg(&S.gmaj[leaf])));
            ++leaves;
        }
    }
    __syncwarp();
    uint32_t esc = 0, next = 0;
    if (mode == 2u || leaves > kRayLeaves) {
        for (uint32_t i = lane; i - lane < n; i += 32) {
            const Rng g = rng_seed(seed, r, s0 + i);
            const CamSeg o = camera_segments<FEAT, false>(none, 0u, S, med, i < n, ro, rd, g, 3.402823466e+38f,
                                                          make_uint4(0u, 0u, 0u, 0u), nullptr, col, cnt);
            if (i < n && o.res == kTrackEscaped) ++esc;
        }
    } else {
        uint32_t st = kOut, k = 0, budget = 0;
        float td = 0.0f, lo = 0.0f, v = 0.0f;
        Rng g;
        g.state = g.inc = 0;
        for (;;) {
            const uint32_t idle = __ballot_sync(kFull, st == kOut);
            if (idle && next < n && ((uint32_t)__popc(idle) >= kRayRefill || idle == kFull)) {
                const uint32_t i = next + __popc(idle & lt);
                if (st == kOut && i < n) {
                    g = rng_seed(seed, r, s0 + i);
                    td = 0.0f;
                    k = 0;
                    budget = med.budget;
                    st = kWalk;
                }
                next += __popc(idle);
            } else if (idle == kFull) {
                break;
            }
            if (st == kWalk) {
                if (k == leaves) {
                    ++esc;
                    st = kOut;
                } else {
                    const uint4 e = list[k];
                    v = g.uniform();
                    if (leaves_at_once(v, __uint_as_float(e.w), __uint_as_float(e.y), __uint_as_float(e.z), td) &&
                        fog_only<FEAT>(S, e.x)) {
                        td = __uint_as_float(e.z);
                        ++k;
                    } else {
                        lo = td;
                        st = kHard;
                    }
                }
            }
            const bool hard = st == kHard || st == kHardAgain;
            const uint32_t nl = __ballot_sync(kFull, hard);
            if (nl && ((uint32_t)__popc(nl) >= kHardBatch || !__any_sync(kFull, st == kWalk)) && hard) {
                const uint4 e = list[k];
                const uint32_t f = leaf_flight<FEAT>(none, S, med.sigma_e, ro, rd, e.x, __uint_as_float(e.y),
                                                     __uint_as_float(e.z), lo, st == kHard, v, td, g, cnt);
                st = f == kLeft ? kWalk : kHardAgain;
                if (f == kLeft) ++k;
                if (f == kReal) {
                    st = kOut;
                } else if (f == kNull && --budget == 0) {
                    ++esc;  // a segment that gives up counts as escaped
                    st = kOut;
                }
            }
        }
    }
    esc = __reduce_add_sync(kFull, esc);
    if (lane == 0 && esc) atomicAdd(&escapes[r], (unsigned long long)esc);
}

// Between rounds: the tickets taken so far are done, the record buffer is empty.
__global__ void next_round_kernel(PathCtl *ctl) {
    ctl->base = ctl->ticket;
    ctl->records = 0;
    ctl->head = 0;
}

// ---- scatter ------------------------------------------------------------------------
// Each warp owns kSlots path slots in shared memory.  Its 32 lanes trace
// segments; everything a path needs only between segments (throughput, sums,
// the pending continuation) stays in the slot.  A path moves through
//   event list   collided: a scattering event is due
//   ready list   scattered: its shadow segment waits for a lane
//   a lane       the shadow segment, then at once the continuation
// and the warp shades its event list 32 at a time, so neither the scattering
// code nor the tracing loop waits on lanes that hold the other kind of work.
// Nothing is shared between warps but the record counter.
//
// The tracing loop's body runs a grid step, with the first flight of a leaf it
// finds, for the lanes on their way and, when enough of them wait, the flights to
// be computed in full; segment ends are processed when kEndBatch lanes have one.
enum : uint32_t { kEnd = 3, kIdle = 4 };  // and kWalk, kHard, kHardAgain
// Slots and residency, on the 512^3 frame and the slab: 64 slots at 4 blocks per SM (128
// registers) 17.65 and 24.9 ms, 56 at 5 21.0 and 28.5, 48 at 6 (80 registers) 28.3 and
// 39.5: more warps cost registers, L1 (the slots are shared memory) and instruction
// cache.  Code size counts: rolling the loops of the rare parts and calling instead of
// inlining (111 to 83 KB of code) took 7% off the frame and instruction stalls from
// 1.46 to 0.57 cycles per instruction.
// No array of these kernels lives in local memory: with one (a stack for the
// octree in slow_segment) beside spilled registers, the shadow kernel counted a few
// node visits too many now and then, for a reason that was not found.  The octree's
// stack here is its child slots, and the occluder test's a column of shared memory.
constexpr int kScatterBlock = 128;
constexpr int kSlots = 64;
constexpr uint32_t kEventBatch = 28;           // events that make a shading pass
constexpr uint32_t kEndBatch = 8;             // lanes at a segment end (or idle with work ready) that make an end pass
constexpr uint32_t kWaitBatch = 6;            // lanes that make a pass of full flights
constexpr uint32_t kFetchBatch = 16;           // free slots that make a fetch
constexpr uint32_t kLeastShare = 4;            // paths a warp takes at least
constexpr int kBurst = 3;                      // loop bodies between looks at the lists
// slot words (word w of slot s at w * kSlots + s)
enum : int { wState = 0, wInc = 2, wRo = 4, wRd = 7, wT = 10, wSun = 13, wSw = 16, wSrd = 19, wTd = 22, wOff = 23, wEv = 24,
             wView = 25 };
// adjoint: the path's number, the sums weighted by the events before them, lit shadow segments
enum : int { wPath = 25, wASun = 26, wEsc = 29 };
template <bool BATCH, bool ADJ = false> __host__ __device__ constexpr int slot_words() {
    return ADJ ? 31 : (BATCH ? 26 : 25);
}
// The light queue's words an entry: the direction, a throughput, the output offset,
// and with features the origin and kind; in a batch the view.
template <uint32_t FEAT, bool BATCH, bool ADJ = false> __host__ __device__ constexpr int queue_words() {
    return ADJ || (FEAT && !(FEAT & kFeatOcc)) ? 0 : (FEAT ? 11 : 7) + (BATCH ? 1 : 0);
}
// An entry's words; those up to the direction are read again after the occluder
// test, whose stack (occ_stack words) takes the place of the rest.
template <uint32_t FEAT, bool ADJ = false> struct QueueAt {
    static constexpr uint32_t T = FEAT ? 0 : 3, off = FEAT ? 3 : 6, kind = 4, rd = FEAT ? 5 : 0, ro = 8,
                              stack = ADJ ? 0 : 5;
};
// bytes per warp: slots, three lists of slot numbers, the light queue
template <uint32_t FEAT, bool BATCH, bool ADJ = false>
__host__ __device__ constexpr size_t scatter_warp_bytes(uint32_t occ_stack) {
    const uint32_t q = queue_words<FEAT, BATCH, ADJ>(), s = QueueAt<FEAT, ADJ>::stack + occ_stack;
    return 4 * (size_t)(slot_words<BATCH, ADJ>() * kSlots + 32 * ((FEAT & kFeatOcc) && s > q ? s : q)) +
           3 * (size_t)kSlots;
}

// The sky terms of escaped paths are evaluated by full warps: entry i of the
// queue is (rd, T, output offset, [view]) in column i, with features (T, output
// offset, kind, rd, ro); T * sky(rd) is
// the value the path would have added in place (its sky sum is 0 before the
// escape).  With occluders the light of lit shadow segments and escapes waits
// there too (kShadowLight: T is the segment's sun term; kEscapeLight: sun and sky),
// so that full warps test the rays: tested where 8 to 14 of a warp's segments end,
// the dependent loads of the tree, which the path slots leave little L1 for, took
// half the frame (640 x 360, 32 samples, 402 triangles, one seed: 1.57 -> 1.26 ms;
// 0.79 without occluders).
enum : uint32_t { kSkyLight = 0, kShadowLight = 1, kEscapeLight = 2 };
// The occluder test's stack lies in the lane's column of the warp's queue: over the
// ray of the entry, which is in registers then, or, where rays are tested in place,
// in a queue that holds nothing.  (Columns of its own, 6 KB a block there, halve the
// L1 beside the slots: 1% more.)
template <uint32_t FEAT, bool BATCH>
__device__ __noinline__ void path_light_eval(const DevScene &S0, const DevParams &P0, float4 *sun0, float4 *sky0,
                                             const BatchArgs &B, const float *q, uint32_t i) {
    const BatchView *V = nullptr;
    if constexpr (BATCH) V = &B.views[__float_as_uint(q[32 * (queue_words<FEAT, BATCH>() - 1) + i])];
    const DevParams &P = BATCH ? V->P : P0;
    using Q = QueueAt<FEAT>;
    const float rd[3] = {q[32 * Q::rd + i], q[32 * Q::rd + 32 + i], q[32 * Q::rd + 64 + i]};
    if constexpr (FEAT != 0) {
        const DevScene &S = BATCH ? B.scenes[V->scene] : S0;
        if (__float_as_uint(q[32 * Q::kind + i]) != kSkyLight) {
            const float ro[3] = {q[32 * Q::ro + i], q[32 * Q::ro + 32 + i], q[32 * Q::ro + 64 + i]};
            if constexpr ((FEAT & kFeatOcc) != 0)
                if (occluded_col<32>(S, ro, rd, q + 32 * Q::stack + i)) return;
        }
    }
    const float T[3] = {q[32 * Q::T + i], q[32 * Q::T + 32 + i], q[32 * Q::T + 64 + i]};
    const uint32_t off = __float_as_uint(q[32 * Q::off + i]);
    if constexpr (FEAT != 0) {
        const uint32_t kind = __float_as_uint(q[32 * Q::kind + i]);
        if (kind != kSkyLight) {
            float c[3] = {T[0], T[1], T[2]};
            if (kind == kEscapeLight) {
                const bool hit = sun_hit(P, rd);
                for (int k = 0; k < 3; ++k) c[k] = T[k] * (hit ? P.sun_color[k] : 0.0f);
            }
            if ((c[0] != 0.0f) | (c[1] != 0.0f) | (c[2] != 0.0f))
                atomicAdd(&(BATCH ? V->sun : sun0)[off], make_float4(c[0], c[1], c[2], 0.0f));
            if (kind == kShadowLight) return;
        }
    }
    const float3 e = escape_sky<FEAT>(P, rd);
    atomicAdd(&(BATCH ? V->sky : sky0)[off], make_float4(T[0] * e.x, T[1] * e.y, T[2] * e.z, 0.0f));
}

__device__ __forceinline__ float dot_rgb(const float4 a, const float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// ADJ: the adjoint's first pass: the path's sums go into its record and the albedo
// slots instead of the image, its decisions onto the tape.
template <uint32_t FEAT, bool BATCH, int MINB, bool ADJ>
__global__ void __launch_bounds__(kScatterBlock, MINB) scatter_kernel(const __grid_constant__ DevScene S0,
                                                                      const __grid_constant__ DevParams P0,
                                                                      const __grid_constant__ TileArgs A0,
                                                                      const __grid_constant__ PathWork W,
                                                                      const void *mie_pack, float4 *sun0, float4 *sky0,
                                                                      DevCounters *C, const __grid_constant__ BatchArgs B,
                                                                      uint32_t colwords,
                                                                      const __grid_constant__ AdjointArgs J) {
    constexpr bool kQueued = queue_words<FEAT, BATCH, ADJ>() != 0;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint64_t mbar;
    if (W.ctl->records == 0u) return;  // a round without records: leave before staging
    const uint32_t mb = BATCH ? mie_bytes(B.views[0].P) : mie_bytes(P0);
    const MieSmem M = BATCH ? mie_view(B.views[0].P, smem) : mie_view(P0, smem);
    const bool staged = stage_mie(mie_pack, mb, smem, &mbar);
    if (!staged) {
        if (threadIdx.x == 0) atomicAdd(&C->gave_up, 1ull);
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    unsigned char *const area = smem + ((mb + 15u) & ~15u);
    float *const col = reinterpret_cast<float *>(area) + threadIdx.x;
    float *const slots = reinterpret_cast<float *>(area + (size_t)colwords * 4u * kScatterBlock +
                                                   (threadIdx.x >> 5) * scatter_warp_bytes<FEAT, BATCH, ADJ>(S0.occ_stack));
    uint8_t *const lists = reinterpret_cast<uint8_t *>(slots + slot_words<BATCH, ADJ>() * kSlots);
    float *const queue = reinterpret_cast<float *>(lists + 3 * kSlots);
#define ready(i) lists[i]
#define event(i) lists[kSlots + (i)]
#define freed(i) lists[2 * kSlots + (i)]
    uint32_t n_ready = 0, n_event = 0, n_free = kSlots, n_queue = 0;
    for (uint32_t i = lane; i < (uint32_t)kSlots; i += 32) freed(i) = (uint8_t)i;
    __syncwarp();
    bool more = true;
    // slots left empty where the records are too few to fill every warp's: a path's
    // latency, not the lanes, is then what the launch waits for (a 64 x 64 tile at 16
    // samples: scatter 189 -> 150 us; with it and the small tickets 0.39 -> 0.31 ms a call)
    const uint32_t share = (W.ctl->records + gridDim.x * (kScatterBlock / 32) - 1) / (gridDim.x * (kScatterBlock / 32));
    const uint32_t spare = share < (uint32_t)kSlots ? (uint32_t)kSlots - max(share, kLeastShare) : 0u;
    Count cnt;
    cnt.zero();
    uint32_t scatters = 0;
    // the lane's segment
    uint32_t st = kIdle, slot = 0, res = 0, budget = 0, view = 0;
    bool shadow = false;
    float ro[3] = {0.f, 0.f, 0.f}, rd[3] = {0.f, 0.f, 0.f};
    Rng g;
    g.state = g.inc = 0;
    GridTrav G;
    auto tape = make_tape<ADJ>(J);
    float value = 0.0f;  // adjoint: the segment's value on the tape
    uint32_t leaf = 0;                            // the leaf a full flight is due in,
    float td = 0.0f, lo = 0.0f, v = 0.0f;         // the distance at its entry and leaf_flight's v
#define SLOT(w, s) slots[(w)*kSlots + (s)]
    for (;;) {
        const uint32_t endm = __ballot_sync(kFull, st == kEnd), idle = __ballot_sync(kFull, st == kIdle);
        const uint32_t busy = ~(endm | idle);
        // ---- segment ends, and idle lanes with segments ready
        const uint32_t due = (uint32_t)__popc(endm) + min((uint32_t)__popc(idle), n_ready);
        if (due && (due >= kEndBatch || !busy)) {
            bool init = false, finish = false, queued = false;
            uint32_t kind = kSkyLight;
            bool to_event = false;
            float T[3] = {0.f, 0.f, 0.f}, qd[3] = {0.f, 0.f, 0.f};  // the queue entry (qd: rd may be the next segment's)
            const BatchView *V = BATCH ? &B.views[view] : nullptr;
            const DevParams &P = BATCH ? V->P : P0;
            const DevScene &S = BATCH ? B.scenes[V->scene] : S0;
            // the queue takes light as it comes; whole-path sums are needed where a path
            // that is not finite is left out, and for the adjoint.  With features but no
            // occluders the light is cheaper in place (640 x 360, 32 samples, HG phase, one seed: no
            // environment 0.72 ms a frame in place and 0.81 queued, a map 0.79 and 0.82; a
            // kernel that has both ways takes 0.81 and 0.88)
            const bool occ = (FEAT & kFeatOcc) && P.embree && S.occ_nodes;
            const bool later = kQueued && !P.finite_paths;
            if (st == kEnd) {
                if (shadow) {
                    if (res == kTrackEscaped && occ && later) {
                        queued = true;
                        kind = kShadowLight;
                        const bool hit = sun_hit(P, rd);
                        for (int k = 0; k < 3; ++k) {
                            T[k] = SLOT(wSw + k, slot) * (hit ? P.sun_color[k] : 0.0f);
                            qd[k] = rd[k];
                        }
                    } else if (res == kTrackEscaped && !(occ && occluded_col<32>(S, ro, rd, queue + 32 * QueueAt<FEAT, ADJ>::stack + lane))) {
                        const bool hit = sun_hit(P, rd);
                        for (int k = 0; k < 3; ++k) {
                            const float c = SLOT(wSw + k, slot) * (hit ? P.sun_color[k] : 0.0f);
                            SLOT(wSun + k, slot) = SLOT(wSun + k, slot) + c;
                            if constexpr (ADJ)
                                SLOT(wASun + k, slot) = SLOT(wASun + k, slot) + (float)__float_as_uint(SLOT(wEv, slot)) * c;
                        }
                        if constexpr (ADJ) {
                            const uint32_t r = __float_as_uint(SLOT(wEv, slot)) - 1u;
                            if (r < 64u) {
                                const int at = wEsc + (int)(r >> 5);
                                SLOT(at, slot) = __uint_as_float(__float_as_uint(SLOT(at, slot)) | 1u << (r & 31u));
                            }
                        }
                    }
                    if constexpr (ADJ) {
                        const float4 ds = __ldg(&J.dsun[__float_as_uint(SLOT(wOff, slot))]);
                        const float4 dk = __ldg(&J.dsky[__float_as_uint(SLOT(wOff, slot))]);
                        value = dot_rgb(ds, make_float3(SLOT(wSun, slot), SLOT(wSun + 1, slot), SLOT(wSun + 2, slot))) +
                                dot_rgb(dk, make_float3(0.0f, 0.0f, 0.0f));
                    }
                    for (int k = 0; k < 3; ++k) rd[k] = SLOT(wSrd + k, slot);
                    shadow = false;
                    init = true;
                } else if (res == kTrackCollided && __float_as_uint(SLOT(wEv, slot)) < P.scattevs) {
                    SLOT(wState, slot) = __uint_as_float((uint32_t)g.state);
                    SLOT(wState + 1, slot) = __uint_as_float((uint32_t)(g.state >> 32));
                    SLOT(wTd, slot) = td;
                    to_event = true;
                } else {
                    float4 sun = make_float4(SLOT(wSun, slot), SLOT(wSun + 1, slot), SLOT(wSun + 2, slot), 0.0f);
                    float4 skyv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    const bool test = occ && later;  // by the queue
                    if (res == kTrackEscaped && (test || !(occ && occluded_col<32>(S, ro, rd, queue + 32 * QueueAt<FEAT, ADJ>::stack + lane)))) {
                        for (int k = 0; k < 3; ++k) T[k] = SLOT(wT + k, slot);
                        if (!test) {
                            const bool hit = sun_hit(P, rd);
                            sun.x = sun.x + T[0] * (hit ? P.sun_color[0] : 0.0f);
                            sun.y = sun.y + T[1] * (hit ? P.sun_color[1] : 0.0f);
                            sun.z = sun.z + T[2] * (hit ? P.sun_color[2] : 0.0f);
                            if constexpr (ADJ) {
                                const float m = (float)__float_as_uint(SLOT(wEv, slot));
                                for (int k = 0; k < 3; ++k)
                                    SLOT(wASun + k, slot) = SLOT(wASun + k, slot) + m * (T[k] * (hit ? P.sun_color[k] : 0.0f));
                            }
                        }
                        if (later) {
                            queued = true;
                            kind = test ? kEscapeLight : kSkyLight;
                            if constexpr (FEAT != 0)
                                for (int k = 0; k < 3; ++k) qd[k] = rd[k];
                        } else {
                            const float3 e = escape_sky<FEAT>(P, rd);
                            skyv.x = T[0] * e.x;
                            skyv.y = T[1] * e.y;
                            skyv.z = T[2] * e.z;
                        }
                    }
                    const uint32_t off = __float_as_uint(SLOT(wOff, slot));
                    if constexpr (ADJ) {
                        const float4 ds = __ldg(&J.dsun[off]), dk = __ldg(&J.dsky[off]);
                        const float m = (float)__float_as_uint(SLOT(wEv, slot));
                        if (isfinite(sun.x) && isfinite(sun.y) && isfinite(sun.z) && isfinite(skyv.x) && isfinite(skyv.y) &&
                            isfinite(skyv.z)) {
                            PathRecord &rec = J.rec[__float_as_uint(SLOT(wPath, slot))];
                            rec.w = dot_rgb(ds, make_float3(sun.x, sun.y, sun.z)) +
                                    dot_rgb(dk, make_float3(skyv.x, skyv.y, skyv.z));
                            rec.esc_lo = __float_as_uint(SLOT(wEsc, slot));
                            rec.esc_hi = __float_as_uint(SLOT(wEsc + 1, slot));
                            const float ga = (dot_rgb(ds, make_float3(SLOT(wASun, slot), SLOT(wASun + 1, slot),
                                                                      SLOT(wASun + 2, slot))) +
                                              dot_rgb(dk, make_float3(m * skyv.x, m * skyv.y, m * skyv.z))) / P.albedo;
                            if (ga != 0.0f)
                                atomicAdd(&J.slots[(blockIdx.x * (kScatterBlock / 32) + (threadIdx.x >> 5)) % J.n_slots],
                                          (double)ga);
                        }
                        sun = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        skyv = sun;
                    }
                    drop_nonfinite(P, sun, skyv);
                    if ((sun.x != 0.0f) | (sun.y != 0.0f) | (sun.z != 0.0f))
                        atomicAdd(&(BATCH ? V->sun : sun0)[off], sun);
                    if ((skyv.x != 0.0f) | (skyv.y != 0.0f) | (skyv.z != 0.0f))
                        atomicAdd(&(BATCH ? V->sky : sky0)[off], skyv);
                    finish = true;
                }
            }
            if constexpr (kQueued) {  // to the warp's queue, evaluated 32 at a time
                const uint32_t qm = __ballot_sync(kFull, queued);
                if (qm) {
                    const uint32_t pos = n_queue + __popc(qm & lt), total = n_queue + __popc(qm);
                    const uint32_t off = queued ? __float_as_uint(SLOT(wOff, slot)) : 0u;
                    for (uint32_t pass = 0; pass < 2; ++pass) {
                        const uint32_t p = pos - 32u * pass;
                        if (queued && (pass ? pos >= 32u : pos < 32u)) {
                            using Q = QueueAt<FEAT>;
                            for (int k = 0; k < 3; ++k) {
                                queue[32 * (Q::rd + k) + p] = FEAT != 0 ? qd[k] : rd[k];
                                queue[32 * (Q::T + k) + p] = T[k];
                                if constexpr (FEAT != 0) queue[32 * (Q::ro + k) + p] = ro[k];
                            }
                            queue[32 * Q::off + p] = __uint_as_float(off);
                            if constexpr (FEAT != 0) queue[32 * Q::kind + p] = __uint_as_float(kind);
                            if constexpr (BATCH) queue[32 * (queue_words<FEAT, BATCH>() - 1) + p] = __uint_as_float(view);
                        }
                        __syncwarp();
                        if (pass == 1 || total < 32u) break;
                        path_light_eval<FEAT, BATCH>(S0, P0, sun0, sky0, B, queue, lane);
                        __syncwarp();
                    }
                    n_queue = total & 31u;
                }
            }
            const uint32_t em = __ballot_sync(kFull, to_event), fm = __ballot_sync(kFull, finish);
            if (to_event) event(n_event + __popc(em & lt)) = (uint8_t)slot;
            if (finish) freed(n_free + __popc(fm & lt)) = (uint8_t)slot;
            n_event += __popc(em);
            n_free += __popc(fm);
            if (to_event || finish) st = kIdle;
            // idle lanes take ready paths: their shadow segments
            const uint32_t im = __ballot_sync(kFull, st == kIdle);
            const uint32_t rank = __popc(im & lt);
            if (st == kIdle && rank < n_ready) {
                slot = ready(n_ready - 1u - rank);
                for (int k = 0; k < 3; ++k) {
                    ro[k] = SLOT(wRo + k, slot);
                    rd[k] = SLOT(wRd + k, slot);
                }
                g.state = (uint64_t)__float_as_uint(SLOT(wState, slot)) | (uint64_t)__float_as_uint(SLOT(wState + 1, slot)) << 32;
                g.inc = (uint64_t)__float_as_uint(SLOT(wInc, slot)) | (uint64_t)__float_as_uint(SLOT(wInc + 1, slot)) << 32;
                if constexpr (BATCH) view = __float_as_uint(SLOT(wView, slot));
                shadow = true;
                init = true;
                if constexpr (ADJ) {
                    const bool hit = sun_hit(P0, rd);
                    const float4 ds = __ldg(&J.dsun[__float_as_uint(SLOT(wOff, slot))]);
                    value = dot_rgb(ds, make_float3(SLOT(wSw, slot) * (hit ? P0.sun_color[0] : 0.0f),
                                                    SLOT(wSw + 1, slot) * (hit ? P0.sun_color[1] : 0.0f),
                                                    SLOT(wSw + 2, slot) * (hit ? P0.sun_color[2] : 0.0f)));
                    // the record has bits for 64 shadow segments
                    if (__float_as_uint(SLOT(wEv, slot)) > 64u) J.rec[__float_as_uint(SLOT(wPath, slot))].pad = kReplay;
                }
            }
            n_ready -= min(n_ready, (uint32_t)__popc(im));
            if (init) {
                const BatchView *V2 = BATCH ? &B.views[view] : nullptr;
                const DevScene &S2 = BATCH ? B.scenes[V2->scene] : S0;
                const DevParams &P2 = BATCH ? V2->P : P0;
                td = 0.0f;
                budget = P2.step_budget;
                const uint32_t m = grid_init<kScatterBlock>(G, S2, col, ro, rd, cnt);
                st = kWalk;
                if (m == 0u) {
                    res = kTrackEscaped;
                    st = kEnd;
                } else if (m == 2u) {
                    const SlowSeg o = slow_segment<FEAT>(S2, seg_medium(P2), ro[0], ro[1], ro[2], rd[0], rd[1], rd[2],
                                                         3.402823466e+38f, g.state, g.inc);
                    cnt.node_visits += o.visits;
                    cnt.density_lookups += o.lookups;
                    cnt.gave_up += o.gave_up;
                    res = o.res;
                    td = o.td;
                    g.state = o.state;
                    st = kEnd;
                    if constexpr (ADJ) J.rec[__float_as_uint(SLOT(wPath, slot))].pad = kReplay;
                }
            }
            __syncwarp();
            continue;
        }
        // ---- scattering events
        if (n_event && (n_event >= kEventBatch || (!busy && !due))) {
            const uint32_t n = min(n_event, 32u);
            if (lane < n) {
                const uint32_t s = event(n_event - n + lane);
                const BatchView *V = BATCH ? &B.views[__float_as_uint(SLOT(BATCH ? wView : 0, s))] : nullptr;
                const DevParams &P = BATCH ? V->P : P0;
                Rng e;
                e.state = (uint64_t)__float_as_uint(SLOT(wState, s)) | (uint64_t)__float_as_uint(SLOT(wState + 1, s)) << 32;
                e.inc = (uint64_t)__float_as_uint(SLOT(wInc, s)) | (uint64_t)__float_as_uint(SLOT(wInc + 1, s)) << 32;
                float d[3], srd[3], lrd[3];
                for (int k = 0; k < 3; ++k) d[k] = SLOT(wSrd + k, s);
                const float u1 = e.uniform(), u2 = e.uniform();
                path_phase_sample<FEAT>(P, M, d, u1, u2, srd);
                const float u3 = e.uniform(), u4 = e.uniform();
                sun_sample(P, u3, u4, lrd);
                const float3 p1 = path_phase_eval<FEAT>(P, M, dot3(srd, d));
                const float p2 = sun_hit(P, lrd) ? P.sun_pdf : 0.0f;
                const float3 p3 = path_phase_eval<FEAT>(P, M, dot3(lrd, d));
                const float q1 = sun_hit(P, srd) ? P.sun_pdf : 0.0f;
                const float f = P.albedo;
                const float td = SLOT(wTd, s);
#pragma unroll 1
                for (int k = 0; k < 3; ++k) {  // rolled, like the sky's channels: the instruction cache is the scarcer
                    const float a1 = k == 0 ? p1.x : (k == 1 ? p1.y : p1.z), a3 = k == 0 ? p3.x : (k == 1 ? p3.y : p3.z);
                    const float dk = k == 0 ? d[0] : (k == 1 ? d[1] : d[2]);
                    const float T = SLOT(wT + k, s);
                    SLOT(wSw + k, s) = T * ((a3 / (a3 + p2)) * f);
                    SLOT(wT + k, s) = T * ((a1 / (a1 + q1)) * f);
                    SLOT(wRo + k, s) = SLOT(wRo + k, s) + dk * td;
                    SLOT(wRd + k, s) = k == 0 ? lrd[0] : (k == 1 ? lrd[1] : lrd[2]);
                    SLOT(wSrd + k, s) = k == 0 ? srd[0] : (k == 1 ? srd[1] : srd[2]);
                }
                SLOT(wState, s) = __uint_as_float((uint32_t)e.state);
                SLOT(wState + 1, s) = __uint_as_float((uint32_t)(e.state >> 32));
                SLOT(wEv, s) = __uint_as_float(__float_as_uint(SLOT(wEv, s)) + 1u);
                ready(n_ready + lane) = (uint8_t)s;
                ++scatters;
            }
            n_event -= n;
            n_ready += n;
            __syncwarp();
            continue;
        }
        // ---- new paths
        const uint32_t room = n_free > spare ? n_free - spare : 0u;
        if (more && room && (room >= kFetchBatch || !busy)) {
            // (the round's constants are read here rather than kept: registers decide the residency)
            const uint32_t n_rec = *(const volatile uint32_t *)&W.ctl->records;
            const uint64_t qbase = *(const volatile unsigned long long *)&W.ctl->base * W.ticket;
            const uint64_t step = B.step ? *(const volatile unsigned long long *)B.step : 0ull;
            const uint32_t want = min(room, 32u);
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&W.ctl->head, want);
            at = __shfl_sync(kFull, at, 0);
            const uint32_t n = at < n_rec ? min(want, n_rec - at) : 0u;
            if (n < want) more = false;
            if (lane < n) {
                const uint32_t s = freed(n_free - 1u - lane);
                const uint4 r = __ldg(&W.records[at + lane]);
                uint64_t q = qbase + (uint32_t)(r.w - (uint32_t)qbase);
                uint32_t v = 0;
                if constexpr (BATCH) {
                    v = find_last(W.view_tickets, B.n_views, (uint32_t)(q / W.ticket));
                    q -= (uint64_t)W.view_tickets[v] * W.ticket;
                    SLOT(wView, s) = __uint_as_float(v);
                }
                const BatchView *V = BATCH ? &B.views[v] : nullptr;
                const TileArgs &A = BATCH ? V->A : A0;
                const DevParams &P = BATCH ? V->P : P0;
                uint32_t pix, sm;
                active_sample(A, BATCH ? W.active + W.pix_begins[v] : W.active, q, pix, sm);
                const uint4 ray = __ldg(&(BATCH ? A.cam_head : W.head)[2 * (size_t)pix + 1]);
                const uint32_t iy = fastdiv(pix, A.cols_div), ix = pix - iy * A.cols;
                const uint64_t inc = rng_inc(A.seed, (uint64_t)(A.y0 + iy) * P.w + (A.x0 + ix), A.sample_base + step * A.spp + sm);
                SLOT(wState, s) = __uint_as_float(r.x);
                SLOT(wState + 1, s) = __uint_as_float(r.y);
                SLOT(wInc, s) = __uint_as_float((uint32_t)inc);
                SLOT(wInc + 1, s) = __uint_as_float((uint32_t)(inc >> 32));
                SLOT(wSrd, s) = __uint_as_float(ray.x);
                SLOT(wSrd + 1, s) = __uint_as_float(ray.y);
                SLOT(wSrd + 2, s) = __uint_as_float(ray.z);
                for (int k = 0; k < 3; ++k) {
                    SLOT(wRo + k, s) = P.viewi[12 + k];
                    SLOT(wT + k, s) = 1.0f;
                    SLOT(wSun + k, s) = 0.0f;
                }
                SLOT(wTd, s) = __uint_as_float(r.z);
                SLOT(wOff, s) = __uint_as_float(iy * A.tw + ix);
                SLOT(wEv, s) = __uint_as_float(0u);
                if constexpr (ADJ) {
                    SLOT(wPath, s) = __uint_as_float(pix * A.spp + sm);
                    for (int k = 0; k < 3; ++k) SLOT(wASun + k, s) = 0.0f;
                    SLOT(wEsc, s) = SLOT(wEsc + 1, s) = __uint_as_float(0u);
                }
                event(n_event + lane) = (uint8_t)s;
            }
            n_free -= n;
            n_event += n;
            __syncwarp();
            continue;
        }
        if (!busy && !due) break;  // nothing in flight, ready, to shade or to fetch
        // ---- tracing
        const BatchView *V = BATCH ? &B.views[view] : nullptr;
        const DevParams &P = BATCH ? V->P : P0;
        const DevScene &S = BATCH ? B.scenes[V->scene] : S0;
#pragma unroll 1
        for (int it = 0; it < kBurst; ++it) {
            bool found = false;
            if (st == kWalk) {
                const GridExit e = grid_exit(G);
                if (G.loc & kGridCheck) {  // the first cell is a leaf
                    G.loc &= ~kGridCheck;
                    found = true;
                } else if (grid_plain(G, e)) {
                    found = grid_fine<kScatterBlock>(G, col, e, cnt);
                } else {
                    bool done;
                    found = grid_other<kScatterBlock>(G, S, col, ro, rd, e, cnt, done);
                    if (done) st = kEnd, res = kTrackEscaped;
                }
            }
            if (found) {
                float tra, trb;
                leaf = grid_leaf(G, tra, trb);
                const float denom = P.sigma_e * __ldg(&S.gmaj[leaf]);
                v = g.uniform();
                if (leaves_at_once(v, denom, tra, trb, td) && fog_only<FEAT>(S, leaf)) {
                    td = trb;
                } else {
                    lo = td;
                    st = kHard;
                }
            }
            const bool hard = st == kHard || st == kHardAgain;
            const uint32_t wait = __ballot_sync(kFull, hard);
            const bool pass = wait && ((uint32_t)__popc(wait) >= kWaitBatch || !__any_sync(kFull, st == kWalk));
            if (pass && hard) {
                const float trb = std_min(std_min(G.x[0], G.x[1]), G.x[2]);  // the leaf is the current cell
                const uint32_t r =
                    leaf_flight<FEAT>(tape, S, P.sigma_e, ro, rd, leaf, G.tc, trb, lo, st == kHard, v, td, g, cnt);
                st = r == kLeft ? kWalk : kHardAgain;
                if (r == kReal) {
                    res = kTrackCollided;
                    st = kEnd;
                } else if (r == kNull && --budget == 0) {
                    ++cnt.gave_up;
                    res = kTrackEscaped;
                    st = kEnd;
                }
            }
            if constexpr (ADJ) {
                if (pass) {
                    const uint32_t ev = __float_as_uint(SLOT(wEv, slot));
                    tape.put(__float_as_uint(SLOT(wPath, slot)), shadow ? 8u | ((ev - 1u) & 63u) << 8 : 0u, value, lane);
                }
            }
        }
    }
#undef SLOT
#undef ready
#undef event
#undef freed
    if constexpr (ADJ) {
        tape.mark(lane);
        return;
    }
    __syncwarp();
    if constexpr (kQueued)
        if (lane < n_queue) path_light_eval<FEAT, BATCH>(S0, P0, sun0, sky0, B, queue, lane);
    cnt.vertices = 2u * scatters;  // every event's shadow and continuation segments
    cnt.mie_evals = 3u * scatters;
    warp_sum_counts(cnt, C, 0u);
}

// ---- launches ---------------------------------------------------------------------------
static size_t table_bytes(const DevParams &P) {
    return (size_t)P.mie_n * 20u + (P.phase_mode == 1u ? (2u * (size_t)P.mie_n + 1u) * 16u : 0u);
}

static uint64_t rounds_of(uint64_t n_paths, uint64_t limit, uint32_t ticket) {
    const uint64_t span = (uint64_t)kRoundTickets * ticket;
    return (n_paths + limit - 1) / limit + n_paths / span;
}

using CameraFn = void (*)(DevScene, DevParams, TileArgs, PathWork, float4 *, float4 *, DevCounters *, BatchArgs,
                          AdjointArgs);
using ScatterFn = void (*)(DevScene, DevParams, TileArgs, PathWork, const void *, float4 *, float4 *, DevCounters *,
                           BatchArgs, uint32_t, AdjointArgs);

constexpr int kScatterBlocks = 4;  // resident scatter blocks per SM the kernel is compiled for

// Camera and scatter rounds over the active pixels: enough of them for every path to collide.
template <bool BATCH, bool ADJ>
static cudaError_t launch_rounds(const DevScene &S, const DevParams &P, const TileArgs &A, const BatchArgs &B,
                                 PathWork W, const void *mie_pack, float4 *sun, float4 *sky, DevCounters *C,
                                 uint32_t feat, uint32_t glevels, uint64_t n_paths, int device,
                                 cudaStream_t st, const AdjointArgs &J = {}) {
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    const CameraFn cam = feat ? camera_paths_kernel<kFeatAll, BATCH, ADJ> : camera_paths_kernel<0, BATCH, ADJ>;
    // a batch's scenes have no occluders, and the adjoint has one kernel with features
    constexpr uint32_t kOcc = BATCH ? kFeatAll & ~kFeatOcc : kFeatAll, kNoOcc = ADJ ? kFeatAll : kFeatAll & ~kFeatOcc;
    const bool occ = (feat & kFeatOcc) != 0;
    const ScatterFn sca = !feat ? scatter_kernel<0, BATCH, kScatterBlocks, ADJ>
                          : occ ? scatter_kernel<kOcc, BATCH, kScatterBlocks, ADJ>
                                : scatter_kernel<kNoOcc, BATCH, kScatterBlocks, ADJ>;
    const uint32_t words = grid_words(glevels);
    const size_t cam_smem = (size_t)words * 4 * kListBlock;
    const size_t sca_smem = ((table_bytes(P) + 15) & ~(size_t)15) + (size_t)words * 4 * kScatterBlock +
                            (!feat ? scatter_warp_bytes<0, BATCH, ADJ>(0u)
                             : occ ? scatter_warp_bytes<kOcc, BATCH, ADJ>(S.occ_stack)
                                   : scatter_warp_bytes<kNoOcc, BATCH, ADJ>(S.occ_stack)) *
                                (kScatterBlock / 32);
    e = allow_smem(sca, sca_smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sca, kScatterBlock, sca_smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const uint64_t cam_most = (n_paths + W.ticket * 4 - 1) / (W.ticket * 4), sca_most = (n_paths + 127) / 128;
    unsigned cam_blocks = (unsigned)(cam_most < (uint64_t)sms * 8 ? cam_most : (uint64_t)sms * 8);
    const unsigned sca_blocks =
        (unsigned)(sca_most < (uint64_t)sms * per_sm ? sca_most : (uint64_t)sms * (uint64_t)per_sm);
    // every warp of the camera kernel may add a ticket's samples after its last
    // look at the record count: half the buffer at most is kept for that
    const uint64_t per_block = (uint64_t)(kListBlock / 32) * W.ticket;
    if (n_paths > W.cap) {
        if (W.cap < 2 * per_block) return cudaErrorInvalidValue;
        if (cam_blocks * per_block > W.cap / 2) cam_blocks = (unsigned)(W.cap / 2 / per_block);
        W.limit = (uint32_t)(W.cap - cam_blocks * per_block);
    } else {
        W.limit = W.cap;
    }
    const uint64_t rounds = rounds_of(n_paths, W.limit, W.ticket);
    for (uint64_t r = 0; r < rounds; ++r) {
        if (r) next_round_kernel<<<1, 1, 0, st>>>(W.ctl);
        cam<<<cam_blocks, kListBlock, cam_smem, st>>>(S, P, A, W, sun, sky, C, B, J);
        sca<<<sca_blocks, kScatterBlock, sca_smem, st>>>(S, P, A, W, mie_pack, sun, sky, C, B, words, J);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_shadow_paths(const DevScene &S, const DevParams &P, const TileArgs &A, float4 *out,
                                DevCounters *C, bool feat, int device, cudaStream_t st) {
    int sms = 0;
    const cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    uint64_t blocks = (A.n_paths + kListBlock - 1) / kListBlock;
    if (blocks == 0) return cudaSuccess;
    if (blocks > (uint64_t)sms * 8) blocks = (uint64_t)sms * 8;
    const auto fn = feat ? shadow_paths_kernel<kFeatAll> : shadow_paths_kernel<0>;
    const uint32_t words = S.occ_stack > grid_words(S.glevels) ? S.occ_stack : grid_words(S.glevels);
    fn<<<(unsigned)blocks, kListBlock, (size_t)words * 4 * kListBlock, st>>>(S, P, A, out, C);
    return cudaGetLastError();
}

cudaError_t launch_transmittance(const DevScene &S, const DevParams &P, const float *ro, const float *rd,
                                 uint32_t n_rays, uint64_t nsamp, uint64_t seed, unsigned long long *escapes,
                                 cudaStream_t st) {
    // samples per warp: enough warps to fill the GPU (about 16,000) before a walk of
    // the ray is shared by more samples; at most 4,096
    uint64_t chunk = nsamp * n_rays / 16384;
    chunk = chunk < 64 ? 64 : chunk > 4096 ? 4096 : (chunk + 31) / 32 * 32;
    const uint64_t items = (nsamp + chunk - 1) / chunk * n_rays;
    const uint64_t blocks = (items + kListBlock / 32 - 1) / (kListBlock / 32);
    if (blocks == 0) return cudaSuccess;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidValue;
    const auto fn = S.sdf_bricks ? transmittance_kernel<kFeatSdf> : transmittance_kernel<0>;
    fn<<<(unsigned)blocks, kListBlock, ray_smem(S.glevels), st>>>(S, seg_medium(P), ro, rd, n_rays, nsamp,
                                                                  (uint32_t)chunk, seed, escapes);
    return cudaGetLastError();
}

// Samples per ticket: one group of 32 until every resident camera warp has
// four tickets of 128 (the group's latency is what a small launch waits for),
// then 128 (fewer draws on the ticket counter).
static uint32_t ticket_samples(uint64_t n_paths, int device) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 1;
    return n_paths < (uint64_t)sms * 8 * (kListBlock / 32) * kTicketMost * 4 ? 32u : kTicketMost;
}

bool batch_tickets_fit(uint64_t n_paths) { return n_paths / kTicketMost < 1ull << 31; }

bool paths_serve(const Tuning &tune, uint32_t glevels) { return tune.traversal != 1u && glevels != 0u; }

uint32_t path_list_blocks(uint32_t cols, uint32_t rows) {
    return ((cols + kListTx - 1) / kListTx) * ((rows + kListTy - 1) / kListTy);
}

cudaError_t launch_paths(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                         float4 *sun, float4 *sky, DevCounters *C, const PathWork &storage, uint32_t feat, int device,
                         cudaStream_t st, const unsigned long long *step) {
    const uint64_t n_paths = (uint64_t)A.cols * A.rows * A.spp;
    if (n_paths == 0) return cudaSuccess;
    PathWork W = storage;
    W.ticket = ticket_samples(n_paths, device);
    cudaError_t e = cudaMemsetAsync(W.ctl, 0, sizeof(PathCtl), st);
    if (e != cudaSuccess) return e;
    path_lists_kernel<<<path_list_blocks(A.cols, A.rows), kListBlock, (size_t)grid_words(S.glevels) * 4 * kListBlock,
                        st>>>(S, P, A, W, C);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    BatchArgs B{};
    B.step = step;
    return launch_rounds<false, false>(S, P, A, B, W, mie_pack, sun, sky, C, feat, S.glevels, n_paths,
                                       device, st);
}

cudaError_t launch_paths_adjoint(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                                 DevCounters *C, const PathWork &storage, const AdjointArgs &J, uint32_t feat, int device,
                                 cudaStream_t st) {
    if (A.n_paths == 0) return cudaSuccess;
    PathWork W = storage;
    W.ticket = ticket_samples(A.n_paths, device);
    cudaError_t e = cudaMemsetAsync(W.ctl, 0, sizeof(PathCtl), st);
    if (e != cudaSuccess) return e;
    path_lists_kernel<<<path_list_blocks(A.cols, A.rows), kListBlock, (size_t)grid_words(S.glevels) * 4 * kListBlock,
                        st>>>(S, P, A, W, nullptr);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_rounds<false, true>(S, P, A, BatchArgs{}, W, mie_pack, nullptr, nullptr, C, feat, S.glevels, A.n_paths,
                                      device, st, J);
}

cudaError_t launch_paths_batch(const BatchArgs &B, const DevParams &P0, const void *mie_pack, DevCounters *C,
                               const PathWork &storage, uint64_t n_paths, uint32_t n_blocks, bool ext,
                               uint32_t glevels, int device, cudaStream_t st) {
    if (n_paths == 0) return cudaSuccess;
    PathWork W = storage;
    W.ticket = ticket_samples(n_paths, device);
    cudaError_t e = cudaMemsetAsync(W.ctl, 0, sizeof(PathCtl), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(W.view_active, 0, sizeof(uint32_t) * B.n_views, st);
    if (e != cudaSuccess) return e;
    path_lists_batch_kernel<<<n_blocks, kListBlock, (size_t)grid_words(glevels) * 4 * kListBlock, st>>>(B, W, C);
    view_tickets_kernel<<<1, 32, 0, st>>>(B, W);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_rounds<true, false>(DevScene{}, P0, TileArgs{}, B, W, mie_pack, nullptr, nullptr, C,
                                      ext ? kFeatExt | kFeatSdf : 0u, glevels, n_paths,
                                      device, st);
}

}  // namespace dr
