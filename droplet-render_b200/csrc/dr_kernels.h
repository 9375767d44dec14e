// Kernel launchers (host side, C++ linkage, internal to the library).
#pragma once
#include <cuda_runtime.h>
#include "dr_internal.h"

namespace dr {

constexpr int kRenderBlock = 128;
constexpr int kPersistentBlock = 128;

// Dynamic shared memory above the default of 48 KB less the kernel's own (a
// barrier) needs the kernel's opt-in on the current device.  The limit belongs to the
// kernel, not to a context: threads that set it to what each of their launches needs
// fail each other's launches.
// So it is raised once, to all that a block can have (227 KB less the kernel's own),
// and never lowered.
cudaError_t raise_smem(const void *fn, size_t smem);
template <class F> cudaError_t allow_smem(F fn, size_t smem) {
    return raise_smem(reinterpret_cast<const void *>(fn), smem);
}

cudaError_t launch_render_tile(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                               float4 *sun_out, float4 *sky_out, DevCounters *C, cudaStream_t st);
cudaError_t launch_shadow_tile(const DevScene &S, const DevParams &P, const TileArgs &A, float4 *out, DevCounters *C,
                               int device, cudaStream_t st);
// Camera leaf list storage for one persistent launch: head[2 * cols * rows],
// pool[cap] and its fill counter (head null: no lists).
struct CamLists {
    uint4 *head = nullptr;
    uint4 *pool = nullptr;
    uint32_t cap = 0;
    unsigned long long *used = nullptr;
    // storage of the path pipeline (null: the persistent kernel runs)
    PathCtl *ctl = nullptr;
    uint32_t *active = nullptr;  // cols * rows
    uint4 *records = nullptr;
    uint32_t rec_cap = 0;
};
// Whether the path pipeline (dr_paths.cu) serves launches with this tuning:
// scenes with a block grid, unless the cell walk is asked for.  No size is left to
// the persistent kernel: a 64 x 64 tile at 16 samples takes 0.33 ms against 0.38, a
// 1920 x 1080 frame at 64 samples 17.6 against 39.4.
bool paths_serve(const Tuning &tune, uint32_t glevels);
// Whether 32 bits number the tickets of a batch's views (view_tickets).
bool batch_tickets_fit(uint64_t n_paths);
// The path pipeline of a tile.  feat: the frame needs the optional features.
// step: a batch's launch counter (its view's samples start at A.sample_base + *step * spp), or null.
cudaError_t launch_paths(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                         float4 *sun, float4 *sky, DevCounters *C, const PathWork &W, uint32_t feat, int device,
                         cudaStream_t st, const unsigned long long *step = nullptr);
// The path pipeline of every view of B (their TileArgs::cam_head set); n_paths:
// their samples, n_blocks: the sum of their path_list_blocks.
cudaError_t launch_paths_batch(const BatchArgs &B, const DevParams &P0, const void *mie_pack, DevCounters *C,
                               const PathWork &W, uint64_t n_paths, uint32_t n_blocks, bool ext, uint32_t glevels,
                               int device, cudaStream_t st);
// The shadow pass and transmittance estimates on a scene with a block grid.
cudaError_t launch_shadow_paths(const DevScene &S, const DevParams &P, const TileArgs &A, float4 *out,
                                DevCounters *C, bool feat, int device, cudaStream_t st);
cudaError_t launch_transmittance(const DevScene &S, const DevParams &P, const float *ro, const float *rd,
                                 uint32_t n_rays, uint64_t nsamp, uint64_t seed, unsigned long long *escapes,
                                 cudaStream_t st);
uint32_t path_list_blocks(uint32_t cols, uint32_t rows);
// Feature bits a frame needs (0: the plain kernels).
uint32_t frame_features(const DevScene &S, const DevParams &P);
// The pipeline's storage in a launch's lists.
inline PathWork path_work(const CamLists &l) {
    PathWork W{};
    W.ctl = l.ctl;
    W.pool_used = &l.ctl->pool_used;
    W.n_active = &l.ctl->n_active;
    W.head = l.head;
    W.pool = l.pool;
    W.pool_cap = l.cap;
    W.active = l.active;
    W.records = l.records;
    W.cap = l.rec_cap;
    return W;
}
// Tile render: the path pipeline where the scene has a block grid (and lists.ctl
// its storage), else the persistent path kernel; Q->next must be 0 (the launcher clears it on st).
// With a stack traversal and lists given, the camera rays' leaf lists are built
// on st first (camera_list_kernel).
cudaError_t launch_render_persistent(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                                     float4 *sun_out, float4 *sky_out, DevCounters *C, WorkQueue *Q,
                                     const Tuning &tune, int device, cudaStream_t st, const CamLists &lists = {});
// Camera leaf lists of a batch: the views' TileArgs::cam_head point at
// lists.head + pix_begins[v]; head null when the views traverse.
struct BatchLists {
    CamLists lists;
    const uint32_t *pix_begins = nullptr;  // first pixel of each view among the batch's pixels
    uint32_t n_pix = 0;
};
// The launches of a batch's graph where the pipeline does not serve it (the
// work queues must be 0):
// the camera leaf lists of every view of B (nothing when lists.head is null);
cudaError_t launch_batch_lists(const BatchArgs &B, const BatchLists &lists, cudaStream_t st);
// one batched persistent kernel over the views of B (P0: the first view's
// parameters, which fix the shared phase tables);
cudaError_t launch_batch_kernel(const BatchArgs &B, const DevParams &P0, const void *mie_pack, DevCounters *C,
                                WorkQueue *Q, const Tuning &tune, bool ext, int device, cudaStream_t st);
// one view of a batch as a plain persistent kernel of its own: the view's
// parameters and tile are kernel arguments (A.cam_head: its lists, already
// built; A.sample_base + *step * spp is its first sample);
cudaError_t launch_batch_view(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                              float4 *sun_out, float4 *sky_out, DevCounters *C, WorkQueue *Q,
                              const unsigned long long *step, const Tuning &tune, int device, cudaStream_t st);
// *step += 1 (the last node of a batch's graph).
cudaError_t launch_batch_step(unsigned long long *step, cudaStream_t st);
cudaError_t launch_probe_leaf(const DevScene &S, const float *ro, const float *rd, uint32_t n, uint32_t maxn,
                              uint32_t *nodes, float *tr0, float *tr1, uint32_t *counts, cudaStream_t st);
cudaError_t launch_probe_occlusion(const DevScene &S, const float *ro, const float *rd, uint32_t n, uint32_t *hit,
                                   cudaStream_t st);
cudaError_t launch_probe_density(const DevScene &S, const uint32_t *nodes, const float *pts, uint32_t n, float *out,
                                 cudaStream_t st);
cudaError_t launch_probe_paths(const DevScene &S, const DevParams &P, const void *mie_pack, const uint32_t *px,
                               const uint32_t *py, const uint64_t *sample, uint32_t n, uint64_t seed,
                               float4 *out_sun, float4 *out_sky, DevCounters *C, cudaStream_t st);
cudaError_t launch_probe_sampler(const DevParams &P, const void *mie_pack, uint32_t what, const float *in, uint32_t n,
                                 float *out, cudaStream_t st);
cudaError_t launch_probe_transmittance(const DevScene &S, const DevParams &P, const float *ro, const float *rd,
                                       uint32_t n_rays, uint64_t nsamp, uint64_t seed, unsigned long long *escapes,
                                       cudaStream_t st);

// Path-replay adjoint of a tile (delta images in tile layout) and of a set of
// transmittance rays; gradients accumulate into grad (brick-pool layout).
// copies > 1: gradients are first spread over `copies` zeroed copies in
// copies_buf (copies * n_leaves * 512 floats), then summed into grad.
// The albedo gradient is gathered in adjoint_slots() zeroed doubles (slots),
// then added to *grad_albedo (and the slots zeroed again).  The paths run in
// chunks of `chunk`: a totals launch writes a 16-byte record per path to
// records (chunk records: the path's weight and which shadow segments escape),
// then a scatter launch replays the chunk's paths.
cudaError_t launch_adjoint_tile(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                                const float4 *dsun, const float4 *dsky, float *grad, float *copies_buf,
                                uint32_t copies, void *records, uint64_t chunk, double *grad_albedo, double *slots,
                                DevCounters *C, cudaStream_t st);
// The same on the path pipeline, the decisions kept on a tape (AdjointArgs):
// chunks are row ranges of the tile (at most 2^23 paths each, records as many),
// tape holds tape_cap entries of 32 bytes.
cudaError_t launch_adjoint_tape(const DevScene &S, const DevParams &P, const TileArgs *chunks, uint32_t n_chunks,
                                const void *mie_pack, const float4 *dsun, const float4 *dsky, float *grad,
                                float *copies_buf, uint32_t copies, void *records, uint4 *tape, uint32_t tape_cap,
                                double *grad_albedo, double *slots, DevCounters *C, const PathWork &W, int device,
                                cudaStream_t st);
// Its first pass: path records, tape and albedo terms of one chunk.
cudaError_t launch_paths_adjoint(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                                 DevCounters *C, const PathWork &W, const AdjointArgs &J, uint32_t feat, int device,
                                 cudaStream_t st);
uint32_t adjoint_slots();
// Reweighted replay of a tile (decisions from S's bricks, weights from pert):
// adds the linearised loss to *loss through the zeroed slots.
cudaError_t launch_reweighted_loss(const DevScene &S, const DevParams &P, const TileArgs &A, const void *mie_pack,
                                   const float4 *dsun, const float4 *dsky, const float *pert, double *loss,
                                   double *slots, DevCounters *C, cudaStream_t st);
cudaError_t launch_adjoint_transmittance(const DevScene &S, const DevParams &P, const float *ro, const float *rd,
                                         const float *wr, uint32_t n_rays, uint64_t nsamp, uint64_t seed, float *grad,
                                         unsigned long long *escapes, cudaStream_t st);
// Leaf majorants of the listed leaf nodes recomputed from the brick pool, in
// the records by node id and by slot (gleaf and gmaj may be null).
cudaError_t launch_leaf_majorants(float4 *leaf, float4 *gleaf, float *gmaj, const uint32_t *leaf_nodes,
                                  uint32_t n_leafnodes, const float *bricks, float scale, cudaStream_t st);

// dst += src, field by field (one thread; a blocking call's counters).
cudaError_t launch_add_counters(DevCounters *dst, const DevCounters *src, cudaStream_t st);

// Allocation-free transmittance: scratch in a file-scope device array.
uint32_t noalloc_max_rays();
cudaError_t noalloc_scratch(int device, unsigned long long **out);
cudaError_t launch_transmittance_noalloc(const DevScene &S, const DevParams &P, unsigned long long *scratch,
                                         const float *ro, const float *rd, uint32_t n_rays, uint64_t nsamp,
                                         uint64_t seed, double *out, cudaStream_t st);

}  // namespace dr
