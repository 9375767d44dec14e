// Internal host/device layouts of the droplet_b200 library (not part of the C ABI).
#pragma once
#include <cstdint>
#include <cstddef>
#include <vector_types.h>

#ifdef __CUDACC__
#define DR_HD __host__ __device__
#else
#define DR_HD
#endif

namespace dr {

constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kLeafBit = 0x80000000u;
constexpr uint32_t kLvox = 8;            // brick edge; the builder and upload enforce it
constexpr uint32_t kBrick = kLvox * kLvox * kLvox;
constexpr int kMaxDepth = 16;            // traversal stack, src/KernelOctree.h:35
constexpr uint32_t kMieMax = 4096;
constexpr uint32_t kStepBudget = 1u << 24;  // tracking steps per segment before a path gives up

// Device scene.  Node ids are the reference's (DFS creation order).
//   child[2*id], child[2*id+1]: the eight child entries of node id, remapped:
//       0 = no child, kLeafBit|c = leaf node c, c = internal node c
//   leaf[2*id]   = (center.xyz, half extent)
//   leaf[2*id+1] = (majorant, FOG brick index bits, SDF brick index bits, slot
//                  bits); an index kNone = no such brick; SDF leaves have
//                  majorant 1; slot: the leaf's place in gleaf (kNone without a block
//                  grid, or when the root does not reach the leaf)
struct DevScene {
    const uint4 *child;
    const float4 *leaf;
    const float *bricks;
    const float *sdf_bricks;   // SDF pool, or null when no leaf has a surface brick
    float root_ce[4];
    uint32_t n_nodes;
    uint32_t n_leaves;
    // Leaf grid for the cell-walk traversal (all leaves at one depth):
    // n = 2^levels leaf cells per axis; macro cells of 8^3 leaf cells;
    // macro[mz][my][mx] = block index or kNone (no leaf in the macro cell);
    // cells[block*512 + z*64 + y*8 + x] = leaf node id or kNone.
    const uint32_t *macro;
    const uint32_t *cells;
    uint32_t levels;     // leaf depth below the root (0 = no grid; stack traversal only)
    uint32_t n;          // leaf cells per axis
    uint32_t mdim;       // macro cells per axis
    // Block grid of the grid traversal (leaves all at one depth, 2 to
    // kGridMaxLevels below the root, fewer than 2^24; glevels = that depth, else
    // 0).  Level j = nodes of 2^j leaf cells per axis.  Blocks are the 4^3-cell
    // nodes; block (x, y, z) has index x + (y << b) + (z << 2b), b = glevels - 2.
    // gblock[i] = (occupancy of cells 0-31, of cells 32-63, first leaf slot | the
    // 2^3-cell nodes present << 24, level of the largest missing octree node
    // holding the block or 1 when it is present); cells in Morton order (x bit 0, y
    // bit 1, z bit 2, then the next bits).  gleaf[2 * slot], [2 * slot + 1] = the
    // leaf records of `leaf`, blocks in index order and cells in Morton order
    // inside one.
    const uint4 *gblock;
    const float4 *gleaf;
    const float *gmaj;  // majorant of each slot (gleaf[2 * slot + 1].x)
    uint32_t glevels;
    float ginv;         // 1 / half extent when all leaves share it, else 0
    // Occluder BVH (null: no occluders).  Node i = occ_nodes[4i .. 4i+3]: left
    // box (min xyz, max x), (max yz, right min xy), (right min z, right max
    // xyz), then (left ref, right ref, left count, right count) as uint32
    // bits: count > 0 = leaf of `count` triangles from ref, count 0 = internal
    // node ref, ref kNone = no child.  Triangle j = occ_tris[3j .. 3j+2]:
    // v0, e1 = v1 - v0, e2 = v2 - v0 (w unused).
    const float4 *occ_nodes;
    const float4 *occ_tris;
    uint32_t occ_n_nodes;
    uint32_t occ_stack;  // entries an any-hit traversal's stack needs: levels of inner nodes below the root
};

constexpr uint32_t kGridMaxLevels = 9;  // block grid: at most 128^3 blocks (32 MB)
constexpr uint32_t kPhaseHG = 2;     // DR_PHASE_HG
constexpr uint32_t kEnvHosek = 0, kEnvNone = 1, kEnvMap = 2;  // DR_ENV_*

constexpr int kOccMaxDepth = 48;     // occluder BVH depth (the traversal stack holds one entry per level)
constexpr float kOccFar = 1e6f;      // MAX_OCCLUSION_DIST, src/SceneOcclusion.h:4

struct DevParams {
    float sigma_s, sigma_a, sigma_e, albedo;   // albedo = sigma_s / (sigma_a + sigma_s) in binary32
    uint32_t scattevs;
    float sun_dir[3], sun_color[3], sun_cos, sun_pdf;
    float sky_cfg[3][9], sky_rad[3];
    const float *mie_pdf;     // mie_n * 3
    const float *mie_cdf;     // mie_n * 3
    const float *mie_exact;   // exact sampler table (mie_n + 1 CDF values of pdf*sin) or null
    uint32_t mie_n;
    uint32_t phase_mode;
    float viewi[16], proji[16];
    uint32_t w, h;
    const float *depth;       // w*h or null
    uint32_t depthcomp;       // KERNEL_DEPTHCOMP: camera rays stop at depth
    uint32_t finite_paths;    // a path whose contribution is not finite adds nothing
    uint32_t embree;          // the reference's USE_EMBREE build: occluder and depth masks on gathered light
    float hg_g;               // kPhaseHG: anisotropy
    uint32_t env_mode;        // kEnvHosek, kEnvNone or kEnvMap
    const float *env_map;     // kEnvMap: env_w * env_h RGBA texels (device)
    uint32_t env_w, env_h;
    float clip_end;           // far clip distance: -z/w of (0,0,1,1) * projInv (src/kernel.cpp:574-575)
    uint32_t step_budget;     // tracking steps per segment before a path gives up (kStepBudget unless set)
};

// What a tracking loop needs of the parameters: the extinction and the step budget.
struct SegMedium {
    float sigma_e;
    uint32_t budget;
};
DR_HD inline SegMedium seg_medium(const DevParams &P) { return SegMedium{P.sigma_e, P.step_budget}; }

// Exact unsigned 32-bit division by an invariant d >= 1 (Granlund and
// Montgomery, "Division by invariant integers using multiplication", PLDI
// 1994, fig. 4.1): with l = ceil(log2 d) and m = floor(2^32 (2^l - d) / d) + 1,
// n / d = (t + ((n - t) >> min(l, 1))) >> max(l - 1, 0), t = mulhi(m, n), for
// every 32-bit n.  The path kernels use it where a path index becomes a pixel.
struct FastDiv {
    uint32_t m, s1, s2;
};

inline FastDiv make_fastdiv(uint32_t d) {
    if (d == 0) d = 1;  // unused divisor (an empty extent)
    uint32_t l = 0;
    while (l < 32 && (1ull << l) < d) ++l;
    FastDiv f;
    f.m = (uint32_t)(((((1ull << l) - d) << 32) / d) + 1);
    f.s1 = l < 1 ? l : 1u;
    f.s2 = l > 0 ? l - 1 : 0u;
    return f;
}

struct TileArgs {
    uint32_t x0, y0, tw, th;
    uint32_t cols, rows;      // rendered extent: even parts of tw, th
    uint32_t spp;
    uint32_t tile;            // persistent kernel: pixel order in tile x tile squares (0 = row-major)
    uint32_t tiles_x;         // squares per row when tile > 0
    uint64_t seed, sample_base;
    uint64_t n_paths;         // path indices: cols * rows * spp (row-major) or squares * tile^2 * spp
    FastDiv spp_div, cols_div, t2_div, tx_div, tile_div;  // division by spp, cols, tile^2, tiles_x, tile
    // Persistent kernel only (its launcher sets it): the sky term of a path
    // that escapes after scattering goes to the warp's queue of sky terms and is
    // evaluated 32 at a time (Hosek sky, no whole-path finiteness check).
    uint32_t defer_sky;
    // The camera rays' leaf sequences, built once per launch by camera_list_kernel
    // (persistent kernel, octree traversal) or path_lists_batch_kernel (a batch on
    // the path pipeline); every sample of a pixel shares its camera ray.  Pixel q = iy * cols + ix: cam_head[2q] = (first
    // entry in cam_pool, leaves, node visits of the root test, node visits
    // after the last leaf), or x = ~0 when the pixel's list did not fit (its
    // samples traverse); cam_head[2q + 1] = (the ray's direction bits, 1 if the
    // pixel has a ray); cam_pool entries = (leaf, tra bits, trb bits, node
    // visits since the previous leaf).  Null: rays are generated per sample and
    // every segment traverses.
    const uint4 *cam_head;
    const uint4 *cam_pool;
};

struct DevCounters {
    unsigned long long paths, vertices, node_visits, density_lookups, mie_evals, gave_up;
};

// Launch-shape choices of the persistent renderer (chosen by the autotuner).
struct Tuning {
    uint32_t kernel;        // 0 = persistent path kernel, 1 = one thread per path
    uint32_t block;         // threads per block (multiple of 32)
    uint32_t blocks_per_sm; // 0 = as many as fit
    uint32_t event_batch;   // lanes of a warp that must be waiting before events run
    uint32_t traversal;     // 0 = octree stack traversal, 1 = leaf-grid cell walk
    uint32_t tile;          // pixel order of the persistent kernel: 0 = row-major, else square side
    uint32_t visits;        // stack traversal: node examinations per loop iteration (0 = to the next leaf)
    uint32_t steps;         // free-flight steps per loop iteration (0 = 1)
};

// One view of a batched launch: its parameters, tile and output, the scene it
// renders and the first global path index it owns.
struct BatchView {
    DevParams P;
    TileArgs A;
    float4 *sun, *sky;
    uint32_t scene;
    uint32_t pad;
    uint64_t begin;
};

// A batched launch: every view's paths form one index space [0, n_paths) in
// view order; begins[v] = views[v].begin (binary-searched per fetched path).
struct BatchArgs {
    const BatchView *views;
    const DevScene *scenes;
    const uint64_t *begins;
    uint32_t n_views;
    uint64_t n_paths;
    const unsigned long long *step;  // launches so far: view samples start at sample_base + step * spp
};

// Work queue of the persistent kernel: next path index to hand out.
struct WorkQueue {
    unsigned long long next;
};

// Control words of the path pipeline (dr_paths.cu), zero before a launch.
struct PathCtl {
    unsigned long long ticket;  // next camera ticket
    unsigned long long base;    // the first ticket of this round
    unsigned long long pool_used;  // leaf list entries asked for (may exceed the pool)
    uint32_t records;           // collided samples recorded in this round
    uint32_t head;              // the next record to scatter
    uint32_t n_active;          // active pixels
    uint32_t tape_used;         // adjoint: tape entries handed out
};
constexpr uint32_t kRoundTickets = 1u << 24;  // tickets of one round: at most 2^31 samples, so 32 bits tell them apart

// What the adjoint's first pass keeps per path (16 bytes): the path's weight
// dsun . C_sun + dsky . C_sky (NaN: left out), the bits of its lit shadow
// segments (0-63), and kReplay when the tape does not hold all its decisions.
struct alignas(16) PathRecord {
    float w;
    uint32_t esc_lo, esc_hi, pad;
};
constexpr uint32_t kReplay = 1;

// Adjoint runs of the path pipeline: the image gradients (the tile's layout),
// the path records (by pixel * spp + sample, preset to NaN) and the tape.  A
// tape entry (two uint4) is one tracking decision: (path, brick sample of the
// lower corner, flags, denominator), (trilinear fractions, segment value).
// Flags: bits 0-2 the upper corner differs in x, y, z; bit 3 a shadow segment,
// whose number is in bits 8-13.  Denominator: the density (a real collision) or
// minus (majorant - density).  Segment value: a shadow segment's dsun . C, else
// what the path had added before the segment.
struct AdjointArgs {
    const float4 *dsun, *dsky;
    PathRecord *rec;
    uint4 *tape;
    uint32_t tape_cap;        // entries
    uint32_t *tape_used;      // entries handed out (may exceed the capacity)
    double *slots;            // albedo gradient, n_slots partial sums
    uint32_t n_slots;
};

// Storage of the path pipeline for one launch at a time.
struct PathWork {
    PathCtl *ctl;
    unsigned long long *pool_used;   // where the list kernel counts
    uint32_t *n_active;
    uint4 *head;                     // leaf list headers, 2 per pixel (TileArgs::cam_head)
    uint4 *pool;                     // leaf list entries: (slot, tra bits, trb bits, node visits since the previous leaf)
    uint32_t pool_cap;
    uint32_t *active;                // pixels (iy * cols + ix) whose camera ray meets a leaf
    // collided camera samples: (stream state, distance bits, sample number mod 2^32)
    uint4 *records;
    uint32_t cap;                    // records that fit
    uint32_t limit;                  // no new ticket above this count (set by the launcher)
    uint32_t ticket;                 // camera samples per ticket (set by the launcher)
    // batches
    uint32_t *view_tickets;          // first ticket of each view, then their number
    uint32_t *view_active;           // active pixels of each view
    const uint32_t *pix_begins;      // first pixel of each view
    const uint32_t *block_begins;    // first block of each view in the list kernel
};

}  // namespace dr
