// Host-side helpers shared by the C-ABI entry points (dr_api.cu, dr_batch.cu):
// error reporting, device buffers, and the validation + conversion of scenes
// and render settings into their device layouts.
#pragma once
#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#include "../../include/droplet_b200.h"
#include "dr_internal.h"

namespace dr {

void set_error(int code, const std::string &msg);
const char *last_error();
int cuda_fail(cudaError_t e, const char *what);
// Returns DR_OK when ok, else records msg and returns code.
int need(bool ok, int code, const char *msg);

#define DR_CUDA(call, what)                                  \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return cuda_fail(e_, what);   \
    } while (0)

template <typename T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaError_t reserve(size_t count) {
        if (count <= n && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        cudaError_t e = cudaMalloc(&p, sizeof(T) * (count ? count : 1));
        if (e == cudaSuccess) n = count;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

// Storage of the camera leaf lists and the path pipeline (TileArgs::cam_head,
// PathWork) for `renders` launches side by side over up to `pixels` pixels in all:
// headers and active pixels per pixel (shared out by rows), and for each launch a pool of list
// entries, a buffer of collided samples and control words, in one allocation.
constexpr uint32_t kCamPool = 1u << 23;
struct ListWant {
    uint32_t renders;     // 1, or 2 for the band streams of the blocking render
    size_t pixels;
    bool pool_set;        // dr_set_camera_lists: pool_entries, else in proportion to the pixels
    uint32_t pool_entries;
    size_t most_records;  // paths the launches have at most (the adjoint's chunks), or ~0
    bool operator==(const ListWant &o) const {
        return renders == o.renders && pixels == o.pixels && pool_set == o.pool_set && pool_entries == o.pool_entries &&
               most_records == o.most_records;
    }
};
struct ListLayout {
    uint32_t rec_cap, pool_cap;
    size_t records, pool, head, active, ctl, used, bytes;  // byte offsets, and their end
};
// shift: records and pool entries as many times halved (to no less than 2^16 and 2^14).
inline ListLayout list_layout(const ListWant &w, uint32_t shift) {
    ListLayout l;
    // Records: 16 MB to 512 MB (128 MB a band stream, which renders an eighth of a
    // large tile's rows at a time), in proportion to the pixels in between.  A render
    // whose paths may exceed them runs in rounds, and a round without work costs about 8 us.
    const bool two = w.renders == 2u;
    const size_t most = two ? (size_t)1 << 23 : (size_t)1 << 25, least = (size_t)1 << 20;
    size_t rec = std::min(most, std::max(least, w.pixels * (two ? 4 : 16)));
    rec = std::min(rec, std::max(least, w.most_records));
    l.rec_cap = (uint32_t)std::max(rec >> shift, std::min(rec, (size_t)1 << 16));
    // list entries: 32 a pixel (8 a band stream) up to kCamPool
    const size_t pool = w.pool_set ? w.pool_entries
                                   : std::min((size_t)kCamPool, std::max((size_t)1 << 18, w.pixels * (two ? 8 : 32)));
    l.pool_cap = (uint32_t)std::max(pool >> shift, std::min(pool, (size_t)1 << 14));
    size_t at = 0;
    auto part = [&at](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255) & ~(size_t)255;
        return o;
    };
    l.records = part(w.renders * (size_t)l.rec_cap * sizeof(uint4));
    l.pool = part(w.renders * (size_t)l.pool_cap * sizeof(uint4));
    l.head = part(2 * w.pixels * sizeof(uint4));
    l.active = part(w.pixels * sizeof(uint32_t));
    l.ctl = part(w.renders * sizeof(PathCtl));
    l.used = part(w.renders * sizeof(unsigned long long));
    l.bytes = at;
    return l;
}
// The largest of those layouts that the memory holds: with fewer records a render takes more
// rounds, with a smaller pool more pixels traverse per sample, without any of it
// the persistent kernel runs, which is half as fast.  The answer is kept until something
// else is wanted; a lack of any memory until retry().  reserve returns a
// cudaError_t; an error that is not about memory (a stream is being captured) says
// nothing about the next call.
struct ListFit {
    ListWant want{};
    ListLayout layout{};
    bool known = false, ok = false;
    void retry() { known = known && ok; }
    template <class R> bool fit(const ListWant &w, R reserve) {
        if (known && want == w) return ok;
        want = w;
        known = true;
        ok = false;
        size_t last = 0;
        for (uint32_t shift = 0; shift < 32; ++shift) {
            layout = list_layout(w, shift);
            if (layout.bytes == last) break;  // the smallest
            last = layout.bytes;
            const cudaError_t e = reserve(layout.bytes);
            ok = e == cudaSuccess;
            if (ok) return true;
            known = e == cudaErrorMemoryAllocation;
            if (!known) return false;
        }
        return false;
    }
};
struct ListStore {
    DevBuf<unsigned char> buf;
    ListFit fit;
};

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

// A validated scene in its device layout, still on the host.
struct HostScene {
    std::vector<uint32_t> child;   // 8 per node (see DevScene)
    std::vector<float4> leaf;      // 2 per node
    std::vector<uint32_t> macro, cells;
    std::vector<uint8_t> leaf_flag;
    uint32_t levels = 0, n = 0, mdim = 0;
    std::vector<uint4> gblock;     // block grid of the grid traversal (DevScene::gblock)
    std::vector<float4> gleaf;     // leaf records by slot (DevScene::gleaf)
    std::vector<float> gmaj;       // majorants by slot (DevScene::gmaj)
    uint32_t glevels = 0;
    float ginv = 0.0f;             // DevScene::ginv
    uint32_t n_nodes = 0, n_leaves = 0;
    float root_ce[4] = {0, 0, 0, 0};
    const float *bricks = nullptr;  // the caller's brick pool (n_leaves * 512 floats)
    const float *sdf = nullptr;     // the caller's SDF pool (n_sdf * 512 floats) or null
    uint32_t n_sdf = 0;
};

// Device buffers of one uploaded scene.
struct SceneBufs {
    DevBuf<uint4> child;
    DevBuf<float4> leaf;
    DevBuf<float> bricks;
    DevBuf<float> sdf;
    DevBuf<uint32_t> macro, cells;
    DevBuf<uint4> gblock;
    DevBuf<float4> gleaf;
    DevBuf<float> gmaj;
    void release() {
        child.release();
        leaf.release();
        bricks.release();
        sdf.release();
        macro.release();
        cells.release();
        gblock.release();
        gleaf.release();
        gmaj.release();
    }
};

// Checks a scene descriptor (src/scene.h:21-31 records) and builds the device
// layout: remapped child entries, leaf records, and the leaf grid of the cell walk.
int prepare_scene(const dr_scene_desc *s, HostScene &out);
// Copies a prepared scene into bufs (synchronously on st) and fills S.
int upload_scene(const HostScene &h, SceneBufs &bufs, bool use_grid, cudaStream_t st, DevScene &S);
// Checks render settings and converts them (the depth pointer is left null);
// pack receives the phase tables as staged in shared memory.
int prepare_params(const dr_render_params *p, DevParams &d, std::vector<unsigned char> &pack);
// Shared-memory pack size of the phase tables for d.
size_t mie_pack_bytes(const DevParams &d);
// Tile arguments of a render call (tile > 0: square pixel order of the persistent kernel).
int make_tile_args(uint32_t x0, uint32_t y0, uint32_t tw, uint32_t th, uint32_t spp, uint64_t seed, uint64_t base,
                   uint32_t tile, TileArgs &A);
bool valid_tuning(const dr_tuning *t);

// Occluder BVH as built on the host (layout of DevScene::occ_nodes/occ_tris,
// 16 and 12 floats per node and triangle); source[j] = the selected triangle
// (in surface order) stored at position j.
struct OccBvh {
    std::vector<float> nodes;
    std::vector<float> tris;
    std::vector<uint32_t> source;
    uint32_t depth = 0;  // levels of inner nodes below the root (DevScene::occ_stack)
};
int build_occluder_bvh(const dr_surface *s, uint32_t n, uint32_t mode, OccBvh &out);

}  // namespace dr

// The context behind the C ABI's opaque dr_ctx handle.
namespace dr {
// Host threads that share the copies from pinned staging into the caller's
// buffers (dr_render_tile).  The costly bands of a frame (the cloud's rows)
// tend to finish last and close together, so one thread copying each 8 MB band
// after it lands (about 1 ms each) put several milliseconds after the last
// kernel; split over the pool's threads and the calling thread, each copy
// takes a fraction of that.  Threads start on the first large copy and stop
// when the pool is destroyed.
class CopyPool {
  public:
    struct Range {
        void *dst;
        const void *src;
        size_t bytes;
    };
    CopyPool() = default;
    CopyPool(const CopyPool &) = delete;
    CopyPool &operator=(const CopyPool &) = delete;
    ~CopyPool() {
        {
            std::lock_guard<std::mutex> lk(m_);
            quit_ = true;
        }
        work_.notify_all();
        for (std::thread &t : threads_) t.join();
    }
    // Copies every range; returns when all bytes are in place.
    void copy(const Range *r, size_t n) {
        size_t total = 0;
        for (size_t i = 0; i < n; ++i) total += r[i].bytes;
        start();
        if (threads_.empty() || total < kMinSplit) {
            for (size_t i = 0; i < n; ++i) std::memcpy(r[i].dst, r[i].src, r[i].bytes);
            return;
        }
        const size_t parts = threads_.size() + 1;
        const size_t chunk = ((total / parts) + 4095) & ~(size_t)4095;
        {
            std::lock_guard<std::mutex> lk(m_);
            jobs_.clear();
            next_ = 0;
            for (size_t i = 0; i < n; ++i)
                for (size_t o = 0; o < r[i].bytes; o += chunk)
                    jobs_.push_back({static_cast<char *>(r[i].dst) + o, static_cast<const char *>(r[i].src) + o,
                                     r[i].bytes - o < chunk ? r[i].bytes - o : chunk});
            pending_ = jobs_.size();
        }
        work_.notify_all();
        for (;;) {  // the calling thread copies too
            Job j;
            {
                std::lock_guard<std::mutex> lk(m_);
                if (next_ >= jobs_.size()) break;
                j = jobs_[next_++];
            }
            run(j);
        }
        std::unique_lock<std::mutex> lk(m_);
        done_.wait(lk, [&] { return pending_ == 0; });
    }

  private:
    static constexpr size_t kMinSplit = 4u << 20;
    struct Job {
        char *dst;
        const char *src;
        size_t n;
    };
    void run(const Job &j) {
        std::memcpy(j.dst, j.src, j.n);
        std::lock_guard<std::mutex> lk(m_);
        if (--pending_ == 0) done_.notify_all();
    }
    void start() {
        if (started_) return;
        started_ = true;
        const unsigned hw = std::thread::hardware_concurrency();
        const unsigned n = hw > 1 ? (hw < 8 ? hw : 8) - 1 : 0;
        try {
            for (unsigned i = 0; i < n; ++i) threads_.emplace_back([this] { loop(); });
        } catch (...) {  // fewer threads (or none): the calling thread copies the rest
        }
    }
    void loop() {
        for (;;) {
            Job j;
            {
                std::unique_lock<std::mutex> lk(m_);
                work_.wait(lk, [&] { return quit_ || next_ < jobs_.size(); });
                if (quit_) return;
                j = jobs_[next_++];
            }
            run(j);
        }
    }
    std::mutex m_;
    std::condition_variable work_, done_;
    std::vector<std::thread> threads_;
    std::vector<Job> jobs_;
    size_t next_ = 0, pending_ = 0;
    bool quit_ = false, started_ = false;
};
}  // namespace dr

struct dr_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::mutex mu;
    bool has_scene = false, has_params = false;
    dr::DevScene scene{};
    dr::DevParams params{};
    dr::SceneBufs bufs;
    dr::DevBuf<unsigned char> mie_pack;
    dr::DevBuf<float> depth;
    dr::DevBuf<float> env;            // environment map texels (DR_ENV_MAP)
    dr::DevBuf<dr::DevCounters> counters;
    dr::DevBuf<dr::DevCounters> call_counters;  // a blocking call's own counts (added to `counters` at its end)
    uint32_t step_budget = dr::kStepBudget;     // dr_set_step_budget
    unsigned long long gave_up_reported = 0;    // counters.gave_up when dr_check_complete last looked
    dr::DevBuf<float4> tile_sun, tile_sky;
    dr::DevBuf<unsigned char> scratch;
    dr::DevBuf<dr::WorkQueue> work;
    dr::DevBuf<uint32_t> leaf_nodes;  // ids of the leaf nodes (majorant updates)
    dr::DevBuf<float> grad_copies;    // adjoint: spread copies of the brick-pool gradient
    dr::DevBuf<double> albedo_slots;  // adjoint: partial sums of the albedo gradient (kept zeroed)
    dr::DevBuf<uint4> path_rec;       // adjoint: one record per path of a chunk (totals pass -> scatter pass)
    dr::DevBuf<uint4> tape;           // adjoint: tracking decisions (AdjointArgs::tape)
    dr::DevBuf<float4> occ_nodes, occ_tris;  // occluder BVH (kept across scene uploads)
    uint32_t occ_n_nodes = 0, occ_stack = 0;
    uint32_t n_leaf_nodes = 0;
    bool use_grid = true;
    dr::Tuning tuning{0u, 128u, 0u, 8u, 0u, 0u, 0u, 0u};
    std::vector<uint8_t> leaf_flag;  // host copy: node i is a leaf (for validating probe inputs)
    // host-buffer render pipeline (dr_render_tile): row bands rendered on two
    // streams, each copied to pinned staging as soon as it is done
    static constexpr int kBands = 8;
    cudaStream_t band_stream[2] = {nullptr, nullptr};
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t ev_clear = nullptr;
    cudaEvent_t band_done[kBands] = {};
    cudaEvent_t copy_done[kBands] = {};
    dr::DevBuf<dr::WorkQueue> band_work;
    // camera leaf lists and path pipeline: the asynchronous render's storage, that of the
    // blocking render's two band streams, and the adjoint's
    uint32_t cam_cap = 0;      // entries per pool when set (dr_set_camera_lists; 0: no lists)
    bool cam_cap_set = false;  // else in proportion to the frame, up to kCamPool
    dr::ListStore lists, band_lists, adjoint_lists;
    uint64_t tape_most = 1ull << 25;  // adjoint: tape entries (32 bytes) at most; halved while the memory does not do
    float *pinned = nullptr;  // 2 * pinned_n float4: sun then sky
    size_t pinned_n = 0;
    dr::CopyPool copies;      // host threads for the staging -> caller copies
};
