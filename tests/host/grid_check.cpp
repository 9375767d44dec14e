// Host check of the grid traversal against the octree traversal, both from the
// device headers: leaves, intervals and node visits after every leaf, one step
// at a time, on random, lattice-aligned, tied and far-away rays.
//   grid_check SCENE RAYS SEED    (SCENE: n_nodes, n_leaves, then the node records)
//   grid_check flights N SEED     leaves_at_once against the flight in full
//   grid_check pool N SEED        ranges of a leaf list pool while N lists ask for them
//   grid_check exact N SEED       draws, logarithms, lookups and collision tests against the plain operations
//   grid_check storage N SEED     list and pipeline storage in N amounts of free memory
#include "cuda_host_shim.h"
#include "../../droplet-render_b200/csrc/dr_device.cuh"
#include "../../include/droplet_b200.h"
#include "../../droplet-render_b200/csrc/dr_host.h"
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
using namespace dr;

static int flights(long long n, int seed) {
    double least = 1e9;
    for (uint32_t k = 0; k < (1u << 23); ++k) {  // every value of Rng::uniform
        const float u = (float)(2 * k + 1) * 5.96046448e-08f;
        least = std::min(least, -(double)dlog(u) / (1.0 - (double)u));
    }
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(0, 1);
    long long bad = 0, quick = 0, left = 0;
    for (long long i = 0; i < n; ++i) {
        const double len = std::pow(10, -8 + 9 * U(g));
        const float td = (float)((g() & 1) ? 0 : std::pow(10, -3 + 6 * U(g)));
        const float tra = (float)((g() & 3) == 0 ? td : (g() & 1) ? td + std::pow(10, -9 + 8 * U(g)) : td - len * U(g));
        const float trb = (g() & 63) ? (float)(tra + len) : tra;
        const float denom = (g() & 255) ? (float)(std::pow(10, -6 + 7 * U(g)) / len) : 0.0f;
        uint32_t k = g() & 0x7fffff;
        if (g() & 1) {  // draws around the decision
            const double x = 1 - 1.0001 * (double)denom * ((trb - td) - (tra > td ? tra - td : 0));
            const long kk = x > 0 && x < 1 ? (long)(x * 8388608) + (long)(g() % 9) - 4 : -1;
            if (kk >= 0 && kk < (1 << 23)) k = (uint32_t)kk;
        }
        const float u = (float)(2 * k + 1) * 5.96046448e-08f;
        const float tr0 = tra - td, tr1 = trb - td;
        const float s0 = tra > td ? tr0 : __uint_as_float(__float_as_uint(tr0) & 1u);
        const float sr = 0.0f - dlog(u) / denom;
        const bool out = !(s0 + sr < tr1), q = leaves_at_once(u, denom, tra, trb, td);
        quick += q;
        left += out;
        bad += q && !out;
    }
    std::printf("least -dlog(u) / (1 - u) %.9f quick %lld left %lld bad %lld\n", least, quick, left, bad);
    return least < 1.0 - 1e-6 || bad || quick < left / 2;
}

static int pool(long long n, int seed) {
    // lists of 1 to 2^20 entries: the ranges handed out lie in the pool one after the other, however many are asked for
    std::mt19937_64 g(seed);
    const uint32_t cap = (1u << 26) - 3;
    unsigned long long used = 0;
    uint64_t end = 0, bad = 0, asked = 0;
    for (long long i = 0; i < n; ++i) {
        const uint32_t k = 1u + (uint32_t)(g() >> (44 + g() % 20)), off = pool_range(&used, k, cap);
        asked += k;
        if (off == kNone) continue;
        bad += off < end || (uint64_t)off + k > cap;
        end = (uint64_t)off + k;
    }
    unsigned long long edge = cap - 5;  // exactly the rest, and one more
    bad += pool_range(&edge, 6, cap) != kNone;
    edge = cap - 5;
    bad += pool_range(&edge, 5, cap) != cap - 5 || pool_range(&edge, 1, cap) != kNone;
    std::printf("asked %llu end %llu bad %llu\n", (unsigned long long)asked, (unsigned long long)end, (unsigned long long)bad);
    return bad || asked < 3ull << 32;
}

static int exact(long long n, int seed) {
    auto bits = [](float f) { return __float_as_uint(f); };
    long long bad[4] = {}, near = 0, close = 0;
    for (uint32_t k = 0; k < (1u << 23); ++k) {  // every value of Rng::uniform
        const float u = (float)(2 * k + 1) * 5.96046448e-08f;
        bad[0] += bits(dlog_unit(u)) != bits(dlog(u));
    }
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> U(0, 1);
    static float brick[512];
    Rng a;
    a.state = g();
    a.inc = g() | 1;
    for (long long i = 0; i < n; ++i) {
        Rng b = a;
        const uint32_t w = b.next();
        bad[1] += bits(a.uniform()) != bits((float)(((w >> 9) << 1) | 1u) * 5.96046448e-08f) || a.state != b.state;
        // rho / smax < q, also within a few ulp of the tie, and with values that are not finite
        const float smax = (g() & 1023) ? (float)std::pow(10, -8 + 16 * U(g)) : (g() & 1) ? 0.0f : INFINITY;
        const float q = (float)(2 * (g() >> 41) + 1) * 5.96046448e-08f;
        float rho = (float)(smax * U(g) * ((g() & 15) ? 1.0 : -1.0));
        if (g() & 1) {
            rho = q * smax;
            for (int d = (int)(g() % 17) - 8; d; d += d < 0 ? 1 : -1) rho = std::nextafterf(rho, d < 0 ? -1e30f : 1e30f);
        }
        if ((g() & 4095) == 0) rho = NAN;
        bad[2] += ratio_below(rho, smax, q) != (rho / smax < q);
        near += rho / smax == q;
        // the lookup's cell and fractions: inside the brick, on its lattice, at its faces and far away
        const float e = (float)std::pow(10, -6 + 8 * U(g)), inv = 1.0f / e;
        float c[3], p[3];
        for (int k = 0; k < 3; ++k) {
            c[k] = (float)((g() & 3) ? e * (double)(g() % 1000) : (2 * U(g) - 1) * 100 * e);
            const double x = (g() & 3) == 0 ? (double)(g() % 15) / 7 - 1 : (g() & 7) ? 2 * U(g) - 1 : 6 * U(g) - 3;
            p[k] = (float)(c[k] + x * e * ((g() & 255) ? 1.0 : std::pow(10, 9 * U(g))));
            for (int d = (int)(g() % 5) - 2; d; d += d < 0 ? 1 : -1) p[k] = std::nextafterf(p[k], d < 0 ? -1e30f : 1e30f);
        }
        uint32_t ia[3], ib[3], ja[3], jb[3];
        float na[3], nb[3];
        const float4 ce = make_float4(c[0], c[1], c[2], e);
        if (!voxel_cell_inv(p, ce, inv, ia, ib, na)) continue;  // far: takes the plain lookup
        ++close;
        voxel_cell(p, ce, ja, jb, nb);
        for (int k = 0; k < 3; ++k) bad[3] += ia[k] != ja[k] || ib[k] != jb[k] || bits(na[k]) != bits(nb[k]);
        if (i % 64 == 0)
            for (float &v : brick) v = (g() & 3) ? (float)U(g) : 0.0f;
        bad[3] += bits(sample_voxel_inv(p, brick, ce, inv)) != bits(sample_voxel_space(p, brick, ce));
    }
    std::printf("ties %lld close %lld bad %lld %lld %lld %lld\n", near, close, bad[0], bad[1], bad[2], bad[3]);
    return bad[0] || bad[1] || bad[2] || bad[3] || near < n / 100 || close < n / 2;
}

static int storage(long long n, int seed) {
    std::mt19937_64 g(seed);
    long long bad = 0, fitted = 0, none = 0;
    for (long long i = 0; i < n; ++i) {
        const size_t pixels = (size_t)1 << (g() % 24);
        ListWant w{1u + (uint32_t)(g() & 1), pixels + g() % pixels, (g() & 3) == 0, (uint32_t)(g() % (1u << 24)), ~(size_t)0};
        if (g() & 1) w.most_records = g() % (1u << 23);
        const size_t room = ((size_t)1 << 20) << (g() % 12);
        int tries = 0;
        auto reserve = [&](size_t bytes) { return ++tries, bytes <= room ? cudaSuccess : cudaErrorMemoryAllocation; };
        ListFit f;
        const bool ok = f.fit(w, reserve);
        const ListLayout full = list_layout(w, 0), least = list_layout(w, 31), &l = f.layout;
        bad += ok != (least.bytes <= room);  // some layout is found whenever the smallest fits
        if (ok) {
            ++fitted;
            bad += l.bytes > room || (full.bytes <= room && l.bytes != full.bytes);
            bad += l.rec_cap < std::min(full.rec_cap, 1u << 16) || l.pool_cap > full.pool_cap;
            // the parts lie one after the other
            bad += l.records + w.renders * (size_t)l.rec_cap * 16 > l.pool || l.pool + w.renders * (size_t)l.pool_cap * 16 > l.head ||
                   l.head + w.pixels * 32 > l.active || l.active + w.pixels * 4 > l.ctl ||
                   l.ctl + w.renders * sizeof(PathCtl) > l.used || l.used + w.renders * 8 > l.bytes;
        }
        none += !ok;
        const int first = tries;  // the same wish asks for no memory again, also where there was none
        bad += f.fit(w, reserve) != ok || tries != first;
        f.retry();
        bad += f.fit(w, reserve) != ok || (ok ? tries != first : tries == first);
        ListFit other;  // any other error: nothing is kept, the next call asks again
        bad += other.fit(w, [](size_t) { return cudaErrorStreamCaptureUnsupported; }) || other.fit(w, reserve) != ok;
        w.pixels += 1000;  // another wish does
        const int before = tries;
        f.fit(w, reserve);
        bad += tries == before;
    }
    std::printf("fitted %lld none %lld bad %lld\n", fitted, none, bad);
    return bad || !fitted || !none;
}

int main(int argc, char **argv) {
    if (argc != 4) return 2;
    if (!std::strcmp(argv[1], "exact")) return exact(atoll(argv[2]), atoi(argv[3]));
    if (!std::strcmp(argv[1], "storage")) return storage(atoll(argv[2]), atoi(argv[3]));
    if (!std::strcmp(argv[1], "pool")) return pool(atoll(argv[2]), atoi(argv[3]));
    if (!std::strcmp(argv[1], "flights")) return flights(atoll(argv[2]), atoi(argv[3]));
    FILE *f = std::fopen(argv[1], "rb");
    uint32_t head[2];
    if (!f || std::fread(head, 4, 2, f) != 2) return 2;
    std::vector<dr_node> N(head[0]);
    if (std::fread(N.data(), 64, head[0], f) != head[0]) return 2;
    std::fclose(f);
    std::vector<float> bricks((size_t)head[1] * 512, 0.f);
    const dr_scene_desc desc{N.data(), head[0], bricks.data(), head[1], 8, nullptr, 0};
    HostScene h;
    if (prepare_scene(&desc, h) != DR_OK) return 2;
    if (!h.glevels) {
        std::printf("no block grid\n");
        return 3;
    }
    DevScene S{};
    S.child = reinterpret_cast<const uint4 *>(h.child.data());
    S.leaf = h.leaf.data();
    S.gblock = h.gblock.data();
    S.gleaf = h.gleaf.data();
    S.glevels = h.glevels;
    for (int k = 0; k < 4; ++k) S.root_ce[k] = h.root_ce[k];
    std::vector<uint32_t> leaves;
    for (uint32_t i = 0; i < head[0]; ++i)
        if (h.leaf_flag[i]) leaves.push_back(i);
    std::mt19937_64 g(atoi(argv[3]));
    std::uniform_real_distribution<double> U(0, 1);
    std::normal_distribution<double> G;
    const double c[3] = {S.root_ce[0], S.root_ce[1], S.root_ce[2]}, e = S.root_ce[3], cell = 2 * e / (1 << h.glevels);
    static const double D[][3] = {{1, 1, 1}, {1, 1, .5}, {1, .5, .25}, {2, 1, 1e-7}, {1e-6, 1, 1}, {3, 2, 1},
                                  {1, 0, 0}, {0, 1, 1}, {1, 1, 0}, {.5, .25, 1}, {1, .75, .5}};
    long long bad = 0, slow = 0, ties = 0, hits = 0;
    for (long long i = 0; i < atoll(argv[2]); ++i) {
        double o[3], v[3] = {G(g), G(g), G(g)};
        const int kind = (int)(i % 8);
        const float4 L = h.leaf[2 * (size_t)leaves[g() % leaves.size()]];
        const double lc[3] = {L.x, L.y, L.z};
        const double n = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        const double far = (g() & 1) ? 2.5 : (g() & 1) ? 1e3 : 1e5;
        const uint64_t pick = g() % 11, half = g() & 1, back = g() & 1;
        for (int k = 0; k < 3; ++k) {
            const double lattice = c[k] - e + cell * (double)(g() % ((1u << h.glevels) + 3)) - cell;
            if (kind < 3) o[k] = lc[k] + (2 * U(g) - 1) * L.w;        // inside a leaf
            else if (kind == 3) o[k] = c[k] + (2 * U(g) - 1) * e * 1.2;  // in and around the root
            else if (kind == 4) o[k] = lattice;
            else if (kind == 5) {
                v[k] = D[pick][(k + i / 8) % 3] * ((g() & 1) ? 1 : -1);
                o[k] = lattice + (half ? cell * .5 : 0);
            } else if (kind == 6) o[k] = lc[k] - far * v[k] / n;      // aimed at a leaf from afar
            else {
                v[k] = (double)(g() % 9) - 4;
                if (k == 2 && v[0] == 0 && v[1] == 0 && v[2] == 0) v[2] = 1;
                o[k] = lattice;
            }
        }
        if (kind == 7 && back)
            for (int k = 0; k < 3; ++k) o[k] -= 1.5 * v[k];
        const double q = std::sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        float ro[3], rd[3];
        for (int k = 0; k < 3; ++k) {
            ro[k] = (float)o[k];
            rd[k] = (float)(kind == 7 && half ? v[k] : v[k] / q);
        }
        Count ca, cb;
        ca.zero();
        cb.zero();
        Trav T;
        uint32_t nstack[kMaxDepth];
        float iv[kMaxDepth][6];
        trav_init(T, S, ro, rd, ca);
        GridTrav Gt;
        float col[grid_words(kGridMaxLevels)];
        const uint32_t mode = grid_init<1>(Gt, S, col, ro, rd, cb);
        if (mode == 2) {
            ++slow;
            continue;
        }
        if ((mode == 0) != !T.active) {
            ++bad;
            continue;
        }
        if (mode == 0) continue;
        ++hits;
        for (;;) {
            uint32_t la = 0, lb = 0, r2;
            float a0 = 0, a1 = 0, b0 = 0, b1 = 0;
            const uint32_t r1 = trav_next_k(T, S, nstack, la, a0, a1, ca, 0xffffffffu, iv);
            long guard = 0;
            do {
                r2 = grid_next<1>(Gt, S, col, ro, rd, lb, b0, b1, cb, 1);
            } while (r2 == kTravMore && ++guard < 100000);
            bool same = r1 == r2 && ca.node_visits == cb.node_visits;
            if (same && r1 == kTravLeaf)
                same = __float_as_uint(h.leaf[2 * (size_t)la + 1].w) == lb && a0 == b0 &&
                       __float_as_uint(a1) == __float_as_uint(b1) &&
                       !std::memcmp(&h.gleaf[2 * (size_t)lb], &h.leaf[2 * (size_t)la], 32) &&
                       h.gmaj[lb] == h.leaf[2 * (size_t)la + 1].x;
            bad += !same;
            if (!same || r1 != kTravLeaf) break;
        }
        ties += Gt.loc >> 16;
    }
    std::printf("levels %u hits %lld ties %lld slow %lld bad %lld\n", h.glevels, hits, ties, slow, bad);
    return bad || hits == 0 || ties == 0;
}
