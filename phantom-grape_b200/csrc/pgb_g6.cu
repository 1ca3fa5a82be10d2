// pgb_g6.cu -- GRAPE-6 API of libpg6 on the B200 engine, plus the batched pgb6_* path.
//
// Drop-in for PG6/libpg6 (gp6util.h:1-101, phantom_g6.c, gravity.c).  Semantics kept:
//  * g6_set_j_particle stores (pos, vel, acc/2, jerk/6, mass, t, id) at address padr
//    (phantom_g6.c:118-125, gravity.c:95-115); the caller supplies acc/2 and jerk/6
//    (banana01.c:206-212).
//  * g6_set_ti sets the prediction time and a flag; the first g6calc_firsthalf after it
//    predicts all nj j-particles to t_i in FP64 (phantom_g6.c:138-164, gravity.c:149-193).
//  * g6calc_lasthalf* evaluate ni <= g6_npipes() i-particles against the nj predicted
//    j-particles, excluding the pair whose id equals the i id, and return
//    acc = sum m dx/r^3, jerk = sum m (dv/r^3 - 3 (dx.dv) dx/r^5), pot = -sum m/r
//    (the reference's -1/8 and 1/2 rescaling, phantom_g6.c:13-14, 200-208), nnb = id of the
//    nearest neighbour, rnnb = its softened distance (-2/key, gravity.c:651-657).
//  * lasthalfn / 2n / 2np also build neighbour lists (softened r <= h_i, gravity.c:788-793),
//    read back with g6_read_neighbour_list / g6_get_neighbour_list (phantom_g6.c:482-504),
//    lists in j-address order as the reference produces them.
//  * g6_set_tunit/xunit/reset/reset_fofpga/setup_njdata are no-ops, as in the reference.
// Deliberate differences:
//  * the self pair is excluded by an exact int id compare (the reference compares ids
//    converted to float, gravity.c:347-351: identical below 2^24 ids);
//  * pot is returned with FP64 precision (the reference stores it as float, avx_type.h:19);
//  * nearest-neighbour ties go to the smallest j address (the reference: lane j%4 first);
//  * a neighbour list longer than the capacity (1024, PGB_G6_NBMAX) is counted, flagged by
//    g6_read_neighbour_list and refused by g6_get_neighbour_list, never written out of bounds
//    (gravity.c:896-906 writes before it checks).
#include <atomic>
#include <chrono>

#include "pgb_g6_kernels.cuh"
#include "pgb_g6_small.cuh"
#include "pgb_hermite.cuh"

using namespace pgb;

namespace {

const char* LIB = "libpg6";
ErrorSlot g_err;

int env_int(const char* name, int dflt, int lo, int hi) {
    const char* s = std::getenv(name);
    if (!s || !*s) return dflt;
    int v = std::atoi(s);
    return v < lo ? lo : (v > hi ? hi : v);
}

int npipes() {
    static int v = env_int("PGB_G6_NPIPES", 48, 1, 1 << 20);
    return v;
}
int jmemsize() {
    static int v = env_int("PGB_G6_JMEMSIZE", 1 << 22, 1024, 1 << 26);
    return v;
}
// neighbour-list capacity per i-particle (the lists are sorted on the device in shared memory:
// at most 8192 entries)
int nbmax() {
    static int v = env_int("PGB_G6_NBMAX", 1024, 1, 1 << 13);
    return v;
}

std::mutex g_init_mu;
int g_device = -1;

bool ensure_device() {
    if (g_device >= 0) {
        PGB_CUDA_OR(g_err, LIB, cudaSetDevice(g_device), return false);
        return true;
    }
    std::lock_guard<std::mutex> g(g_init_mu);
    if (g_device < 0) {
        int n = 0;
        if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) {
            raise(g_err, LIB, PGB_ERR_NOGPU, "no CUDA device available");
            return false;
        }
        int d = env_int("PGB_DEVICE", 0, 0, n - 1);
        PGB_CUDA_OR(g_err, LIB, cudaSetDevice(d), return false);
        g_device = d;
    }
    PGB_CUDA_OR(g_err, LIB, cudaSetDevice(g_device), return false);
    return true;
}

// ------------------------------------------------------------------------------------------
// kernel configurations (cfg_kernel: threads per CTA, i per thread, j-lanes, form).  CFG_MED, CFG_128x1
// and CFG_*J have a j-paired form (1: g6_jpair, 2: stage-ordered g6_jquad2, 3: g6_jpair with the best
// j-quad kept) for double-float positions without neighbour lists.

enum Cfg {
    CFG_SMALL = 0, CFG_MED = 1, CFG_LARGE = 2, CFG_128x1 = 3, CFG_128x4 = 4, CFG_256x2 = 5,
    CFG_128x2J = 6, CFG_256x2J = 7, CFG_128x4J = 8, CFG_128x2JS = 9, NCFG = 10,
    // CFG_MED's form of one i per thread also where the j-paired one applies: a choice of the default rules
    // and the tuner, not settable and reported as CFG_MED, whose i-tile it has
    CFG_MED1 = NCFG
};
constexpr int ITILE_MAX = 512;

// One kernel of a configuration: a launch (info == nullptr), or what the host needs to know of it: its
// resident CTAs per SM, j records and i a tile, and forms.
struct KernelInfo {
    int occ = 0, tile = 0, itile = 0;
    bool paired = false;    // the j-paired form
    double task_j = 64.0;   // best_nch's
    double tail = 0.2;      // best_tile_chunk's (the stage-ordered form loses more with few CTAs on an SM:
                            // 65536 x 65536 in 8 chunks 4996 us, in 16 to 19 4664)
    bool resolve = false;   // leaves the nearest-neighbour lookups of split i-tiles to g6_resolve_kernel
};
template <int NT, int IPT, int JL, bool FF, bool NN, bool NBL, int JP>
void one_kernel(int grid, const G6Args& a, cudaStream_t s, KernelInfo* info) {
    auto k = g6_kernel<NT, IPT, JL, FF, NN, NBL, JP>;
    if (info) {
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k, NT, 0);
        info->occ = b > 0 ? b : 1;
        info->tile = g6_tile_j<NT, JL, g6_uses_jp<IPT, FF, NBL, JP>()>();
        info->itile = NT / JL * IPT;
        info->paired = g6_uses_jp<IPT, FF, NBL, JP>();
        info->task_j = NT == 512 ? 256.0 : 64.0;
        info->tail = JP == 2 ? 0.5 : 0.2;
        info->resolve = NN && !NBL && IPT % 2 == 0 && !g6_quad_min<IPT, FF, NBL, JP>();
        return;
    }
    k<<<grid, NT, 0, s>>>(a);
}

// CFG_MED: the j-paired form over two j-lanes (two i per thread) where it applies, else one i per
// thread over two lanes; the i-tile is the same.
template <bool FF, bool NN, bool NBL>
void med_kernel(int grid, const G6Args& a, cudaStream_t s, KernelInfo* info) {
    if constexpr (FF && !NBL) one_kernel<128, 2, 2, FF, NN, NBL, 3>(grid, a, s, info);
    else one_kernel<256, 1, 2, FF, NN, NBL, 0>(grid, a, s, info);
}

// CFG_128x1: the j-paired form of CFG_128x2J with the best j-quad kept (256 i a tile, no lookup
// kernel) where it applies, else one i per thread.
template <bool FF, bool NN, bool NBL>
void quad_kernel(int grid, const G6Args& a, cudaStream_t s, KernelInfo* info) {
    if constexpr (FF && !NBL) one_kernel<128, 2, 1, FF, NN, NBL, 3>(grid, a, s, info);
    else one_kernel<128, 1, 1, FF, NN, NBL, 0>(grid, a, s, info);
}

template <bool FF, bool NN, bool NBL>
void cfg_kernel(int cfg, int grid, const G6Args& a, cudaStream_t s, KernelInfo* info) {
    switch (cfg) {
        case CFG_SMALL: one_kernel<512, 1, 8, FF, NN, NBL, 0>(grid, a, s, info); break;
        case CFG_MED: med_kernel<FF, NN, NBL>(grid, a, s, info); break;
        case CFG_MED1: one_kernel<256, 1, 2, FF, NN, NBL, 0>(grid, a, s, info); break;
        case CFG_128x1: quad_kernel<FF, NN, NBL>(grid, a, s, info); break;
        case CFG_128x4: one_kernel<128, 4, 1, FF, NN, NBL, 0>(grid, a, s, info); break;
        case CFG_256x2: one_kernel<256, 2, 1, FF, NN, NBL, 0>(grid, a, s, info); break;
        case CFG_128x2J: one_kernel<128, 2, 1, FF, NN, NBL, 1>(grid, a, s, info); break;
        case CFG_256x2J: one_kernel<256, 2, 1, FF, NN, NBL, 1>(grid, a, s, info); break;
        case CFG_128x4J: one_kernel<128, 4, 1, FF, NN, NBL, 1>(grid, a, s, info); break;
        case CFG_128x2JS: one_kernel<128, 2, 1, FF, NN, NBL, 2>(grid, a, s, info); break;
        default: one_kernel<128, 2, 1, FF, NN, NBL, 0>(grid, a, s, info); break;
    }
}

void any_kernel(int cfg, bool ff, bool nn, bool nbl, int grid, const G6Args& a, cudaStream_t s, KernelInfo* info) {
    switch ((ff ? 4 : 0) | (nn ? 2 : 0) | (nbl ? 1 : 0)) {
        case 0: cfg_kernel<false, false, false>(cfg, grid, a, s, info); break;
        case 1: cfg_kernel<false, false, true>(cfg, grid, a, s, info); break;
        case 2: cfg_kernel<false, true, false>(cfg, grid, a, s, info); break;
        case 3: cfg_kernel<false, true, true>(cfg, grid, a, s, info); break;
        case 4: cfg_kernel<true, false, false>(cfg, grid, a, s, info); break;
        case 5: cfg_kernel<true, false, true>(cfg, grid, a, s, info); break;
        case 6: cfg_kernel<true, true, false>(cfg, grid, a, s, info); break;
        default: cfg_kernel<true, true, true>(cfg, grid, a, s, info); break;
    }
}

KernelInfo kernel_info(int cfg, bool ff, bool nn, bool nbl) {
    static std::mutex mu;
    static KernelInfo cache[NCFG + 1][8];
    std::lock_guard<std::mutex> g(mu);
    KernelInfo& v = cache[cfg][(ff ? 4 : 0) | (nn ? 2 : 0) | (nbl ? 1 : 0)];
    if (!v.occ) any_kernel(cfg, ff, nn, nbl, 0, G6Args{}, nullptr, &v);
    return v;
}
int occupancy(int cfg, bool ff, bool nn, bool nbl) { return kernel_info(cfg, ff, nn, nbl).occ; }
int reported_cfg(int cfg) { return cfg == CFG_MED1 ? (int)CFG_MED : cfg; }

cudaError_t launch_kernel(int cfg, bool ff, bool nn, bool nbl, int grid, const G6Args& a, cudaStream_t s) {
    any_kernel(cfg, ff, nn, nbl, grid, a, s, nullptr);
    return cudaGetLastError();
}

// Whether a force launch of this shape leaves nearest-neighbour lookups to g6_resolve_kernel (the
// kernel's tile-minimum search, split i-tiles (ngroups > 0), j addresses below the G6_NN_TILE
// mark: g6_task's `defer`).
bool needs_resolve(int cfg, bool ff, bool nn, bool nbl, int ngroups, int jn) {
    return nn && ngroups > 0 && jn < G6_NN_TILE && kernel_info(cfg, ff, nn, nbl).resolve;
}

// The deferred nearest-neighbour lookups of a force launch (after it, on the same stream).
cudaError_t launch_resolve(int cfg, bool ff, bool nn, bool nbl, int ngroups, const G6Args& a, cudaStream_t s) {
    if (!needs_resolve(cfg, ff, nn, nbl, ngroups, a.jn)) return cudaSuccess;
    constexpr int rpb = 128 / G6_RES_LANES;
    const long long grid = (long long)ngroups * ((a.itile + rpb - 1) / rpb);
    const int tile = kernel_info(cfg, ff, nn, nbl).tile;
    if (ff) g6_resolve_kernel<true><<<(unsigned)grid, 128, 0, s>>>(a, ngroups, tile);
    else g6_resolve_kernel<false><<<(unsigned)grid, 128, 0, s>>>(a, ngroups, tile);
    return cudaGetLastError();
}

// The small-call cluster kernel (pgb_g6_small.cuh): i-slots x j-lanes by the call's i count.
struct SmallShape {
    int isl, jl;
};
inline SmallShape small_shape(int ni) {
    if (ni <= 16) return {16, 32};
    if (ni <= 32) return {32, 16};
    if (ni <= 48) return {48, 10};
    return {64, 8};
}
// CTAs per cluster: 71 co-resident clusters of 4 (284 CTAs) leave 12 of the 148 SMs with one
// CTA, where the 33 clusters of 8 left 32 (the others, with two, set the call's time): the
// 48 x 65536 call 27.2 -> 26.6 us, 48 x 16384 23.0 -> 19.7 us
constexpr int SMALL_CL = 4;
constexpr int SMALL_WORDS = sizeof(G6Out) / 4;   // host words of a result

template <int ISL, int JL, bool FF, bool NN, bool NBL>
cudaError_t small_launch(int grid, int cl, const G6SmallArgs& a, const G6I* irec, cudaStream_t s,
                         int* max_clusters) {
    auto kern = g6_small_kernel<ISL, JL, FF, NN, NBL>;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(ISL * JL);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (max_clusters) return cudaOccupancyMaxActiveClusters(max_clusters, (void*)kern, &cfg);
    G6IBlock<ISL> ib;
    std::memcpy(ib.rec, irec, (size_t)a.ni * sizeof(G6I));
    return cudaLaunchKernelEx(&cfg, kern, a, ib);
}

template <int ISL, int JL, bool FF>
cudaError_t small_launch_nn(bool nn, bool nbl, int grid, int cl, const G6SmallArgs& a,
                            const G6I* irec, cudaStream_t s, int* mc) {
    if (nn && nbl) return small_launch<ISL, JL, FF, true, true>(grid, cl, a, irec, s, mc);
    if (nn) return small_launch<ISL, JL, FF, true, false>(grid, cl, a, irec, s, mc);
    if (nbl) return small_launch<ISL, JL, FF, false, true>(grid, cl, a, irec, s, mc);
    return small_launch<ISL, JL, FF, false, false>(grid, cl, a, irec, s, mc);
}

template <bool FF>
cudaError_t small_launch_ff(SmallShape sh, bool nn, bool nbl, int grid, int cl, const G6SmallArgs& a,
                            const G6I* irec, cudaStream_t s, int* mc) {
    if (sh.isl == 16) return small_launch_nn<16, 32, FF>(nn, nbl, grid, cl, a, irec, s, mc);
    if (sh.isl == 32) return small_launch_nn<32, 16, FF>(nn, nbl, grid, cl, a, irec, s, mc);
    if (sh.isl == 48) return small_launch_nn<48, 10, FF>(nn, nbl, grid, cl, a, irec, s, mc);
    return small_launch_nn<64, 8, FF>(nn, nbl, grid, cl, a, irec, s, mc);
}

// Launch (mc == nullptr) or query the co-resident clusters of cl CTAs (into *mc).
cudaError_t small_kernel(SmallShape sh, bool ff, bool nn, bool nbl, int grid, int cl, const G6SmallArgs& a,
                         const G6I* irec, cudaStream_t s, int* mc) {
    return ff ? small_launch_ff<true>(sh, nn, nbl, grid, cl, a, irec, s, mc)
              : small_launch_ff<false>(sh, nn, nbl, grid, cl, a, irec, s, mc);
}

// Chunks (= CTAs, all co-resident) and cluster size of a small call over nj j-records: at least
// 128 j per chunk, at most the co-resident clusters' CTAs (queried once per kernel variant).
void small_grid(SmallShape sh, bool ff, bool nn, bool nbl, int nj, int& grid, int& cl) {
    static int cache[4][2][2][2] = {};
    const int v = sh.isl / 16 - 1;
    int& mc = cache[v][ff][nn][nbl];
    if (!mc) {
        G6SmallArgs a{};
        int n = 0;
        if (small_kernel(sh, ff, nn, nbl, SMALL_CL, SMALL_CL, a, nullptr, nullptr, &n) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = sm_count(g_device) / SMALL_CL;
        }
        mc = n;
    }
    static const int forced = env_int("PGB_G6_SMALL_CTAS", 0, 0, 1 << 16);
    int by_j = nj / 128;
    int want = mc * SMALL_CL;
    if (forced) want = std::min(want, forced);
    want = std::min(want, by_j);
    if (want < 1) want = 1;
    cl = 1;
    while (cl < SMALL_CL && cl * 2 <= want) cl *= 2;
    grid = want / cl * cl;
    if (grid == SMALL_CL_MAX) cl = grid;   // one cluster: no rows of partial sums in memory
}

// Relative-coordinate arithmetic of the library's own calls: double-float (default) or FP64
// subtraction + conversion (PGB_G6_DX=f64), see rel1() in pgb_g6_kernels.cuh.
bool dx_ff() {
    static int v = -1;
    if (v < 0) {
        const char* e = std::getenv("PGB_G6_DX");
        v = (e && std::strcmp(e, "f64") == 0) ? 0 : 1;
    }
    return v == 1;
}

// The default configuration (PGB_G6_CFG forces one for sweeps) of a call or plan of one item of ni i
// against nj j.  With double-float positions and no neighbour lists: SMALL (512 threads, 8 j-lanes)
// while the launch's latency counts more than its pairs, MED (j-paired, 128 i a tile, two j-lanes)
// for the middle, the stage-ordered j-paired form for the largest.  Measured (us, SMALL / MED / JS, and
// the scalar two-i form that was the default from 4097 i up):
//   777 x 4096     14.6 /   22.8 /   41    777 x 65536    98.6 /  102   /  127
//   2086 x 2134    17.4 /   23.1 /   -     3000 x 4096    29.3 /   33.4 /   51
//   1500 x 16384   49.9 /   51.5 /   70    2086 x 16384   70.2 /   64.4 /   82
//   4096 x 16384  140   /  101   /  121    8192 x 16384  244   /  177   /  198   (220)
//   8192 x 65536  876   /  646   /  632 (749)   16384 x 16384  458 / 329 / 344 (399)
//   16384 x 65536  1718 / 1260 / 1208 (1457)    65536 x 65536  6754 / 4890 / 4664 (5488)
// Few j: the scalar forms, whose tasks start and end sooner, up to 4096 i against 256 j (CFG_MED1 / MED: 4096 x
// 32 6.4 / 8.4, x 200 12.5 / 15.0) and for the most i against the fewest j (LARGE / MED: 131072 x 4 10.5 / 15.3,
// x 32 20 / 19; without neighbours 65536 x 64 12.5 / 14.6).
int pick_cfg(long long ni, long long nj, bool ff, bool nn, bool nbl) {
    static int forced = env_int("PGB_G6_CFG", -1, -1, NCFG - 1);
    if (forced >= 0) return forced;
    if (ff && !nbl) {
        if (ni <= 3072 && ni * nj <= (ni <= 1024 ? 48LL << 20 : 24LL << 20)) return CFG_SMALL;
        if (ni <= 4096 && nj <= 256) return CFG_MED1;
        if (ni >= 32768 && nj <= (nn ? 16 : 64)) return CFG_LARGE;
        return ni * nj < (1LL << 29) ? CFG_MED : CFG_128x2JS;
    }
    if (ni <= 64) return CFG_SMALL;
    if (ni <= 4096) return CFG_MED;
    return CFG_LARGE;
}

// The same for a batch of several items.
//  * Short work, up to 2^20 pairs of SMALL's 64-i tiles (at least 128 j): SMALL (us, SMALL / MED: 4 items of 16 i x
//    4096 j 12.5 / 14.6, 64 of 100 x 128 8.4 / 9.5).
//  * Items of at most 64 i, whose tiles of 128 MED leaves half empty: SMALL where its tasks, one wave of a
//    few long ones, fill the GPU, that is for many items of many j (256 of 1 i x 1024 j 37 / 55, 64 of 4 x 4096
//    50 / 59, 96 of 1 x 1024 27 / 29) and for two to four (2 of 48 x 65536 39 / 48, 2 of 64 x 16384 20.7 / 22.8, 4 of 64 x
//    65536 64 / 69); else MED (8 of 8 x 65536 115 / 99, 2 of 32 x 16384 20.7 / 18.7, 32 of 8 x 1024 18.6 / 14.6, 1024 of 4 x
//    128 37 / 28).
//  * Middle work of up to 32 tiles: MED1, whose threads have one i where MED's have two (4 items of 128 x 4096
//    17.6 / 23.8, 2 of 100 x 16384 24.8 / 29.2, 16 of 128 x 1024 14.4 / 16.6); from 2^25 pairs on MED (4 of 100 x 65536 84 / 79).
//  * Then by the i count that the average pair sees: MED's smaller i-tiles up to 6000, above that
//    CFG_128x1's j-paired form (us, MED / 128x1 / the scalar form that was the default: 40 clusters of
//    300 to 5000 particles 220 / 234 / 327, 96 of 64 to 2048 110 / 122 / 192, 96 of 256 to 16384 4352 / 4227 / 5136).
int pick_batch_cfg(int nitem, const int* items, bool ff, bool nn) {
    double w = 0.0, wi = 0.0;
    long long nimax = 0, njmax = 0, total_i = 0, tiles = 0, pairs64 = 0, pairs128 = 0;
    for (int k = 0; k < nitem; k++) {
        const long long ni = items[4 * k + 1], nj = items[4 * k + 3];
        nimax = std::max(nimax, ni);
        njmax = std::max(njmax, nj);
        total_i += ni;
        tiles += (ni + 127) / 128;
        pairs64 += (ni + 63) / 64 * 64 * nj;
        pairs128 += (ni + 127) / 128 * 128 * nj;
        w += (double)ni * (double)nj;
        wi += (double)ni * (double)nj * (double)ni;
    }
    if (nitem == 1) return pick_cfg(nimax, njmax, ff, nn, false);
    if (!ff) return pick_cfg(std::max(nimax, total_i / 4), njmax, ff, nn, false);
    static int forced = env_int("PGB_G6_CFG", -1, -1, NCFG - 1);
    if (forced >= 0) return forced;
    if (pairs64 <= (1 << 20) && njmax >= 128) return CFG_SMALL;
    if (nimax <= 64) {
        const bool many = nitem >= 48 && njmax >= 512 && pairs64 >= (5 << 20);
        const bool few = (nitem <= 4 && nimax > 32) || (nitem <= 3 && njmax > 32768);
        return many || few ? CFG_SMALL : CFG_MED;
    }
    if (tiles <= 32 && pairs128 < (1 << 25)) return CFG_MED1;
    return wi <= 6000.0 * w ? CFG_MED : CFG_128x1;
}

// The chunk length of a single item: the j-paired kernels' whole tiles, else the wave model's.
long long model_chunk(const KernelInfo& K, long long itiles, int nj, int slots, int maxch) {
    if (K.paired) return best_tile_chunk(itiles, nj, sm_count(g_device), K.tile, maxch, K.tail);
    const int nch = best_nch(itiles, nj, slots, maxch, K.task_j);
    return (nj + nch - 1) / nch;
}

// Plan one batch of items ([k][4] = i_off, i_cnt, j_off, j_cnt) for a configuration:
// about 4 tasks per resident CTA, chunks of at least 128 j, at most 512 chunks per i-tile
// (their partial rows are summed by the cooperative reduction of the group's last CTA).
long long plan_items(std::vector<Task>& tasks, std::vector<Group>& groups, int& rows, int nitem, const int* items,
                     int cfg, bool ff, bool nn, bool nbl, int nch_fixed = 0) {
    const KernelInfo K = kernel_info(cfg, ff, nn, nbl);
    int slots = sm_count(g_device) * K.occ;
    int itile = K.itile;
    long long work = 0;
    for (int k = 0; k < nitem; k++) {
        long long ni = items[4 * k + 1];
        long long tiles = (ni + itile - 1) / itile;
        work += tiles * itile * (long long)items[4 * k + 3];
    }
    // about 4 tasks per resident CTA for load balance of uneven items; a single item (equal
    // tasks) or a small call (the drop-in API's npipes-sized calls) instead gets one wave of one
    // fat task per resident CTA, which keeps the number of partial rows (the reduction depth) low
    long long per_task = (cfg == CFG_SMALL || nitem == 1) ? work / slots + 1 : work / (4LL * slots) + 1;
    long long inter = 0;
    rows = 0;
    static const long long maxch = env_int("PGB_G6_MAXCHUNKS", 512, 1, 4096);
    for (int k = 0; k < nitem; k++) {
        int ni = items[4 * k + 1], nj = items[4 * k + 3];
        long long jc;
        int align = K.paired ? K.tile : 1;
        if (nitem == 1) {
            // one item of equal tasks: the chunk count that minimises the wave quantisation, or
            // the autotuner's (nch_fixed)
            long long itiles = (ni + itile - 1) / itile;
            static const int forced_nch = env_int("PGB_G6_NCH", 0, 0, 4096);   // profiling: a pinned count
            const int nch = forced_nch > 0 ? forced_nch : (nch_fixed < 0 ? -nch_fixed : nch_fixed);
            if (nch_fixed < 0) align = 1;
            if (nch > 0) jc = (nj + nch - 1) / nch;
            else jc = model_chunk(K, itiles, nj, slots, (int)maxch);
        } else {
            jc = per_task / itile;
            if (jc < 128) jc = 128;
            if (jc * maxch < nj) jc = (nj + maxch - 1) / maxch;
        }
        if (jc > nj) jc = nj;
        if (jc < 1) jc = 1;   // no j-records: one empty task
        rows += plan_item(tasks, groups, items[4 * k], ni, items[4 * k + 2], nj, itile, (int)jc, rows,
                          align);
        inter += (long long)ni * nj;
    }
    std::stable_sort(tasks.begin(), tasks.end(), [](const Task& a, const Task& b) {
        return (long long)a.ni * a.nj > (long long)b.ni * b.nj;
    });
    return inter;
}

// The chunk counts the autotuner tries for a single item besides the wave model's choice m:
// m x 3/4, 5/4, 3/2, and the counts whose chunks are whole 128-record j-tiles (nj / nch a
// multiple of 128) between m/2 and 2m.  Measured on the largest Hermite calls, the time moves
// by up to 5 % from one count to the next (the persistent CTAs' last wave; counts whose chunks
// are whole tiles were within 1 % of the best and never bimodal), which the model cannot predict.
std::vector<int> chunk_candidates(int m, int nj, int maxch) {
    std::vector<int> c;
    auto add = [&](long long v) {
        const long long hi = std::max<long long>(1, std::min<long long>(maxch, nj / 128));
        v = std::max<long long>(1, std::min<long long>(v, hi));
        if (std::find(c.begin(), c.end(), (int)v) == c.end()) c.push_back((int)v);
    };
    add(m);
    add((3LL * m + 2) / 4);
    add((5LL * m + 2) / 4);
    add((3LL * m + 1) / 2);
    for (long long n = std::max(1, m / 2); n <= 2LL * m; n++)
        if (nj % n == 0 && (nj / n) % 128 == 0) add(n);
    return c;
}

// ------------------------------------------------------------------------------------------
// library state (the reference keeps one global j-memory, gravity.c:31-47)

struct State {
    std::mutex mu;
    bool ready = false;
    cudaStream_t stream = nullptr;
    HostBuf<G6Ptcl> jh;
    DevBuf<G6Ptcl> jd;
    DevBuf<G6PredJ> pred;
    int jcap = 0, jdirty_lo = 1 << 30, jdirty_hi = 0;
    // sparse updates (a block step re-sends only its active particles): dirty addresses
    std::vector<int> dirty;
    std::vector<unsigned char> dirty_flag;
    bool all_dirty = true;
    HostBuf<G6Ptcl> sbuf;   // mapped: packed dirty records
    HostBuf<int> sidx;      // mapped: their addresses
    // the stream may still read jh, sbuf or sidx (g6calc_firsthalf does not wait for its upload)
    bool uploading = false;
    G6Ptcl* sbuf_dev = nullptr;
    int* sidx_dev = nullptr;
    double ti = 0.0;
    int predict_flag = 0;
    HostBuf<G6I> ibuf;
    HostBuf<G6Out> outh;    // mapped: the kernel writes the final results into it
    G6Out* outh_dev = nullptr;            // its device address (looked up once per allocation)
    const G6Out* outh_seen = nullptr;     // the allocation outh_dev belongs to
    DevBuf<int> pcnt;       // self-resetting counters of the parameter-block launches
    DevBuf<G6Out> spart;    // cluster rows of the small-call kernel
    HostBuf<uint2> words;     // mapped: the small-call kernel's results, (value, call number) words
    uint4* words_dev = nullptr;
    unsigned seq = 0;         // number of the last small call
    bool wait_words = false;  // the call's results come in `words` (else in outh, after the stream)
    HostBuf<uint2> nbw;       // mapped: its neighbour lists, [ni][nbmax + 1] of (value, call number)
    uint2* nbw_dev = nullptr;
    bool nbc_zero = false;    // the list counts nbc_d are zero
    Stager<G6I, G6Out> st;
    // neighbour lists of the last lasthalf*n call
    DevBuf<int> nbc_d, nbl_d;
    HostBuf<int> nbc_h, nbl_h;
    std::vector<int> nbids;   // one after another, list i from nboff[i]
    std::vector<size_t> nboff;
    std::vector<int> nbcounts;
    // device-time accounting of the drop-in calls (pgb6_set_call_timing): CUDA events around the
    // j-update + prediction of g6calc_firsthalf and the force launch of g6calc_lasthalf*
    bool time_calls = false;
    cudaEvent_t tev[2] = {nullptr, nullptr};
    double dev_ms = 0.0;
    int nb_ni = 0, nb_error = 0;
};
State S;

bool init_state() {
    if (!ensure_device()) return false;
    if (!S.ready) {
        PGB_CUDA_OR(g_err, LIB, cudaStreamCreateWithFlags(&S.stream, cudaStreamNonBlocking), return false);
        S.ready = true;
    }
    return true;
}

// Before the host changes what an upload reads.
bool wait_upload() {
    if (!S.uploading) return true;
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(S.stream), return false);
    S.uploading = false;
    return true;
}

bool grow_j(int need) {
    if (need > jmemsize()) {
        raise(g_err, LIB, PGB_ERR_CAPACITY, "j-memory overflow: address %d >= jmemsize %d", need - 1, jmemsize());
        return false;
    }
    if (need <= S.jcap) return true;
    int cap = S.jcap ? S.jcap : 8192;
    while (cap < need) cap *= 2;
    if (cap > jmemsize()) cap = jmemsize();
    if (!wait_upload()) return false;
    PGB_CUDA_OR(g_err, LIB, S.jh.reserve(cap, true), return false);
    std::memset((void*)(S.jh.p + S.jcap), 0, (size_t)(cap - S.jcap) * sizeof(G6Ptcl));
    S.dirty_flag.resize(cap, 0);
    S.all_dirty = true;  // new device buffer: upload everything
    S.jdirty_lo = 0;
    S.jdirty_hi = cap;
    S.jcap = cap;
    return true;
}

void mark_dirty(int padr) {
    if (padr < S.jdirty_lo) S.jdirty_lo = padr;
    if (padr + 1 > S.jdirty_hi) S.jdirty_hi = padr + 1;
    if (!S.all_dirty && !S.dirty_flag[padr]) {
        S.dirty_flag[padr] = 1;
        S.dirty.push_back(padr);
    }
}

// Room for `want` items in a mapped buffer, and its device address (looked up when it is allocated).
template <class T, class D>
bool reserve_mapped(HostBuf<T>& b, size_t want, D*& dev) {
    const T* old = b.p;
    PGB_CUDA_OR(g_err, LIB, b.reserve(want, false, cudaHostAllocPortable | cudaHostAllocMapped), return false);
    if (b.p != old || !dev) {
        dev = nullptr;
        PGB_CUDA_OR(g_err, LIB, cudaHostGetDevicePointer((void**)&dev, b.p, 0), return false);
    }
    return true;
}

// Upload the j-memory changes and predict j-records [0, nj) to the set time: the contiguous dirty
// range by a copy, or, when the changed records are sparse in it (a block step's active set), only
// those, which the device reads from mapped host memory -- up to G6_UPD_MAX in the prediction's
// own launch, more by a scatter before it (its address list would make the launch's parameters grow;
// two copies and a scatter instead: 47 against 36 us a call of 7 i with 7 of 1024 records sent).
bool launch_update(int nj) {
    PGB_CUDA_OR(g_err, LIB, S.pred.reserve(S.jcap), return false);
    const bool dirty = S.jdirty_hi > S.jdirty_lo;
    const size_t n = S.dirty.size();
    const bool sparse = dirty && !S.all_dirty && n * 4 < (size_t)(S.jdirty_hi - S.jdirty_lo);
    const bool fused = sparse && n <= (size_t)G6_UPD_MAX;
    G6Ptcl* rec_d = nullptr;
    if (dirty) {
        PGB_CUDA_OR(g_err, LIB, S.jd.reserve(S.jcap), return false);
        if (!wait_upload()) return false;
        S.uploading = true;
    }
    if (sparse) {
        if (!reserve_mapped(S.sbuf, n, S.sbuf_dev)) return false;
        rec_d = S.sbuf_dev;
        for (size_t k = 0; k < n; k++) S.sbuf.p[k] = S.jh.p[S.dirty[k]];
    }
    if (fused) {
        G6Update U;
        U.rec = rec_d;
        U.n = (int)n;
        std::memcpy(U.idx, S.dirty.data(), n * sizeof(int));
        const int top = std::max(nj, S.jdirty_hi);
        g6_update_predict_kernel<<<(top + 255) / 256, 256, 0, S.stream>>>(S.jd.p, S.jcap, U, nj, S.ti, S.pred.p,
                                                                          dx_ff());
    } else {
        if (sparse) {
            if (!reserve_mapped(S.sidx, n, S.sidx_dev)) return false;
            std::memcpy(S.sidx.p, S.dirty.data(), n * sizeof(int));
            g6_scatter_kernel<<<(int)((n + 255) / 256), 256, 0, S.stream>>>(rec_d, S.sidx_dev, (int)n, S.jcap, S.jd.p);
            PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return false);
        } else if (dirty) {
            const size_t lo = S.jdirty_lo, range = (size_t)(S.jdirty_hi - S.jdirty_lo);
            PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(S.jd.p + lo, S.jh.p + lo, range * sizeof(G6Ptcl),
                                                    cudaMemcpyHostToDevice, S.stream), return false);
        }
        g6_predict_kernel<<<(nj + 255) / 256, 256, 0, S.stream>>>(S.jd.p, nj, S.ti, S.pred.p, dx_ff());
    }
    PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return false);
    if (dirty) {
        for (int a : S.dirty) S.dirty_flag[a] = 0;
        S.dirty.clear();
        S.all_dirty = false;
        S.jdirty_lo = 1 << 30;
        S.jdirty_hi = 0;
    }
    return true;
}

// Call timing: start / stop marks on the library's stream; stop adds the device time between
// them once the stop mark has completed.
bool time_mark(int k) {
    if (!S.time_calls) return true;
    if (!S.tev[k]) PGB_CUDA_OR(g_err, LIB, cudaEventCreate(&S.tev[k]), return false);
    PGB_CUDA_OR(g_err, LIB, cudaEventRecord(S.tev[k], S.stream), return false);
    return true;
}

bool time_add() {
    if (!S.time_calls) return true;
    float ms = 0.f;
    PGB_CUDA_OR(g_err, LIB, cudaEventSynchronize(S.tev[1]), return false);
    PGB_CUDA_OR(g_err, LIB, cudaEventElapsedTime(&ms, S.tev[0], S.tev[1]), return false);
    S.dev_ms += ms;
    return true;
}

// The upload and prediction of g6calc_firsthalf, left running: g6calc_lasthalf* follows on the same
// stream and waits for both, and what would change the upload's source waits first (wait_upload).  Waiting
// here cost the call of 48 i against 65536 j 42 -> 31.5 us.  (The prediction inside the force kernel
// instead of its own launch is no faster: it then starts with the force, not while the host prepares it.)
bool flush_and_predict(int nj) {
    if (nj <= 0) return true;
    if (!grow_j(nj) || !time_mark(0) || !launch_update(nj) || !time_mark(1)) return false;
    return time_add();
}

// Shared memory of g6_nb_sort_kernel: the power of two at or above nbmax entries.
size_t nb_sort_smem() {
    size_t p = 1;
    while (p < (size_t)nbmax()) p <<= 1;
    return p * sizeof(int);
}

// The small-call path: one launch of the cluster kernel (i-records in its parameter block) and, with
// neighbour lists, one that sorts them; results and lists come as words in mapped buffers, which the
// host takes as they arrive (33 i against 20011 j with lists: 114 -> 61 us, 27 of them the caller's reading
// of the lists).
bool run_small(int nj, int ni, float eps2, bool nn, bool nbl) {
    const bool ff = dx_ff();
    const SmallShape sh = small_shape(ni);
    int grid = 1, cl = 1;
    small_grid(sh, ff, nn, nbl, nj, grid, cl);
    PGB_CUDA_OR(g_err, LIB, S.spart.reserve((size_t)(grid / cl) * sh.isl), return false);
    if (!S.pcnt.p) {
        PGB_CUDA_OR(g_err, LIB, S.pcnt.reserve(SMALL_CL), return false);
        PGB_CUDA_OR(g_err, LIB, S.pcnt.zero_fill(S.stream), return false);
    }
    G6SmallArgs a;
    a.jpred = S.pred.p;
    a.eps2 = eps2;
    a.ni = ni;
    a.nj = nj;
    a.partial = S.spart.p;
    a.counter = S.pcnt.p;
    a.nb_count = nullptr;
    a.nb_list = nullptr;
    a.nb_maxlen = nbmax();
    if (nbl) {
        if (!S.nbc_zero || !S.nbc_d.p) {
            PGB_CUDA_OR(g_err, LIB, S.nbc_d.reserve(G6_SMALL_MAXI), return false);
            PGB_CUDA_OR(g_err, LIB, cudaMemsetAsync(S.nbc_d.p, 0, G6_SMALL_MAXI * sizeof(int), S.stream), return false);
        }
        PGB_CUDA_OR(g_err, LIB, S.nbl_d.reserve((size_t)ni * nbmax()), return false);
        a.nb_count = S.nbc_d.p;
        a.nb_list = S.nbl_d.p;
    }
    // no word of the buffers carries the number of a call to come: they start with the number of a call
    // that is over, and are cleared when the numbers start again
    const size_t nword = SMALL_WORDS * G6_SMALL_MAXI, nnb = (size_t)G6_SMALL_MAXI * (nbmax() + 1);
    const bool fresh = !S.words.p, fresh_nb = nbl && !S.nbw.p;
    if (!reserve_mapped(S.words, nword, S.words_dev)) return false;
    if (nbl && !reserve_mapped(S.nbw, nnb, S.nbw_dev)) return false;
    const bool wrap = ++S.seq == 0;
    if (wrap) S.seq = 1;
    if (fresh || wrap) std::memset((void*)S.words.p, 0, sizeof(uint2) * nword);
    if (fresh_nb || (wrap && S.nbw.p)) std::memset((void*)S.nbw.p, 0, sizeof(uint2) * nnb);
    a.words = S.words_dev;
    a.seq = S.seq;
    S.wait_words = true;
    PGB_CUDA_OR(g_err, LIB, small_kernel(sh, ff, nn, nbl, grid, cl, a, S.ibuf.p, S.stream, nullptr), return false);
    if (nbl) {
        S.nbc_zero = false;
        g6_nb_sort_kernel<<<ni, 256, nb_sort_smem(), S.stream>>>(S.nbc_d.p, S.nbl_d.p, nbmax(), S.jd.p, S.nbw_dev,
                                                                S.seq);
        PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return false);
        S.nbc_zero = true;
    }
    return true;
}

// Words of a small call as they arrive: take() returns true when it has them all.  A bounded spin, then
// the stream synchronisation that reports a failed launch.
template <class Take>
bool take_words(Take take) {
    auto t0 = std::chrono::steady_clock::now();
    for (long it = 0;; it++) {
        if (take()) return true;
        if ((it & 1023) == 1023 && std::chrono::steady_clock::now() - t0 > std::chrono::seconds(5)) break;
    }
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(S.stream), return false);
    if (take()) return true;
    raise(g_err, LIB, PGB_ERR_DEVICE, "a call's results did not arrive");
    return false;
}
// Word w's value into v when it carries call number seq.
template <class T>
bool take_word(const uint2* w, unsigned seq, T& v) {
    const unsigned long long x = *(const volatile unsigned long long*)w;
    if ((unsigned)(x >> 32) != seq) return false;
    v = (T)(unsigned)x;
    return true;
}

// Wait for the results of the last call in S.outh: word by word when the call sends words, else the
// stream.
bool wait_results(int ni) {
    if (!S.wait_words) {
        PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(S.stream), return false);
        return true;
    }
    unsigned* out = (unsigned*)S.outh.p;
    const int n = SMALL_WORDS * ni;
    int k = 0;
    return take_words([&] {
        while (k < n && take_word(S.words.p + k, S.seq, out[k])) k++;
        return k == n;
    });
}

// One drop-in API call: ni i-particles (in S.ibuf) against j-records [0, nj), results into
// the mapped pinned buffer S.outh (the kernel writes them there: no device-to-host copy).
// Up to G6_SMALL_MAXI i-particles (the reference's 48 pipes): the small-call cluster kernel, one
// launch.  More (PGB_G6_NPIPES > 64): the general kernel in regular mode -- it derives its i-tile
// x j-chunk tasks from the shape, so only the i-records are uploaded, and its task counter
// resets itself.
bool run_force(int nj, int ni, float eps2, bool nn, bool nbl) {
    PGB_CUDA_OR(g_err, LIB, S.outh.reserve(ni, false, cudaHostAllocPortable | cudaHostAllocMapped), return false);
    if (S.outh_seen != S.outh.p) {
        PGB_CUDA_OR(g_err, LIB, cudaHostGetDevicePointer((void**)&S.outh_dev, S.outh.p, 0), return false);
        S.outh_seen = S.outh.p;
    }
    if (ni <= G6_SMALL_MAXI && nj > 0) return run_small(nj, ni, eps2, nn, nbl);
    const bool ff = dx_ff();
    const int cfg = pick_cfg(ni, nj, ff, nn, nbl);
    const KernelInfo K = kernel_info(cfg, ff, nn, nbl);
    const int itile = K.itile;
    const int slots = sm_count(g_device) * K.occ;
    static const int maxch = env_int("PGB_G6_MAXCHUNKS", 512, 1, 4096);
    const int itiles = (ni + itile - 1) / itile;
    int nch = best_nch(itiles, nj, slots, maxch, K.paired ? 256.0 : K.task_j);
    if (nch > nj) nch = nj > 0 ? nj : 1;
    const int rows = nch > 1 ? itiles * nch : 0;
    static const std::vector<Task> no_tasks;
    static const std::vector<Group> no_groups;
    PGB_CUDA_OR(g_err, LIB, S.st.stage(S.stream, no_tasks, no_groups, rows, ITILE_MAX, S.ibuf.p, ni, (size_t)itiles),
                return false);
    G6Args a;
    a.ipart = S.st.irecs();
    a.jpred = S.pred.p;
    a.eps2 = eps2;
    a.tasks = nullptr;
    a.ntasks = itiles * nch;
    a.task_counter = S.st.counter();
    a.groups = nullptr;
    a.group_counters = S.st.dgcnt.p;
    a.partial = S.st.dpart.p;
    a.out = S.outh_dev;
    a.itile = itile;
    a.bundle_counters = S.st.bundle_counters();
    a.nb_count = nullptr;
    a.nb_list = nullptr;
    a.nb_maxlen = nbmax();
    a.reg_ni = ni;
    a.reg_nj = nj;
    a.reg_nch = nch;
    a.jn = nj;
    if (nbl) {
        S.nbc_zero = false;
        PGB_CUDA_OR(g_err, LIB, S.nbc_d.reserve(ni), return false);
        PGB_CUDA_OR(g_err, LIB, S.nbl_d.reserve((size_t)ni * nbmax()), return false);
        PGB_CUDA_OR(g_err, LIB, cudaMemsetAsync(S.nbc_d.p, 0, (size_t)ni * sizeof(int), S.stream), return false);
        a.nb_count = S.nbc_d.p;
        a.nb_list = S.nbl_d.p;
    }
    if (a.ntasks == 0) return true;
    const int grid = a.ntasks < slots ? a.ntasks : slots;
    PGB_CUDA_OR(g_err, LIB, launch_kernel(cfg, ff, nn, nbl, grid, a, S.stream), return false);
    PGB_CUDA_OR(g_err, LIB, launch_resolve(cfg, ff, nn, nbl, nch > 1 ? itiles : 0, a, S.stream), return false);
    return true;
}

// Counts + lists back to the host; each list is sorted by j address (the reference's order,
// gravity.c:888-900) and mapped to particle ids on the device (g6_nb_sort_kernel).  Lists longer than
// the capacity keep only their count and set the overflow flag.
void nblist_collect(int ni) {
    S.nb_ni = ni;
    S.nb_error = 0;
    S.nbcounts.assign(ni, 0);
    const int cap = nbmax();
    S.nbids.clear();
    S.nboff.assign(ni, 0);
    auto add_list = [](int i, int count, int stored) {
        S.nbcounts[i] = count;
        S.nboff[i] = S.nbids.size();
        S.nbids.resize(S.nbids.size() + stored);
        return S.nbids.data() + S.nboff[i];
    };
    if (S.wait_words) {
        int i = 0, k = 0, c = -1;   // row, entry, entries (-1: not known yet)
        int* list = nullptr;
        const bool ok = take_words([&] {
            for (; i < ni; i++, c = -1) {
                const uint2* row = S.nbw.p + (size_t)i * (cap + 1);
                if (c < 0) {
                    int count;
                    if (!take_word(row, S.seq, count)) return false;
                    c = count > cap ? 0 : count;
                    list = add_list(i, count, c);
                    k = 0;
                }
                while (k < c && take_word(row + 1 + k, S.seq, list[k])) k++;
                if (k < c) return false;
            }
            return true;
        });
        if (!ok) S.nbcounts.assign(ni, 0);
    } else {
        if (ni > 0) {
            g6_nb_sort_kernel<<<ni, 256, nb_sort_smem(), S.stream>>>(S.nbc_d.p, S.nbl_d.p, cap, S.jd.p, nullptr, 0);
            PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return);
        }
        if (S.nbc_h.reserve(ni) != cudaSuccess || S.nbl_h.reserve((size_t)ni * cap) != cudaSuccess) {
            raise(g_err, LIB, PGB_ERR_CUDA, "pinned neighbour-list buffer allocation failed");
            return;
        }
        PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(S.nbc_h.p, S.nbc_d.p, (size_t)ni * sizeof(int), cudaMemcpyDeviceToHost,
                                                S.stream), return);
        PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(S.nbl_h.p, S.nbl_d.p, (size_t)ni * cap * sizeof(int),
                                                cudaMemcpyDeviceToHost, S.stream), return);
        PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(S.stream), return);
        for (int i = 0; i < ni; i++) {
            const int count = S.nbc_h.p[i], c = count > cap ? 0 : count;
            int* list = add_list(i, count, c);
            if (c > 0) std::memcpy(list, S.nbl_h.p + (size_t)i * cap, (size_t)c * sizeof(int));
        }
    }
    for (int i = 0; i < ni; i++)
        if (S.nbcounts[i] > cap) S.nb_error = 1;
}

// The common body of every g6calc_lasthalf* variant.
int lasthalf_impl(int nj, int ni, const int* pidx, const double (*pos)[3], const double (*vel)[3], double eps2,
                  const double* h2, double (*acc)[3], double (*jrk)[3], double* pot, int* nnb, float* rnnb,
                  bool nbl) {
    if (ni < 0 || ni > npipes()) {
        raise(g_err, LIB, PGB_ERR_ARG, "ni = %d outside [0, %d] pipes", ni, npipes());
        return 0;
    }
    if (nj < 0) {
        raise(g_err, LIB, PGB_ERR_ARG, "nj = %d is negative", nj);
        return 0;
    }
    if (ni == 0) return 0;
    std::lock_guard<std::mutex> g(S.mu);
    // checked under the lock: a concurrent g6_set_j_particle may grow the j store
    if (nj > S.jcap) {
        raise(g_err, LIB, PGB_ERR_ARG, "nj = %d but only %d j-particles were set", nj, S.jcap);
        return 0;
    }
    if (!init_state()) return 0;
    if (S.ibuf.reserve(ni) != cudaSuccess) {
        raise(g_err, LIB, PGB_ERR_CUDA, "pinned i-buffer allocation failed");
        return 0;
    }
    for (int i = 0; i < ni; i++) {
        G6I& r = S.ibuf.p[i];
        store_pos(r.p, pos[i][0], pos[i][1], pos[i][2], dx_ff());
        r.vx = (float)vel[i][0];
        r.vy = (float)vel[i][1];
        r.vz = (float)vel[i][2];
        r.id = pidx[i];
        r.h2 = (nbl && h2) ? (float)h2[i] : 0.f;
        r.pad = 0.f;
    }
    bool nn = (nnb != nullptr);
    // eps2 is a per-call scalar, used as float (phantom_g6.c:191)
    S.wait_words = false;
    if (!time_mark(0)) return 0;
    if (!run_force(nj, ni, (float)eps2, nn, nbl)) return 0;
    if (!time_mark(1)) return 0;
    if (!wait_results(ni) || !time_add()) return 0;
    S.uploading = false;   // the upload came before the results
    for (int i = 0; i < ni; i++) {
        const G6Out& o = S.outh.p[i];
        acc[i][0] = o.ax;
        acc[i][1] = o.ay;
        acc[i][2] = o.az;
        jrk[i][0] = o.jx;
        jrk[i][1] = o.jy;
        jrk[i][2] = o.jz;
        pot[i] = o.pot;
        if (nnb) nnb[i] = (o.jadr >= 0 && o.jadr < S.jcap) ? S.jh.p[o.jadr].idx : -1;
        if (rnnb) rnnb[i] = -2.0f / o.key;
    }
    if (nbl) nblist_collect(ni);
    return 0;
}

}  // namespace

// ============================================================================================
// GRAPE-6 API (PG6/libpg6/gp6util.h:1-101)

PGB_EXPORT void g6_open(int gpid) {
    (void)gpid;
    std::lock_guard<std::mutex> g(S.mu);
    init_state();
}
PGB_EXPORT void g6_close(int gpid) {
    (void)gpid;
    std::lock_guard<std::mutex> g(S.mu);
    if (!S.ready) return;
    cudaSetDevice(g_device);
    cudaStreamSynchronize(S.stream);
    S.jd.release();
    S.pred.release();
    S.st.release();
    S.pcnt.release();
    S.spart.release();
    S.wait_words = false;
    S.nbc_zero = false;
    S.nbc_d.release();
    S.nbl_d.release();
    S.uploading = false;
    for (int a : S.dirty) S.dirty_flag[a] = 0;
    S.dirty.clear();
    S.all_dirty = true;
    S.jdirty_lo = 0;
    S.jdirty_hi = S.jcap;
}
PGB_EXPORT void g6_set_tunit(int) {}
PGB_EXPORT void g6_set_xunit(int) {}
PGB_EXPORT void g6_reset(int) {}
PGB_EXPORT void g6_reset_fofpga(int) {}
PGB_EXPORT int g6_npipes(void) { return npipes(); }
PGB_EXPORT void g6_setup_njdata(int, int) {}

PGB_EXPORT void g6_set_j_particle(int gpid, int padr, int pidx, double t, double dt, double mss, double* snp,
                                  double* jrk, double* acc, double* vel, double* pos) {
    (void)gpid;
    (void)dt;
    (void)snp;
    if (padr < 0) {
        raise(g_err, LIB, PGB_ERR_ARG, "g6_set_j_particle: negative address %d", padr);
        return;
    }
    std::lock_guard<std::mutex> g(S.mu);
    if (!grow_j(padr + 1) || !wait_upload()) return;
    G6Ptcl& p = S.jh.p[padr];
    for (int d = 0; d < 3; d++) {
        p.pos[d] = pos[d];
        p.vel[d] = vel[d];
        p.acc2[d] = acc[d];
        p.jrk6[d] = jrk[d];
    }
    p.mass = mss;
    p.tim = t;
    p.idx = pidx;
    mark_dirty(padr);
}

PGB_EXPORT void g6_set_ti(int gpid, double time) {
    (void)gpid;
    std::lock_guard<std::mutex> g(S.mu);
    S.ti = time;
    S.predict_flag = 1;
}

PGB_EXPORT void g6calc_firsthalf(int gpid, int nj, int ni, int* pidx, double (*pos)[3], double (*vel)[3],
                                 double (*acc)[3], double (*jrk)[3], double* pot, double eps2, double* h2) {
    (void)gpid; (void)ni; (void)pidx; (void)pos; (void)vel; (void)acc; (void)jrk; (void)pot; (void)eps2; (void)h2;
    std::lock_guard<std::mutex> g(S.mu);
    if (!init_state()) return;
    if (S.predict_flag == 1) {
        if (!flush_and_predict(nj)) return;
        S.predict_flag = 0;
    }
    S.nb_error = 0;  // avx_initialize_neighbourlist (gravity.c:123-128)
}

#define LASTHALF_ARGS int gpid, int nj, int ni, int *pidx, double(*pos)[3], double(*vel)[3], double eps2, double *h2, \
                      double(*acc)[3], double(*jrk)[3], double *pot

PGB_EXPORT int g6calc_lasthalf(LASTHALF_ARGS) {
    (void)gpid;
    return lasthalf_impl(nj, ni, pidx, pos, vel, eps2, h2, acc, jrk, pot, nullptr, nullptr, false);
}
PGB_EXPORT int g6calc_lasthalf2(LASTHALF_ARGS, int* nnb) {
    (void)gpid;
    return lasthalf_impl(nj, ni, pidx, pos, vel, eps2, h2, acc, jrk, pot, nnb, nullptr, false);
}
PGB_EXPORT int g6calc_lasthalf2p(LASTHALF_ARGS, int* nnb, float* rnnb) {
    (void)gpid;
    return lasthalf_impl(nj, ni, pidx, pos, vel, eps2, h2, acc, jrk, pot, nnb, rnnb, false);
}
PGB_EXPORT int g6calc_lasthalfn(LASTHALF_ARGS) {
    (void)gpid;
    return lasthalf_impl(nj, ni, pidx, pos, vel, eps2, h2, acc, jrk, pot, nullptr, nullptr, true);
}
PGB_EXPORT int g6calc_lasthalf2n(LASTHALF_ARGS, int* nnb) {
    (void)gpid;
    return lasthalf_impl(nj, ni, pidx, pos, vel, eps2, h2, acc, jrk, pot, nnb, nullptr, true);
}
PGB_EXPORT int g6calc_lasthalf2np(LASTHALF_ARGS, int* nnb, float* rnnb) {
    (void)gpid;
    return lasthalf_impl(nj, ni, pidx, pos, vel, eps2, h2, acc, jrk, pot, nnb, rnnb, true);
}

// 0: success, 1: a list of the last lasthalf*n call overflowed (phantom_g6.c:482-486)
PGB_EXPORT int g6_read_neighbour_list(int gpid) {
    (void)gpid;
    return S.nb_error;
}

// 0: success, 1: nb > maxlen (phantom_g6.c:495-499, gravity.c:135-147)
PGB_EXPORT int g6_get_neighbour_list(int gpid, int ipipe, int maxlen, int* nblen, int* nbl) {
    (void)gpid;
    if (ipipe < 0 || ipipe >= S.nb_ni) {
        raise(g_err, LIB, PGB_ERR_ARG, "g6_get_neighbour_list: ipipe %d outside [0, %d)", ipipe, S.nb_ni);
        return 1;
    }
    if (S.nbcounts[ipipe] > maxlen || S.nbcounts[ipipe] > nbmax()) return 1;
    *nblen = S.nbcounts[ipipe];
    if (*nblen > 0) std::memcpy(nbl, S.nbids.data() + S.nboff[ipipe], (size_t)*nblen * sizeof(int));
    return 0;
}

PGB_EXPORT void g6_debugfunc(int tmp) {
    FILE* fp = std::fopen("dump.dat", "a");
    if (!fp) return;
    std::fprintf(fp, "%d\n", tmp);
    std::fclose(fp);
}
PGB_EXPORT void g6_debugfunc_double(double tmp) {
    FILE* fp = std::fopen("dump.dat", "a");
    if (!fp) return;
    std::fprintf(fp, "%+e\n", tmp);
    std::fclose(fp);
}
PGB_EXPORT void g6_dump(double tim, int n, double* m, double (*x)[3], double (*v)[3]) {
    char out[64];
    std::snprintf(out, sizeof out, "dump.dat.%05d", (int)tim);
    FILE* fp = std::fopen(out, "w");
    if (!fp) return;
    for (int i = 0; i < n; i++) {
        std::fprintf(fp, "%+.16e", m[i]);
        std::fprintf(fp, " %+.16e %+.16e %+.16e", x[i][0], x[i][1], x[i][2]);
        std::fprintf(fp, " %+.16e %+.16e %+.16e", v[i][0], v[i][1], v[i][2]);
        std::fprintf(fp, "\n");
    }
    std::fclose(fp);
}

// Fortran twins (phantom_g6.c: every entry point has a `_` variant taking pointers)
PGB_EXPORT void g6_open_(int* gpid) { g6_open(*gpid); }
PGB_EXPORT void g6_close_(int* gpid) { g6_close(*gpid); }
PGB_EXPORT void g6_set_tunit_(int* v) { g6_set_tunit(*v); }
PGB_EXPORT void g6_set_xunit_(int* v) { g6_set_xunit(*v); }
PGB_EXPORT void g6_reset_(int* v) { g6_reset(*v); }
PGB_EXPORT void g6_reset_fofpga_(int* v) { g6_reset_fofpga(*v); }
PGB_EXPORT int g6_npipes_(void) { return g6_npipes(); }
PGB_EXPORT void g6_setup_njdata_(int* gpid, int* nj) { g6_setup_njdata(*gpid, *nj); }
PGB_EXPORT void g6_set_j_particle_(int* gpid, int* padr, int* pidx, double* t, double* dt, double* mss, double* snp,
                                   double* jrk, double* acc, double* vel, double* pos) {
    g6_set_j_particle(*gpid, *padr, *pidx, *t, *dt, *mss, snp, jrk, acc, vel, pos);
}
PGB_EXPORT void g6_set_ti_(int* gpid, double* t) { g6_set_ti(*gpid, *t); }
PGB_EXPORT void g6calc_firsthalf_(int* gpid, int* nj, int* ni, int* pidx, double (*pos)[3], double (*vel)[3],
                                  double (*acc)[3], double (*jrk)[3], double* pot, double* eps2, double* h2) {
    g6calc_firsthalf(*gpid, *nj, *ni, pidx, pos, vel, acc, jrk, pot, *eps2, h2);
}
#define LASTHALF_FARGS int *gpid, int *nj, int *ni, int *pidx, double(*pos)[3], double(*vel)[3], double *eps2, \
                       double *h2, double(*acc)[3], double(*jrk)[3], double *pot
#define LASTHALF_FCALL *gpid, *nj, *ni, pidx, pos, vel, *eps2, h2, acc, jrk, pot
PGB_EXPORT int g6calc_lasthalf_(LASTHALF_FARGS) { return g6calc_lasthalf(LASTHALF_FCALL); }
PGB_EXPORT int g6calc_lasthalf2_(LASTHALF_FARGS, int* nnb) { return g6calc_lasthalf2(LASTHALF_FCALL, nnb); }
PGB_EXPORT int g6calc_lasthalf2p_(LASTHALF_FARGS, int* nnb, float* rnnb) {
    return g6calc_lasthalf2p(LASTHALF_FCALL, nnb, rnnb);
}
PGB_EXPORT int g6calc_lasthalfn_(LASTHALF_FARGS) { return g6calc_lasthalfn(LASTHALF_FCALL); }
PGB_EXPORT int g6calc_lasthalf2n_(LASTHALF_FARGS, int* nnb) { return g6calc_lasthalf2n(LASTHALF_FCALL, nnb); }
PGB_EXPORT int g6calc_lasthalf2np_(LASTHALF_FARGS, int* nnb, float* rnnb) {
    return g6calc_lasthalf2np(LASTHALF_FCALL, nnb, rnnb);
}
PGB_EXPORT int g6_read_neighbour_list_(int* gpid) { return g6_read_neighbour_list(*gpid); }
PGB_EXPORT int g6_get_neighbour_list_(int* gpid, int* ipipe, int* maxlen, int* nblen, int* nbl) {
    return g6_get_neighbour_list(*gpid, *ipipe, *maxlen, nblen, nbl);
}
PGB_EXPORT void g6_debugfunc_(int* v) { g6_debugfunc(*v); }
PGB_EXPORT void g6_debugfunc_double_(double* v) { g6_debugfunc_double(*v); }
PGB_EXPORT void g6_dump_(double* tim, int* n, double* m, double (*x)[3], double (*v)[3]) { g6_dump(*tim, *n, m, x, v); }

// ============================================================================================
// Library status and the batched path (no reference counterpart; declared in include/pgb_g6.h)

PGB_EXPORT int pgb6_last_error(char* buf, int len) {
    std::lock_guard<std::mutex> g(g_err.mu);
    if (buf && len > 0) {
        std::strncpy(buf, g_err.msg.c_str(), (size_t)len - 1);
        buf[len - 1] = 0;
    }
    return g_err.code;
}
PGB_EXPORT void pgb6_clear_error(void) {
    std::lock_guard<std::mutex> g(g_err.mu);
    g_err.code = 0;
    g_err.msg.clear();
}
PGB_EXPORT void pgb6_set_abort(int on) {
    std::lock_guard<std::mutex> g(g_err.mu);
    g_err.abort_on_error = on ? 1 : 0;
}

// Sizes of the device record types, so callers can lay out device buffers:
// G6Ptcl (j-memory), G6PredJ (predicted j), G6I (i-particle), G6Out (result).
// Device-time accounting of the drop-in calls (no counterpart in the reference): with on != 0,
// every g6calc_firsthalf (j-memory update + prediction) and g6calc_lasthalf* (force launch, with the
// sort of a small call's neighbour lists)
// adds the device time between CUDA events recorded around its work on the library's stream
// to a running total; pgb6_call_device_ms returns that total in ms (and clears it when reset
// != 0).  It separates the device work of the plain API from its host overhead.
PGB_EXPORT void pgb6_set_call_timing(int on) {
    std::lock_guard<std::mutex> g(S.mu);
    S.time_calls = on != 0;
}

PGB_EXPORT double pgb6_call_device_ms(int reset) {
    std::lock_guard<std::mutex> g(S.mu);
    const double v = S.dev_ms;
    if (reset) S.dev_ms = 0.0;
    return v;
}

PGB_EXPORT void pgb6_record_sizes(int* ptcl, int* predj, int* irec, int* out) {
    if (ptcl) *ptcl = (int)sizeof(G6Ptcl);
    if (predj) *predj = (int)sizeof(G6PredJ);
    if (irec) *irec = (int)sizeof(G6I);
    if (out) *out = (int)sizeof(G6Out);
}

namespace {
// Autotune cache: work-item-table shape -> best kernel configuration measured by
// pgb6_plan_tune.  The shape key buckets the item count, the largest i and j counts (powers of
// two) and the variant flags, so plans of the same shape reuse a measured choice.
std::mutex g_tune_mu;
struct Tuned {
    int cfg, nch;   // nch 0: the model's chunk count; below 0: -nch chunks, not of whole tiles
};
std::vector<std::pair<long long, Tuned>> g_tune;

int ilog2up(long long v) {
    int k = 0;
    while ((1LL << k) < v && k < 62) k++;
    return k;
}

long long shape_key(int nitem, const int* items, bool ff, bool nn) {
    long long nimax = 0, njmax = 0;
    for (int k = 0; k < nitem; k++) {
        nimax = std::max<long long>(nimax, items[4 * k + 1]);
        njmax = std::max<long long>(njmax, items[4 * k + 3]);
    }
    return ((long long)ilog2up(nitem + 1) << 24) | ((long long)ilog2up(nimax + 1) << 16) |
           ((long long)ilog2up(njmax + 1) << 8) | (ff ? 2 : 0) | (nn ? 1 : 0);
}

Tuned tuned_cfg(long long key) {
    std::lock_guard<std::mutex> g(g_tune_mu);
    for (auto& e : g_tune)
        if (e.first == key) return e.second;
    return Tuned{-1, 0};
}

void set_tuned(long long key, Tuned t) {
    std::lock_guard<std::mutex> g(g_tune_mu);
    for (auto& e : g_tune)
        if (e.first == key) {
            e.second = t;
            return;
        }
    g_tune.emplace_back(key, t);
}
}  // namespace

// The largest j_offset + j_count of an item table ([k][4] = i_off, i_cnt, j_off, j_cnt).
int items_jend(int nitem, const int* items) {
    long long e = 0;
    for (int k = 0; k < nitem; k++) e = std::max<long long>(e, (long long)items[4 * k + 2] + items[4 * k + 3]);
    return (int)std::min<long long>(e, 0x7fffffff);
}

struct pgb6_plan {
    int cfg;
    bool nn;
    bool ff;
    std::vector<int> items;    // the work-item table, kept for re-planning (autotuning)
    int jend = 0;              // the items' largest j_offset + j_count (the j records they read)
    long long shape_key = 0;   // autotune cache key of this work-item table
    int nch = 0;               // a single item's chunk count (0: the wave model's, see plan_items)
    std::vector<Task> tasks;
    std::vector<Group> groups;
    int rows = 0;
    long long interactions = 0;
    Stager<G6I, G6Out> st;
    cudaEvent_t launched = nullptr;   // recorded after every stream (not graph-captured) launch
};

enum { PGB6_NN = 1, PGB6_POS_F64 = 2 };

// items: [nitem][4] = (i_offset, i_count, j_offset, j_count) into the i- and j-arrays.
// flags: PGB6_NN (1) also computes the nearest neighbour (key, j address); PGB6_POS_F64 (2):
// the i/j records hold FP64 positions (default: double-float positions, see Pos3).
PGB_EXPORT int pgb6_plan_create(pgb6_plan** out, int nitem, const int* items, int flags) {
    if (!out || nitem < 0 || (nitem && !items)) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_create: bad arguments");
        return PGB_ERR_ARG;
    }
    for (int k = 0; k < nitem; k++)
        if (items[4 * k] < 0 || items[4 * k + 1] < 0 || items[4 * k + 2] < 0 || items[4 * k + 3] < 0) {
            raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_create: item %d has a negative offset or count", k);
            return PGB_ERR_ARG;
        }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    auto* P = new pgb6_plan();
    P->nn = (flags & PGB6_NN) != 0;
    P->ff = (flags & PGB6_POS_F64) == 0;
    P->items.assign(items, items + 4 * (size_t)nitem);
    P->jend = items_jend(nitem, items);
    P->shape_key = shape_key(nitem, items, P->ff, P->nn);
    const Tuned tuned = tuned_cfg(P->shape_key);
    P->cfg = tuned.cfg >= 0 ? tuned.cfg : pick_batch_cfg(nitem, items, P->ff, P->nn);
    P->nch = tuned.cfg >= 0 ? tuned.nch : 0;
    P->interactions = plan_items(P->tasks, P->groups, P->rows, nitem, items, P->cfg, P->ff, P->nn, false, P->nch);
    cudaStream_t s = nullptr;
    bool ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && P->st.stage(s, P->tasks, P->groups, P->rows, ITILE_MAX, (const G6I*)nullptr, 0) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(s) == cudaSuccess;
    if (s) cudaStreamDestroy(s);
    if (!ok) {
        P->st.release();
        delete P;
        raise(g_err, LIB, PGB_ERR_CUDA, "pgb6_plan_create: staging failed");
        return PGB_ERR_CUDA;
    }
    *out = P;
    return PGB_OK;
}

PGB_EXPORT long long pgb6_plan_interactions(const pgb6_plan* P) { return P ? P->interactions : 0; }
PGB_EXPORT int pgb6_plan_tasks(const pgb6_plan* P) { return P ? (int)P->tasks.size() : 0; }
PGB_EXPORT int pgb6_plan_config(const pgb6_plan* P) { return P ? reported_cfg(P->cfg) : -1; }
// j-chunks per i-tile of a one-item plan (1: the j-range unsplit); 0 for plans of several items.
PGB_EXPORT int pgb6_plan_chunks(const pgb6_plan* P) {
    if (!P || P->items.size() != 4 || P->tasks.empty()) return 0;
    return P->groups.empty() ? 1 : (int)(P->tasks.size() / P->groups.size());
}
// Kernels one pgb6_plan_launch issues: the force kernel, and the nearest-neighbour lookups of
// split i-tiles when the plan's configuration defers them.
PGB_EXPORT int pgb6_plan_kernels(const pgb6_plan* P) {
    if (!P || P->tasks.empty()) return 0;
    return 1 + (needs_resolve(P->cfg, P->ff, P->nn, false, (int)P->groups.size(), P->jend) ? 1 : 0);
}

// Device-resident launch (capturable in a CUDA graph): ipart = G6I[], jpred = G6PredJ[],
// out = G6Out[] indexed by absolute i (acc, jerk, pot final; key = -2/r_soft of the nearest
// neighbour, jadr = its j address, when the plan has PGB6_NN).
PGB_EXPORT int pgb6_plan_launch(pgb6_plan* P, const void* ipart, const void* jpred, double eps2, void* out,
                                void* stream) {
    if (!P || !ipart || !jpred || !out) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_launch: null argument");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    if (P->st.ntasks == 0) return PGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    G6Args a;
    a.ipart = (const G6I*)ipart;
    a.jpred = (const G6PredJ*)jpred;
    a.eps2 = (float)eps2;
    a.tasks = P->st.tasks();
    a.ntasks = P->st.ntasks;
    a.task_counter = P->st.counter();
    a.groups = P->st.groups();
    a.group_counters = P->st.dgcnt.p;
    a.partial = P->st.dpart.p;
    a.out = (G6Out*)out;
    a.itile = kernel_info(P->cfg, P->ff, P->nn, false).itile;
    a.bundle_counters = P->st.bundle_counters();
    a.nb_count = nullptr;
    a.nb_list = nullptr;
    a.nb_maxlen = 0;
    a.jn = P->jend;
    int slots = sm_count(g_device) * occupancy(P->cfg, P->ff, P->nn, false);
    int grid = a.ntasks < slots ? a.ntasks : slots;
    PGB_CUDA_OR(g_err, LIB, launch_kernel(P->cfg, P->ff, P->nn, false, grid, a, s), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, launch_resolve(P->cfg, P->ff, P->nn, false, (int)P->groups.size(), a, s),
                return PGB_ERR_CUDA);
    // completion marker for pgb6_plan_update (none for a launch captured into a CUDA graph)
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    PGB_CUDA_OR(g_err, LIB, cudaStreamIsCapturing(s, &cap), return PGB_ERR_CUDA);
    if (cap == cudaStreamCaptureStatusNone) {
        if (!P->launched)
            PGB_CUDA_OR(g_err, LIB, cudaEventCreateWithFlags(&P->launched, cudaEventDisableTiming),
                        return PGB_ERR_CUDA);
        PGB_CUDA_OR(g_err, LIB, cudaEventRecord(P->launched, s), return PGB_ERR_CUDA);
    }
    return PGB_OK;
}

// Pin one kernel configuration (0 .. NCFG-1) and re-plan for it (after the plan's previous
// stream launches have finished).
PGB_EXPORT int pgb6_plan_set_config(pgb6_plan* P, int cfg) {
    if (!P || cfg < 0 || cfg >= NCFG) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_set_config: configuration %d outside [0, %d)", cfg, (int)NCFG);
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    P->cfg = cfg;
    P->nch = 0;
    const int nitem = (int)(P->items.size() / 4);
    P->tasks.clear();
    P->groups.clear();
    P->interactions = plan_items(P->tasks, P->groups, P->rows, nitem, P->items.data(), cfg, P->ff, P->nn, false);
    if (P->launched) PGB_CUDA_OR(g_err, LIB, cudaEventSynchronize(P->launched), return PGB_ERR_CUDA);
    cudaStream_t s = nullptr;
    bool ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && P->st.stage(s, P->tasks, P->groups, P->rows, ITILE_MAX, (const G6I*)nullptr, 0) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(s) == cudaSuccess;
    if (s) cudaStreamDestroy(s);
    if (!ok) {
        raise(g_err, LIB, PGB_ERR_CUDA, "pgb6_plan_set_config: staging failed");
        return PGB_ERR_CUDA;
    }
    return PGB_OK;
}

// New items for an existing plan (same flags; its configuration kept), re-planned on the host
// and staged into the plan's own buffers, which grow only when needed: a code whose active sets
// or clusters change every step keeps one plan instead of creating and destroying one per step
// (no device allocation, hence no device-wide synchronisation, in its step).  Waits until the
// plan's previous stream launches have finished reading its task list.
PGB_EXPORT int pgb6_plan_update(pgb6_plan* P, int nitem, const int* items) {
    if (!P || nitem < 0 || (nitem && !items)) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_update: null plan or bad item count %d", nitem);
        return PGB_ERR_ARG;
    }
    for (int k = 0; k < nitem; k++)
        if (items[4 * k] < 0 || items[4 * k + 1] < 0 || items[4 * k + 2] < 0 || items[4 * k + 3] < 0) {
            raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_update: item %d has a negative offset or count", k);
            return PGB_ERR_ARG;
        }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    P->items.assign(items, items + 4 * (size_t)nitem);
    P->jend = items_jend(nitem, items);
    P->shape_key = shape_key(nitem, items, P->ff, P->nn);
    const Tuned tuned = tuned_cfg(P->shape_key);
    P->nch = (tuned.cfg == P->cfg) ? tuned.nch : 0;
    P->tasks.clear();
    P->groups.clear();
    P->interactions = plan_items(P->tasks, P->groups, P->rows, nitem, items, P->cfg, P->ff, P->nn, false, P->nch);
    if (P->launched) PGB_CUDA_OR(g_err, LIB, cudaEventSynchronize(P->launched), return PGB_ERR_CUDA);
    cudaStream_t s = nullptr;
    bool ok = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && P->st.stage(s, P->tasks, P->groups, P->rows, ITILE_MAX, (const G6I*)nullptr, 0) == cudaSuccess;
    ok = ok && cudaStreamSynchronize(s) == cudaSuccess;
    if (s) cudaStreamDestroy(s);
    if (!ok) {
        raise(g_err, LIB, PGB_ERR_CUDA, "pgb6_plan_update: staging failed");
        return PGB_ERR_CUDA;
    }
    return PGB_OK;
}

// Autotuner: launches the plan with every kernel configuration (threads per CTA x i per
// thread x j-lanes) on the caller's data -- a plan of one item also with the chunk counts of
// chunk_candidates for its three fastest configurations -- keeps the fastest (CUDA-event time,
// the median of three launches after a warm-up launch, so that a shape whose time alternates
// between launches is judged by its usual time), re-stages the plan with it and records it for
// plans of the same shape.  Returns the chosen configuration index; *best_ms (optional)
// receives its launch time.  Overwrites `out`.  Not capturable (it synchronises the stream).
PGB_EXPORT int pgb6_plan_tune(pgb6_plan* P, const void* ipart, const void* jpred, double eps2, void* out,
                              void* stream, float* best_ms) {
    if (!P || !ipart || !jpred || !out) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_plan_tune: null argument");
        return -1;
    }
    if (!ensure_device()) return -1;
    cudaStream_t s = (cudaStream_t)stream;
    cudaEvent_t e0, e1;
    PGB_CUDA_OR(g_err, LIB, cudaEventCreate(&e0), return -1);
    PGB_CUDA_OR(g_err, LIB, cudaEventCreate(&e1), return -1);
    const int nitem = (int)(P->items.size() / 4);
    // one (configuration, chunk count): the median of three timed launches after a warm-up
    auto time_plan = [&](int cfg, int nch, float* t) -> bool {
        P->tasks.clear();
        P->groups.clear();
        P->cfg = cfg;
        P->nch = nch;
        plan_items(P->tasks, P->groups, P->rows, nitem, P->items.data(), cfg, P->ff, P->nn, false, nch);
        if (P->st.stage(s, P->tasks, P->groups, P->rows, ITILE_MAX, (const G6I*)nullptr, 0) != cudaSuccess) return false;
        if (pgb6_plan_launch(P, ipart, jpred, eps2, out, stream) != PGB_OK) return false;
        float ts[3];
        for (int rep = 0; rep < 3; rep++) {
            cudaEventRecord(e0, s);
            if (pgb6_plan_launch(P, ipart, jpred, eps2, out, stream) != PGB_OK) return false;
            cudaEventRecord(e1, s);
            if (cudaEventSynchronize(e1) != cudaSuccess) return false;
            cudaEventElapsedTime(&ts[rep], e0, e1);
        }
        std::sort(ts, ts + 3);
        *t = ts[1];
        return true;
    };
    std::vector<std::pair<float, int>> by_cfg;
    // CFG_MED1 is CFG_MED with FP64 positions, and has not been the fastest above 2^25 pairs
    const int ncfg = P->ff && P->interactions < (1LL << 26) ? NCFG + 1 : NCFG;
    for (int cfg = 0; cfg < ncfg; cfg++) {
        float t;
        if (!time_plan(cfg, 0, &t)) break;
        by_cfg.emplace_back(t, cfg);
    }
    std::sort(by_cfg.begin(), by_cfg.end());
    Tuned best{P->cfg, 0};
    float best_t = 1e30f;
    if (!by_cfg.empty()) {
        best = Tuned{by_cfg[0].second, 0};
        best_t = by_cfg[0].first;
    }
    if (nitem == 1 && P->items[1] > 0 && P->items[3] > 0) {
        static const int maxch = env_int("PGB_G6_MAXCHUNKS", 512, 1, 4096);
        const int ni = P->items[1], nj = P->items[3];
        for (size_t r = 0; r < by_cfg.size() && r < 3; r++) {
            const int cfg = by_cfg[r].second;
            const KernelInfo K = kernel_info(cfg, P->ff, P->nn, false);
            const long long jc = model_chunk(K, (ni + K.itile - 1) / K.itile, nj, sm_count(g_device) * K.occ, maxch);
            const int m = (int)((nj + jc - 1) / jc);
            std::vector<int> cand = chunk_candidates(m, nj, maxch);
            // of whole tiles a j-paired kernel may have no count that fills one wave of CTAs: the wave
            // model's, in plain chunks (3479 x 11705 without neighbours: 21 chunks of 557 records,
            // 85.8 us, against 87.7 for the best of whole tiles)
            if (K.paired)
                cand.push_back(-best_nch((ni + K.itile - 1) / K.itile, nj, sm_count(g_device) * K.occ, maxch));
            for (int nch : cand) {
                if (nch == m) continue;   // timed above
                float t;
                if (!time_plan(cfg, nch, &t)) break;
                if (t < best_t) {
                    best_t = t;
                    best = Tuned{cfg, nch};
                }
            }
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    P->tasks.clear();
    P->groups.clear();
    P->cfg = best.cfg;
    P->nch = best.nch;
    plan_items(P->tasks, P->groups, P->rows, nitem, P->items.data(), best.cfg, P->ff, P->nn, false, best.nch);
    PGB_CUDA_OR(g_err, LIB, P->st.stage(s, P->tasks, P->groups, P->rows, ITILE_MAX, (const G6I*)nullptr, 0),
                return -1);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(s), return -1);
    set_tuned(P->shape_key, best);
    if (best_ms) *best_ms = best_t;
    return reported_cfg(best.cfg);
}

PGB_EXPORT void pgb6_plan_destroy(pgb6_plan* P) {
    if (!P) return;
    if (g_device >= 0) cudaSetDevice(g_device);
    P->st.release();
    if (P->launched) cudaEventDestroy(P->launched);
    delete P;
}

// FP64 predictor on device records: pred[j] = predict(ptcl[j], ti) for j < nj.
// flags: PGB6_POS_F64 (2) writes FP64 positions, else the double-float layout.
PGB_EXPORT int pgb6_predict(const void* ptcl, int nj, double ti, void* pred, int flags, void* stream) {
    if (nj < 0 || (nj > 0 && (!ptcl || !pred))) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_predict: bad arguments");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    if (nj == 0) return PGB_OK;
    g6_predict_kernel<<<(nj + 255) / 256, 256, 0, (cudaStream_t)stream>>>((const G6Ptcl*)ptcl, nj, ti, (G6PredJ*)pred,
                                                                           (flags & PGB6_POS_F64) == 0);
    PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return PGB_ERR_CUDA);
    return PGB_OK;
}

namespace {
struct HostBatch {
    std::mutex mu;
    cudaStream_t s = nullptr;
    HostBuf<G6I> ih;
    HostBuf<G6PredJ> jh;
    HostBuf<G6Out> oh;
    DevBuf<G6I> id;
    DevBuf<G6PredJ> jd;
    DevBuf<G6Out> od;
};
HostBatch HB;
}  // namespace

// Host-buffer batch: the whole list of items in one launch, inputs and outputs in host memory
// (copies included).  Positions FP64; velocities, masses rounded to float as the GRAPE-6 path
// does.  nnb / rnnb may be NULL.
PGB_EXPORT int pgb6_batch_host(int nitem, const int* items, int ni, const double (*xi)[3], const double (*vi)[3],
                               const int* idi, int nj, const double (*xj)[3], const double (*vj)[3], const double* mj,
                               const int* idj, double eps2, double (*acc)[3], double (*jrk)[3], double* pot, int* nnb,
                               float* rnnb) {
    if (ni < 0 || nj < 0) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_batch_host: negative sizes");
        return PGB_ERR_ARG;
    }
    for (int k = 0; k < nitem; k++) {
        const int* it = items + 4 * k;
        if (it[0] < 0 || it[1] < 0 || it[2] < 0 || it[3] < 0 || it[0] + it[1] > ni || it[2] + it[3] > nj) {
            raise(g_err, LIB, PGB_ERR_ARG, "pgb6_batch_host: item %d outside the arrays", k);
            return PGB_ERR_ARG;
        }
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(HB.mu);
    if (!HB.s) PGB_CUDA_OR(g_err, LIB, cudaStreamCreateWithFlags(&HB.s, cudaStreamNonBlocking), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, HB.ih.reserve(ni + 1), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, HB.jh.reserve(nj + 1), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, HB.oh.reserve(ni + 1), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, HB.id.reserve(ni + 1), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, HB.jd.reserve(nj + 1), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, HB.od.reserve(ni + 1), return PGB_ERR_CUDA);
    for (int i = 0; i < ni; i++) {
        G6I& r = HB.ih.p[i];
        store_pos(r.p, xi[i][0], xi[i][1], xi[i][2], dx_ff());
        r.vx = (float)vi[i][0]; r.vy = (float)vi[i][1]; r.vz = (float)vi[i][2];
        r.id = idi[i];
        r.h2 = 0.f;
        r.pad = 0.f;
    }
    for (int j = 0; j < nj; j++) {
        G6PredJ& r = HB.jh.p[j];
        store_pos(r.p, xj[j][0], xj[j][1], xj[j][2], dx_ff());
        r.vx = (float)vj[j][0]; r.vy = (float)vj[j][1]; r.vz = (float)vj[j][2];
        r.m = (float)mj[j];
        r.id = idj[j];
        r.pad = 0.f;
    }
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(HB.id.p, HB.ih.p, (size_t)ni * sizeof(G6I), cudaMemcpyHostToDevice, HB.s),
                return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(HB.jd.p, HB.jh.p, (size_t)nj * sizeof(G6PredJ), cudaMemcpyHostToDevice, HB.s),
                return PGB_ERR_CUDA);
    pgb6_plan* P = nullptr;
    int rc = pgb6_plan_create(&P, nitem, items, ((nnb || rnnb) ? PGB6_NN : 0) | (dx_ff() ? 0 : PGB6_POS_F64));
    if (rc) return rc;
    rc = pgb6_plan_launch(P, HB.id.p, HB.jd.p, eps2, HB.od.p, HB.s);
    if (!rc && ni > 0)
        PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(HB.oh.p, HB.od.p, (size_t)ni * sizeof(G6Out), cudaMemcpyDeviceToHost, HB.s),
                    rc = PGB_ERR_CUDA);
    if (!rc) PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(HB.s), rc = PGB_ERR_CUDA);
    pgb6_plan_destroy(P);
    if (rc) return rc;
    // outputs only for i covered by an item
    for (int k = 0; k < nitem; k++) {
        for (int i = items[4 * k]; i < items[4 * k] + items[4 * k + 1]; i++) {
            const G6Out& o = HB.oh.p[i];
            acc[i][0] = o.ax; acc[i][1] = o.ay; acc[i][2] = o.az;
            jrk[i][0] = o.jx; jrk[i][1] = o.jy; jrk[i][2] = o.jz;
            pot[i] = o.pot;
            if (nnb) nnb[i] = (o.jadr >= 0 && o.jadr < nj) ? idj[o.jadr] : -1;
            if (rnnb) rnnb[i] = -2.0f / o.key;
        }
    }
    return PGB_OK;
}

// ============================================================================================
// Allocation-free Hermite force call (no counterpart in the reference).
//
// For callers that must not allocate GPU memory: codes whose device memory is owned by their
// own pool allocator (a simulation that reserves most of HBM at start-up and hands libraries
// fixed buffers), and time-step loops that cannot afford the device-wide synchronisation a
// cudaMalloc / cudaFree may cause.  pgb6_force_noalloc runs the same force kernel as the
// plans, but its work list, group counters and partial sums live in one fixed array in the
// library's own static device memory (g6_noalloc_scratch below, 16 MiB, held on every GPU the
// library is loaded on until the process exits).  It never calls cudaMalloc or cudaFree.
//
// Set-up: the first call on a device looks up the array's device address there (this first
// call should come before any stream capture).  Every call shares the array and leaves its
// contents behind; each call clears the counters it needs first.  Calls whose launches overlap
// on the GPU (different streams, or different host threads) race on the array and corrupt
// each other's results: serialise them.

namespace {
constexpr size_t NOALLOC_BYTES = size_t(16) << 20;     // the whole scratch array
constexpr int NOALLOC_MAX_ITILES = 4096;                // i-tiles (one group counter each)
constexpr int NOALLOC_MAX_TASKS = 16384;
constexpr size_t NA_OFF_GCNT = 256;                                        // task counter first
constexpr size_t NA_OFF_TASKS = NA_OFF_GCNT + sizeof(int) * NOALLOC_MAX_ITILES;
constexpr size_t NA_OFF_GROUPS = NA_OFF_TASKS + sizeof(Task) * NOALLOC_MAX_TASKS;
constexpr size_t NA_OFF_PART = (NA_OFF_GROUPS + sizeof(Group) * NOALLOC_MAX_ITILES + 255) & ~size_t(255);
constexpr size_t NOALLOC_MAX_PART = (NOALLOC_BYTES - NA_OFF_PART) / sizeof(G6Out);
}  // namespace

static __device__ __align__(256) unsigned char g6_noalloc_scratch[NOALLOC_BYTES];

namespace {
std::mutex g_na_mu;
void* g_na_addr[64];  // device address of g6_noalloc_scratch per device (set-up once)

// Regular decomposition of one (ni x nj) item into itiles x nch tasks of jc j, written to the scratch
// work list (the layout the force kernel reads from a staged plan).
__global__ void g6_regular_tasks(Task* tasks, Group* groups, int ni, int nj, int itile, int itiles, int nch, int jc) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= itiles * nch) return;
    int it = t / nch, c = t % nch;
    int i0 = it * itile;
    int nii = min(itile, ni - i0);
    int j0 = c * jc, j1 = c + 1 < nch ? j0 + jc : nj;
    if (nch == 1) {
        tasks[t] = Task{i0, nii, 0, nj, -1, 0, -1, 0};
        return;
    }
    tasks[t] = Task{i0, nii, j0, j1 - j0, it, c, it * nch + c, 0};
    if (c == 0) groups[it] = Group{i0, nii, nch, it * nch};
}
}  // namespace

// One item: ni i-records (G6I) against nj predicted j-records (G6PredJ), results G6Out per i
// in out (device pointers, caller-owned).  flags: PGB6_NN, PGB6_POS_F64 as for plans.
// Limits: ni <= 4096 i-tiles (1,048,576 particles with the 256-particle tile that large calls
// use); larger ni is refused
// with PGB_ERR_CAPACITY.  Returns PGB_OK or an error code (message in pgb6_last_error).
PGB_EXPORT int pgb6_force_noalloc(const void* ipart, int ni, const void* jpred, int nj, double eps2, void* out,
                                  int flags, void* stream) {
    if (ni < 0 || nj < 0 || (ni > 0 && (!ipart || !out)) || (nj > 0 && !jpred)) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_force_noalloc: bad arguments (ni %d, nj %d)", ni, nj);
        return PGB_ERR_ARG;
    }
    if (ni == 0) return PGB_OK;
    if (!ensure_device()) return PGB_ERR_NOGPU;
    const bool nn = (flags & PGB6_NN) != 0, ff = (flags & PGB6_POS_F64) == 0;
    int cfg = pick_cfg(ni, nj, ff, nn, false);
    int itile = kernel_info(cfg, ff, nn, false).itile;
    if (ni > (long long)NOALLOC_MAX_ITILES * itile) {   // too many small tiles: the 256-particle tile
        cfg = ff ? CFG_128x2JS : CFG_LARGE;
        itile = kernel_info(cfg, ff, nn, false).itile;
    }
    const long long itiles = (ni + (long long)itile - 1) / itile;
    if (itiles > NOALLOC_MAX_ITILES) {
        raise(g_err, LIB, PGB_ERR_CAPACITY, "pgb6_force_noalloc: ni = %d exceeds the fixed scratch (%d i-tiles of %d)",
              ni, NOALLOC_MAX_ITILES, itile);
        return PGB_ERR_CAPACITY;
    }
    void* base = nullptr;
    {
        std::lock_guard<std::mutex> g(g_na_mu);
        if (g_device < 0 || g_device >= 64) {
            raise(g_err, LIB, PGB_ERR_NOGPU, "pgb6_force_noalloc: device %d outside the supported range [0, 64)",
                  g_device);
            return PGB_ERR_NOGPU;
        }
        if (!g_na_addr[g_device]) {
            cudaError_t e = cudaGetSymbolAddress(&g_na_addr[g_device], g6_noalloc_scratch);
            if (e != cudaSuccess) {
                g_na_addr[g_device] = nullptr;
                raise(g_err, LIB, PGB_ERR_CUDA, "pgb6_force_noalloc: cudaGetSymbolAddress failed: %s",
                      cudaGetErrorString(e));
                return PGB_ERR_CUDA;
            }
        }
        base = g_na_addr[g_device];
    }
    // j-chunks per i-tile: a single-item plan's (model_chunk), within the scratch's task and
    // partial-row capacity.  (About four tasks per resident CTA instead: 777 x 65536 201 us, 2048 x 4096 47.)
    const KernelInfo K = kernel_info(cfg, ff, nn, false);
    const int slots = sm_count(g_device) * K.occ;
    long long maxch = std::min<long long>(512, NOALLOC_MAX_TASKS / itiles);
    maxch = std::min<long long>(maxch, (long long)(NOALLOC_MAX_PART / ((size_t)itiles * itile)));
    if (maxch < 1) maxch = 1;
    const long long jc = nj > 0 ? std::min<long long>(nj, model_chunk(K, itiles, nj, slots, (int)maxch)) : 1;
    const long long nch = nj > 0 ? (nj + jc - 1) / jc : 1;
    const int ntasks = (int)(itiles * nch);
    unsigned char* b = (unsigned char*)base;
    cudaStream_t s = (cudaStream_t)stream;
    // the task counter and the group counters must start at zero
    PGB_CUDA_OR(g_err, LIB, cudaMemsetAsync(b, 0, NA_OFF_TASKS, s), return PGB_ERR_CUDA);
    g6_regular_tasks<<<(ntasks + 255) / 256, 256, 0, s>>>((Task*)(b + NA_OFF_TASKS), (Group*)(b + NA_OFF_GROUPS), ni,
                                                          nj, itile, (int)itiles, (int)nch, (int)jc);
    PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return PGB_ERR_CUDA);
    G6Args a;
    a.ipart = (const G6I*)ipart;
    a.jpred = (const G6PredJ*)jpred;
    a.eps2 = (float)eps2;
    a.tasks = (const Task*)(b + NA_OFF_TASKS);
    a.ntasks = ntasks;
    a.task_counter = (int*)b;
    a.groups = (const Group*)(b + NA_OFF_GROUPS);
    a.group_counters = (int*)(b + NA_OFF_GCNT);
    a.partial = (G6Out*)(b + NA_OFF_PART);
    a.out = (G6Out*)out;
    a.itile = itile;
    a.nb_count = nullptr;
    a.nb_list = nullptr;
    a.nb_maxlen = 0;
    a.jn = nj;
    int grid = ntasks < slots ? ntasks : slots;
    PGB_CUDA_OR(g_err, LIB, launch_kernel(cfg, ff, nn, false, grid, a, s), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, launch_resolve(cfg, ff, nn, false, nch > 1 ? (int)itiles : 0, a, s), return PGB_ERR_CUDA);
    return PGB_OK;
}

// ------------------------------------------------------------------------------------------
// Hermite block-time-step integrator on the device (pgb_hermite.cuh): the reference's sample
// integrator PG6/banana (hermite.c, timestep.c; banana01.c:96-183 main loop) with the particle
// state, the j-memory and the per-step bookkeeping resident in HBM.  One cooperative launch
// runs block steps until the global time reaches the caller's tend: the host launches once per
// call and reads the clock back.

struct pgb6_hermite {
    std::mutex mu;
    int n = 0, nseg = 0, grid = 0;
    double eps2 = 0.0, eta = 0.0, eta_s = 0.0, dtmax = 0.0;
    bool ff = true;
    cudaStream_t s = nullptr;
    DevBuf<double> state;          // t, dt, pot, mass [n]; pos, vel, acc, jrk [n][3]
    DevBuf<unsigned char> work;    // HmWork's arrays
    HmState P{};
    HmWork W{};
    double* energy = nullptr;      // [2] device
    HmClock clk{};                 // the device clock as of the last synchronisation
};

namespace {

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

const void* hm_kernel(bool ff, bool start) {
    if (start) return ff ? (const void*)hm_run_kernel<true, true> : (const void*)hm_run_kernel<false, true>;
    return ff ? (const void*)hm_run_kernel<true, false> : (const void*)hm_run_kernel<false, false>;
}

// Co-resident CTAs of the persistent kernel (its cooperative grid, the same for both instances).
int hm_grid(bool ff) {
    static int cache[2] = {0, 0};
    int& g = cache[ff ? 1 : 0];
    if (!g) {
        int least = 0;
        for (bool start : {false, true}) {
            int per = 0;
            const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, hm_kernel(ff, start), HM_NT, 0);
            if (e != cudaSuccess || per < 1) per = 1;
            least = least ? std::min(least, per) : per;
        }
        g = least * sm_count(g_device);
    }
    return g;
}

bool hm_alloc(pgb6_hermite* H) {
    const size_t n = (size_t)H->n;
    PGB_CUDA_OR(g_err, LIB, H->state.reserve(16 * n), return false);
    double* b = H->state.p;
    H->P.n = H->n;
    H->P.t = b;
    H->P.dt = b + n;
    H->P.pot = b + 2 * n;
    H->P.mass = b + 3 * n;
    H->P.pos = b + 4 * n;
    H->P.vel = b + 7 * n;
    H->P.acc = b + 10 * n;
    H->P.jrk = b + 13 * n;
    H->nseg = (int)((n + HM_SEG - 1) / HM_SEG);
    H->grid = hm_grid(H->ff);
    if (H->nseg > HM_OWN * H->grid) {
        raise(g_err, LIB, PGB_ERR_CAPACITY, "pgb6_hermite_create: %d co-resident CTAs are too few", H->grid);
        return false;
    }
    // partial rows: at most (grid + i-tiles) rows of at most 512 entries; force tasks: at most
    // grid + i-tiles of at least 16
    const long long part_cap = (long long)H->grid * 512 + (long long)n + 512;
    const int task_cap = H->grid + (int)(n / 16) + 2;
    size_t off = 0;
    const size_t o_hdr = off;
    off = align256(off + sizeof(HmClock));
    const size_t o_rec = off;
    off = align256(off + sizeof(HmWord) * HM_RSLOTS * H->nseg);
    const size_t o_list = off;
    off = align256(off + (size_t)HM_RSLOTS * H->nseg * HM_SEG);
    const size_t o_ack = off;
    off = align256(off + sizeof(unsigned) * (size_t)H->grid);
    const size_t o_sums = off;
    off = align256(off + sizeof(HmWord) * HM_SUMW * HM_SMALL * (size_t)H->grid);
    const size_t o_sflag = off;
    off = align256(off + sizeof(unsigned) * H->nseg);
    const size_t o_tflag = off;
    off = align256(off + sizeof(unsigned) * ((size_t)task_cap + H->grid));
    const size_t o_act = off;
    off = align256(off + sizeof(int) * n);
    const size_t o_irec = off;
    off = align256(off + sizeof(G6I) * n);
    const size_t o_jpred = off;
    off = align256(off + sizeof(G6PredJ) * n);
    const size_t o_out = off;
    off = align256(off + sizeof(G6Out) * n);
    const size_t o_part = off;
    off = align256(off + sizeof(G6Out) * (size_t)part_cap);
    const size_t o_en = off;
    off = align256(off + 2 * sizeof(double));
    PGB_CUDA_OR(g_err, LIB, H->work.reserve(off), return false);
    unsigned char* w = H->work.p;
    H->W.clk = (HmClock*)(w + o_hdr);
    H->W.rec = (HmWord*)(w + o_rec);
    H->W.seg_list = w + o_list;
    H->W.ack = (unsigned*)(w + o_ack);
    H->W.sums = (HmWord*)(w + o_sums);
    H->W.chunks = H->grid;
    H->W.seg_flag = (unsigned*)(w + o_sflag);
    H->W.task_flag = (unsigned*)(w + o_tflag);
    H->W.task_cap = task_cap;
    H->W.active = (int*)(w + o_act);
    H->W.irec = (G6I*)(w + o_irec);
    H->W.jpred = (G6PredJ*)(w + o_jpred);
    H->W.out = (G6Out*)(w + o_out);
    H->W.partial = (G6Out*)(w + o_part);
    H->W.part_cap = part_cap;
    H->energy = (double*)(w + o_en);
    // clock, records and flags zero; the step numbers that tag them start at 1
    PGB_CUDA_OR(g_err, LIB, cudaMemsetAsync(w, 0, o_act, H->s), return false);
    return true;
}

// Wait for the stream and read the device clock; a wait that gave up is an error.
bool hm_sync_clock(pgb6_hermite* H) {
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(&H->clk, H->W.clk, sizeof(HmClock), cudaMemcpyDeviceToHost, H->s),
                return false);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(H->s), return false);
    if (H->clk.err) {
        raise(g_err, LIB, PGB_ERR_DEVICE, "hermite: a wait of the step kernel timed out");
        return false;
    }
    return true;
}

// One cooperative launch: the start-up step, or block steps while the time is below tend (at
// most max_steps).
bool hm_launch(pgb6_hermite* H, bool startup, double tend, int max_steps) {
    HmRun R;
    R.P = H->P;
    R.W = H->W;
    R.eps2 = (float)H->eps2;
    R.eta = H->eta;
    R.eta_s = H->eta_s;
    R.dtmax = H->dtmax;
    R.tend = tend;
    // the clock of the last launch, which has been read back (hm_sync_clock); every step counted one
    R.step0 = 1u + (unsigned)H->clk.bsteps;
    R.time0 = H->clk.time;
    R.t_mod0 = H->clk.t_mod;
    R.startup = startup ? 1 : 0;
    R.max_steps = max_steps;
    R.nseg = H->nseg;
    // j per force chunk at least (fewer, longer tasks mean fewer partial rows for the owners
    // to sum; N = 16384 block steps: 64 -> 114, 128 -> 120, 256 -> 123, 512 -> 108 Gint/s)
    static const int minj = env_int("PGB_HM_MINJ", 256, 16, 1 << 20);
    R.minj = minj;
    // hm_shape's chunk count of a single i-tile of at most HM_SMALL (its buffers never limit that)
    R.nch1 = std::min(H->grid, std::max(1, H->n / minj));
    R.dtinv = 1.0 / H->dtmax;
    void* args[] = {&R};
    const void* fn = hm_kernel(H->ff, startup && H->n > HM_SMALL);
    PGB_CUDA_OR(g_err, LIB, cudaLaunchCooperativeKernel(fn, dim3(H->grid), dim3(HM_NT), args, 0, H->s),
                return false);
    return true;
}

void hm_free(pgb6_hermite* H) {
    if (H->s) cudaStreamSynchronize(H->s);
    H->state.release();
    H->work.release();
    if (H->s) cudaStreamDestroy(H->s);
    H->s = nullptr;
}

constexpr int HM_STEPS_PER_LAUNCH = 1 << 16;
}  // namespace

// Create an integrator for n particles (n >= 2) and take its start-up step: every particle's
// force, jerk and potential at t = 0 and its first step (startup_sgmotion).  eps2: softening^2;
// eta / eta_s: accuracy parameters of dt_criterion / dt_startup; dtmax: the largest step and the
// interval after which the times restart from 0 (the reference's dtstar).
PGB_EXPORT int pgb6_hermite_create(pgb6_hermite** out, int n, const double* mass, const double (*pos)[3],
                                   const double (*vel)[3], double eps2, double eta, double eta_s, double dtmax) {
    if (!out || n < 2 || n > HM_MAXSEG * HM_SEG || !mass || !pos || !vel || !(eps2 >= 0.0) || !(eta > 0.0) ||
        !(eta_s > 0.0) || !(dtmax > 0.0)) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_create: bad arguments (n %d, eps2 %g, eta %g, eta_s %g, dtmax %g)",
              n, eps2, eta, eta_s, dtmax);
        return PGB_ERR_ARG;
    }
    *out = nullptr;
    if (!ensure_device()) return PGB_ERR_NOGPU;
    auto* H = new pgb6_hermite();
    H->n = n;
    H->eps2 = eps2;
    H->eta = eta;
    H->eta_s = eta_s;
    H->dtmax = dtmax;
    H->ff = dx_ff();
    bool ok = cudaStreamCreateWithFlags(&H->s, cudaStreamNonBlocking) == cudaSuccess;
    if (!ok) raise(g_err, LIB, PGB_ERR_CUDA, "pgb6_hermite_create: stream creation failed");
    ok = ok && hm_alloc(H);
    if (ok) {
        const size_t nn = (size_t)n;
        // t, dt, pot zero; acc, jrk zero; mass, pos, vel from the caller
        ok = cudaMemsetAsync(H->state.p, 0, 16 * nn * sizeof(double), H->s) == cudaSuccess &&
             cudaMemcpyAsync(H->P.mass, mass, nn * sizeof(double), cudaMemcpyHostToDevice, H->s) == cudaSuccess &&
             cudaMemcpyAsync(H->P.pos, pos, 3 * nn * sizeof(double), cudaMemcpyHostToDevice, H->s) == cudaSuccess &&
             cudaMemcpyAsync(H->P.vel, vel, 3 * nn * sizeof(double), cudaMemcpyHostToDevice, H->s) == cudaSuccess;
        if (!ok) raise(g_err, LIB, PGB_ERR_CUDA, "pgb6_hermite_create: upload failed");
    }
    ok = ok && hm_launch(H, true, 0.0, 1) && hm_sync_clock(H);
    const int bad = ok ? H->clk.bad : 0;
    if (ok && bad) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_create: the start-up step of %d particles is below dtmax/2^51",
              bad);
        hm_free(H);
        delete H;
        return PGB_ERR_ARG;
    }
    if (!ok) {
        hm_free(H);
        delete H;
        return PGB_ERR_CUDA;
    }
    *out = H;
    return PGB_OK;
}

// One block step: the particles with the smallest t + dt advance to it.  *time (optional): the
// global time after the step; *ni (optional): the number of particles advanced.
PGB_EXPORT int pgb6_hermite_step(pgb6_hermite* H, double* time, int* ni) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_step: null integrator");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    if (!hm_launch(H, false, INFINITY, 1) || !hm_sync_clock(H)) return H->clk.err ? PGB_ERR_DEVICE : PGB_ERR_CUDA;
    if (time) *time = H->clk.time;
    if (ni) *ni = H->clk.ni;
    return PGB_OK;
}

// Block steps while the global time is below tend (banana01.c:146 loop condition, evaluated on
// the device before every step).  *psteps / *bsteps (optional): the particle steps and block
// steps this call took.
PGB_EXPORT int pgb6_hermite_advance(pgb6_hermite* H, double tend, long long* psteps, long long* bsteps) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_advance: null integrator");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    const long long p0 = H->clk.psteps, b0 = H->clk.bsteps;
    while (H->clk.time < tend)
        if (!hm_launch(H, false, tend, HM_STEPS_PER_LAUNCH) || !hm_sync_clock(H))
            return H->clk.err ? PGB_ERR_DEVICE : PGB_ERR_CUDA;
    if (psteps) *psteps = H->clk.psteps - p0;
    if (bsteps) *bsteps = H->clk.bsteps - b0;
    return PGB_OK;
}

PGB_EXPORT double pgb6_hermite_time(pgb6_hermite* H) { return H ? H->clk.time : 0.0; }

// The limit, in SM cycles, of every wait of the step kernel (segment records and their
// acknowledgements, chunk sums, segment and task flags); cycles <= 0 restores the default (about a
// second).  A wait that runs out sets the integrator's error word: every CTA returns at its next wait,
// the call reports PGB_ERR_DEVICE and the integrator is unusable afterwards (its records and flags no longer
// agree).  For fault-handling tests; a production run keeps the default.
PGB_EXPORT int pgb6_hermite_set_wait_limit(pgb6_hermite* H, long long cycles) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_set_wait_limit: null integrator");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    const long long v = cycles > 0 ? cycles : 0;
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(&H->W.clk->spin_limit, &v, sizeof v, cudaMemcpyHostToDevice, H->s),
                return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(H->s), return PGB_ERR_CUDA);
    return PGB_OK;
}

// The step kernel's failure record, read from the device: *gave_up (a wait ran out, so the
// integrator is unusable), *exits (CTAs that have returned from the kernel, over every launch
// so far) and *grid (CTAs per launch).  Any pointer may be NULL.
PGB_EXPORT int pgb6_hermite_wait_status(pgb6_hermite* H, int* gave_up, int* exits, int* grid) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_wait_status: null integrator");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    HmClock c;
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(&c, H->W.clk, sizeof c, cudaMemcpyDeviceToHost, H->s),
                return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(H->s), return PGB_ERR_CUDA);
    if (gave_up) *gave_up = c.err;
    if (exits) *exits = c.exits;
    if (grid) *grid = H->grid;
    return PGB_OK;
}

// The particle state (any pointer may be NULL): t, dt, pos, vel, acc, jerk, pot as the
// reference's struct Particle holds them (jerk and pot with float values).
PGB_EXPORT int pgb6_hermite_get(pgb6_hermite* H, double* t, double* dt, double (*pos)[3], double (*vel)[3],
                                double (*acc)[3], double (*jrk)[3], double* pot) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_get: null integrator");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    const size_t n = (size_t)H->n;
    struct {
        void* dst;
        const double* src;
        size_t cnt;
    } cp[7] = {{t, H->P.t, n},           {dt, H->P.dt, n},          {pos, H->P.pos, 3 * n}, {vel, H->P.vel, 3 * n},
               {acc, H->P.acc, 3 * n},   {jrk, H->P.jrk, 3 * n},    {pot, H->P.pot, n}};
    for (auto& c : cp)
        if (c.dst)
            PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(c.dst, c.src, c.cnt * sizeof(double), cudaMemcpyDeviceToHost, H->s),
                        return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(H->s), return PGB_ERR_CUDA);
    return PGB_OK;
}

// The last block step's active particles (index order) and the force, jerk and potential the
// force phase returned for them (before the corrector's rounding of jerk and pot to float).
// Returns the number of active particles, or a negative error code.
PGB_EXPORT int pgb6_hermite_last_step(pgb6_hermite* H, int* active, double (*acc)[3], double (*jrk)[3],
                                      double* pot) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_last_step: null integrator");
        return -PGB_ERR_ARG;
    }
    if (!ensure_device()) return -PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    const int ni = H->clk.ni;
    std::vector<G6Out> o((size_t)ni);
    if (active)
        PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(active, H->W.active, ni * sizeof(int), cudaMemcpyDeviceToHost, H->s),
                    return -PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(o.data(), H->W.out, ni * sizeof(G6Out), cudaMemcpyDeviceToHost, H->s),
                return -PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(H->s), return -PGB_ERR_CUDA);
    for (int k = 0; k < ni; k++) {
        if (acc) {
            acc[k][0] = o[k].ax;
            acc[k][1] = o[k].ay;
            acc[k][2] = o[k].az;
        }
        if (jrk) {
            jrk[k][0] = o[k].jx;
            jrk[k][1] = o[k].jy;
            jrk[k][2] = o[k].jz;
        }
        if (pot) pot[k] = o[k].pot;
    }
    return ni;
}

// Kinetic and potential energy of the current state (calc_energy.c:9-33), FP64, fixed order.
PGB_EXPORT int pgb6_hermite_energy(pgb6_hermite* H, double* ek, double* ew) {
    if (!H) {
        raise(g_err, LIB, PGB_ERR_ARG, "pgb6_hermite_energy: null integrator");
        return PGB_ERR_ARG;
    }
    if (!ensure_device()) return PGB_ERR_NOGPU;
    std::lock_guard<std::mutex> g(H->mu);
    double e[2] = {0.0, 0.0};
    hm_energy_kernel<<<1, 1024, 0, H->s>>>(H->P, H->energy);
    PGB_CUDA_OR(g_err, LIB, cudaGetLastError(), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaMemcpyAsync(e, H->energy, sizeof e, cudaMemcpyDeviceToHost, H->s), return PGB_ERR_CUDA);
    PGB_CUDA_OR(g_err, LIB, cudaStreamSynchronize(H->s), return PGB_ERR_CUDA);
    if (ek) *ek = e[0];
    if (ew) *ew = e[1];
    return PGB_OK;
}

// Particle and block steps since creation (the start-up step counts n and 1).
PGB_EXPORT void pgb6_hermite_counts(pgb6_hermite* H, long long* psteps, long long* bsteps) {
    if (psteps) *psteps = H ? H->clk.psteps : 0;
    if (bsteps) *bsteps = H ? H->clk.bsteps : 0;
}

// The integrator's CUDA stream (for callers that time it with CUDA events or order their own
// work after it).
PGB_EXPORT void* pgb6_hermite_stream(pgb6_hermite* H) { return H ? (void*)H->s : nullptr; }

// Pair interactions of the force phases so far (active particles x n) and the steps taken with
// each force decomposition (i-tile 16, 32, 64, 128, 512); any pointer may be NULL.
PGB_EXPORT void pgb6_hermite_stats(pgb6_hermite* H, long long* pairs, long long* steps_by_tile) {
    if (pairs) *pairs = H ? H->clk.force_pairs : 0;
    for (int k = 0; k < 5; k++)
        if (steps_by_tile) steps_by_tile[k] = H ? H->clk.variant_steps[k] : 0;
}

PGB_EXPORT void pgb6_hermite_destroy(pgb6_hermite* H) {
    if (!H) return;
    if (g_device >= 0) cudaSetDevice(g_device);
    hm_free(H);
    delete H;
}
