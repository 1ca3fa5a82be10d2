// pgb_g6_small.cuh -- the Hermite force kernel of the drop-in API's small calls: at most 64
// i-particles (the reference's g6calc_lasthalf* take at most NPIPES = 48 per call,
// PG6/libpg6/avx_type.h:1) against the whole j-memory.
//
// Such a call has far too few i-particles to fill the GPU by i, so the j-range is cut into one
// chunk per CTA (gridDim.x chunks, every CTA resident) and the partial sums are reduced in
// three fixed-order stages, none of which round-trips through a task scheduler:
//   1. the JL j-lanes of the CTA, word by word through shared memory: groups of lanes in lane
//      order, then the groups (all lanes one after another took 2.5 us of a 7 x 1024 call, this
//      0.8);
//   2. the CTAs of a thread-block cluster (CL consecutive chunks), through distributed shared
//      memory: CTA `rank` sums its slice of the words over the cluster's CTAs (rank order) and
//      writes the cluster's row of partial sums;
//   3. the cluster rows: slice r of the words of every row is written by rank r of each
//      cluster, and the rank-r CTA that arrives last on a per-slice counter sums the slice over
//      the rows (reduce_rows: fixed row order) and writes the final scaled result -- CL CTAs
//      share the final stage and no cluster waits for another.  A call of one cluster ends with
//      stage 2.
// The i-records come in the parameter block (no upload; staged to shared memory with
// broadcast reads) and the j-chunks are a pure function of (blockIdx, nj, gridDim), so a call
// is one launch.  The result is deterministic for a given
// grid and cluster size.  Per pair the arithmetic is g6_pair(), identical to g6_kernel.
// The results go to the host as numbered words (G6HostWords).  Latency bounds the kernel: 4 us for
// 7 x 1024 (1.2 to the last pair), 14 us for 48 x 65536 (7.3 to the last pair, 3 in the clusters, 2.5 in
// the last stage), before 14 and 22 us to the flag behind the results' fence.
#pragma once

#include <cooperative_groups.h>

#include "pgb_g6_kernels.cuh"

namespace pgb {

struct G6SmallArgs {
    const G6PredJ* jpred;
    float eps2;
    int ni, nj;        // i-particles (<= ISL) and j-records [0, nj)
    G6Out* partial;    // [gridDim.x / CL][ISL] cluster sums
    int* counter;      // [cluster size] arrivals per word slice; zero at launch, reset by the last
    int* nb_count;     // neighbour lists (NBL), indexed by i
    int* nb_list;
    int nb_maxlen;
    // final results in mapped host memory: result word f (16 bytes, 4 to a G6Out) as words[2f],
    // words[2f + 1], each two 32-bit values with the call's number after each
    uint4* words;
    unsigned seq;
};

// A result word for the host.  Every 8 bytes carry the call's number themselves, so the host takes a
// word as soon as it is there and no store waits for another: with plain words, a system fence and a
// flag after it the fence alone took 6.3 us of the 14 us of a call of 7 i against 1024 j.
struct G6HostWords {
    uint4* words;
    unsigned seq;
    __device__ __forceinline__ void operator()(int f, double2 v) const {
        const unsigned long long x = __double_as_longlong(v.x), y = __double_as_longlong(v.y);
        __stwt(words + 2 * f, make_uint4((unsigned)x, seq, (unsigned)(x >> 32), seq));
        __stwt(words + 2 * f + 1, make_uint4((unsigned)y, seq, (unsigned)(y >> 32), seq));
    }
};

constexpr int G6_SMALL_MAXI = 64;
constexpr int SMALL_CL_MAX = 8;   // CTAs per cluster at most (the portable limit)

// The i-records of a small call, passed by value in the kernel's parameter block: no separate
// upload (and no host-to-device copy latency) for a call of up to G6_SMALL_MAXI i-particles.
template <int ISL>
struct G6IBlock {
    G6I rec[ISL];
};

template <int ISL, int JL, bool FF, bool NN, bool NBL>
__global__ void __launch_bounds__(ISL * JL, 2)
    g6_small_kernel(const G6SmallArgs A, const __grid_constant__ G6IBlock<ISL> ib) {
    namespace cg = cooperative_groups;
    constexpr int NT = ISL * JL;
    static_assert(ISL <= G6_SMALL_MAXI, "i-slots within the i-block");
    __shared__ __align__(16) unsigned char smem[NT * sizeof(G6Out)];  // j tile, then per-thread sums
    __shared__ double2 cta_w[4 * ISL];                                 // this CTA's sums, by word
    __shared__ G6I s_i[ISL];
    __shared__ int s_flag;
    G6PredJ* sj = reinterpret_cast<G6PredJ*>(smem);
    const int slot = threadIdx.x % ISL, jl = threadIdx.x / ISL;
    const int nch = gridDim.x, c = blockIdx.x;
    const int j0 = (int)((long long)c * A.nj / nch), j1 = (int)((long long)(c + 1) * A.nj / nch);

    // the first j tile's loads go out first; meanwhile the i-records are staged from the
    // parameter block into shared memory with warp-uniform (broadcast) constant-bank reads --
    // per-thread reads of different records would serialise in the constant cache
    int jt = j0;
    int nt = min(NT, j1 - jt);
    G6PredJ jr;
    if (threadIdx.x < nt) jr = A.jpred[jt + threadIdx.x];
    for (int r = threadIdx.x / 32; r < A.ni; r += NT / 32) {
        const uint4* src = reinterpret_cast<const uint4*>(&ib.rec[r]);
        const uint4 w0 = src[0], w1 = src[1], w2 = src[2];
        if ((threadIdx.x & 31) == 0) {
            uint4* d = reinterpret_cast<uint4*>(&s_i[r]);
            d[0] = w0;
            d[1] = w1;
            d[2] = w2;
        }
    }
    if (threadIdx.x < nt) sj[threadIdx.x] = jr;
    __syncthreads();

    const int ii = slot < A.ni ? slot : 0;
    const G6I P = s_i[ii];
    const float hinv = g6_hkey(slot < A.ni, P.h2);
    double S[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    float kmin = G6_KEY0;  // gravity_kernel2's initial key and index (:495-496)
    int kadr = -1;
    int* nbc = NBL ? A.nb_count + ii : nullptr;
    int* nbl = NBL ? A.nb_list + (size_t)ii * A.nb_maxlen : nullptr;

    for (;;) {
        G6Acc a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
        for (int j = jl; j < nt; j += JL)
            g6_pair<FF, NN, NBL>(sj[j], jt + j, P.p, P.vx, P.vy, P.vz, P.id, A.eps2, hinv, a, kmin, kadr, nbc, nbl,
                                 A.nb_maxlen);
        S[0] += (double)a.ax;
        S[1] += (double)a.ay;
        S[2] += (double)a.az;
        S[3] += (double)a.jx;
        S[4] += (double)a.jy;
        S[5] += (double)a.jz;
        S[6] += (double)a.pot;
        jt += NT;
        if (jt >= j1) break;
        nt = min(NT, j1 - jt);
        __syncthreads();
        if (threadIdx.x < nt) sj[threadIdx.x] = A.jpred[jt + threadIdx.x];
        __syncthreads();
    }

    // 1. j-lanes, word by word: thread (g, wd, s) sums word wd of slot s over its NT / (4 ISL)-th of
    //    the lanes in order, then the parts are added in order
    constexpr int NW = 4 * ISL, NG = NT / NW, PER = (JL + NG - 1) / NG;
    double2* sw = reinterpret_cast<double2*>(smem);   // [4][NT], word by word: no bank conflicts
    const G6HostWords host{A.words, A.seq};
    const int nw = 4 * A.ni;
    const int wd = (int)threadIdx.x / ISL % 4, g = (int)threadIdx.x / NW;
    __syncthreads();
    sw[threadIdx.x] = make_double2(S[0], S[1]);
    sw[NT + threadIdx.x] = make_double2(S[2], S[3]);
    sw[2 * NT + threadIdx.x] = make_double2(S[4], S[5]);
    sw[3 * NT + threadIdx.x] = make_double2(
        S[6], __longlong_as_double((long long)((unsigned long long)(unsigned)kadr << 32 |
                                               (unsigned)__float_as_int(kmin))));
    __syncthreads();
    const bool mine = g < NG && slot < A.ni, w3 = wd == 3;
    double2 v = word_zero(w3);
    if (mine) {
        const double2* col = sw + wd * NT + slot;
        double2 u[PER];
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (g * PER + k < JL) u[k] = col[(g * PER + k) * ISL];
        v = u[0];
#pragma unroll
        for (int k = 1; k < PER; k++)
            if (g * PER + k < JL) v = word_add(v, u[k], w3);
    }
    __syncthreads();
    if (mine && g > 0) sw[threadIdx.x] = v;
    __syncthreads();
    if (mine && g == 0) {
#pragma unroll
        for (int k = 1; k < NG; k++) v = word_add(v, sw[k * NW + threadIdx.x], w3);
        const int f = 4 * slot + wd;
        if (nch == 1) host(f, word_finish(v, w3));   // the whole call in one CTA
        cta_w[f] = v;
    }
    if (nch == 1) return;

    // 2. the cluster: CTA `rank` reduces words [f0, f1) over the cluster's CTAs, in rank order,
    //    into the cluster's row (the only cluster: into the result)
    cg::cluster_group cl = cg::this_cluster();
    const int CL = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    cl.sync();
    const int nclus = nch / CL;
    const int f0 = rank * nw / CL, f1 = (rank + 1) * nw / CL;
    const int f = f0 + (int)threadIdx.x;
    if (f < f1) {
        const bool fw3 = (f & 3) == 3;
        double2 q[SMALL_CL_MAX];
#pragma unroll
        for (int k = 0; k < SMALL_CL_MAX; k++)
            if (k < CL) q[k] = *cl.map_shared_rank(&cta_w[f], k);
        double2 t = q[0];
#pragma unroll
        for (int k = 1; k < SMALL_CL_MAX; k++)
            if (k < CL) t = word_add(t, q[k], fw3);
        if (nclus == 1) host(f, word_finish(t, fw3));
        else reinterpret_cast<double2*>(A.partial + (size_t)(c / CL) * ISL)[f] = t;
    }

    // 3. slice `rank` of every cluster row was written by that cluster's CTA `rank`: those CTAs
    //    arrive on counter[rank], and the last of them sums the slice over the rows in order
    if (nclus > 1) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            const int prev = atomicAdd(&A.counter[rank], 1);
            const int last = (prev == nclus - 1);
            if (last) atomicExch(&A.counter[rank], 0);
            __threadfence();
            s_flag = last;
        }
        __syncthreads();
        if (s_flag)
            reduce_rows<NT>(A.partial, (size_t)ISL, nclus, f0, f1 - f0, host, true, reinterpret_cast<double2*>(smem));
    }
    cl.sync();  // no CTA leaves while a peer may still read its cta_w
}

}  // namespace pgb
