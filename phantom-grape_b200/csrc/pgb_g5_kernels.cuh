// pgb_g5_kernels.cuh -- PG5 Newtonian (plain and symmetric softening) and quadrupole-cell
// interaction kernels for sm_100a.
//
// Work decomposition (all kernels): a persistent grid of CTAs pulls Tasks (i-tile x j-chunk)
// from a global counter.  A CTA of NT threads owns NT*IPT i-particles (IPT per thread, kept
// in registers), streams its j-chunk through shared memory in tiles of NT records (one
// coalesced 16-byte load per thread per record word), and every thread reads each j record
// with a broadcast LDS.128.  Sums are accumulated in FP32 over at most 128 terms (G5_FOLD) and
// then added into FP64 accumulators (the cross-block reduction runs in FP64).  Split j-ranges
// write FP64 partial rows; the last CTA of a group reduces them in chunk order.
//
// Formulae, with the pair scale s of 1/r (pgb::pair_scale: the MUFU estimate 1/r by default,
// -2/r in the reference's Newton-refined form with PGB_RSQRT_NEWTON):
//   pot_sum += m s,  acc_sum += (m s^3) dx,  acc = S_ACC acc_sum,  pot_raw = S_POT pot_sum
//   = -sum m/r
// i.e. the reference's GravityKernel accumulators (PG5/newton/libpg5/gravity_avx2.c:95-153:
// phi -= m/r, acc += m dx / r^3) without its 12-bit rsqrt.
#pragma once

#include "pgb_common.cuh"

namespace pgb {

struct G5Args {
    const float4* ipos;     // [.] x, y, z, eps2 of each i-particle
    const float4* jpos;     // [.] x, y, z, m of each j-particle (or cell word 0)
    const float4* jaux;     // symmetric: [.] eps2_j in .x; quad: [2*nc] (q0 q1 q2 q3)(q4 q5 - -)
    const int* jidx;        // nullptr: task j-ranges address jpos/jaux directly; else they address
                            // this index list (interaction lists of a tree: j = jidx[k])
    const Task* tasks;
    int ntasks;
    int* task_counter;      // zero before launch
    const Group* groups;
    int* group_counters;    // zero at allocation, self-cleaning
    double4* partial;       // [rows][itile]
    double4* out;           // [.] (ax, ay, az, pot_raw) per i, indexed by absolute i
    // not nullptr (the slot kernel only): the results go to mapped host memory instead, [.][4] of two
    // 32-bit values with the call's number after each
    uint4* words;
    unsigned seq;
    int itile;              // NT*IPT
    // table kind only: force-shape table (f, df/ds) in s = 2 + |dx'|^2, 2^(EXP+FRC) entries
    const float2* table;
    int tbl_size;
    int tbl_shift;          // 23 - FRC_BIT
    float r2cut;            // float with bits (1<<30) | ((tbl_size-1) << tbl_shift)
    double ascale;          // 1 / xscale
};

// kinds
enum { G5_NEWTON = 0, G5_SYMMETRIC = 1, G5_QUAD = 2, G5_TABLE = 3 };
constexpr int G5_TBL_MAX = 4096;   // largest table held in shared memory (32 KB)
// FP32 partial sums cover at most G5_FOLD terms (per thread and i) before they are added into
// the FP64 sums: the rounding of a 128-term FP32 sum stays near the level of the FP32 pair
// arithmetic, a whole 1024-record tile (the direct sum's CTA) adds several times more
// (acc 1.4e-7 rms against FP64 with 1024-term sums, 4.7e-8 with 64-term sums on N = 16384)
constexpr int G5_FOLD = 128;

template <int KIND>
struct JWords { static constexpr int n = (KIND == G5_SYMMETRIC) ? 2 : (KIND == G5_QUAD ? 3 : 1); };

// FP32 block sums per i: (acc, pot) for the point-mass and table kinds; the quadrupole kind
// keeps [0..2] sum (w dr + K s^5 v), [3] sum m s, [4] sum K s^5 D (g5_quad_pair), which g5_fold
// scales and combines into (acc, phi_p + phi_q).
template <int KIND>
struct NAcc { static constexpr int n = KIND == G5_QUAD ? 5 : 4; };

// The cells' moments as staged in shared memory, Q' = G5_QSCALE Q, and the constant K of the
// (Q dr) r^-5 term (g5_quad_pair).  For s = -2/r: Q' = (5/32) Q, which makes the coefficient of
// the monopole and of the D s^7 term of the acceleration the same, and K = -8/5 puts the
// (Q dr) r^-5 term into the same sums; the sums are scaled by G5_QACC (acc) and G5_QP3, G5_QP4
// (phi_p + phi_q = G5_QP3 a[3] + G5_QP4 a[4]).  For s = 1/r the moments are staged 16 times
// larger and K is a quarter: every term is the same term times an exact power of two (K is the
// FP32 -8/5 divided by 4), and the constants remove them.
#ifdef PGB_RSQRT_NEWTON
constexpr float G5_QSCALE = 0.15625f;
constexpr float G5_QK = -1.6f;
constexpr double G5_QACC = -0.125, G5_QP3 = -0.5, G5_QP4 = -(0.1 / (double)(-1.6f));
#else
constexpr float G5_QSCALE = 2.5f;
constexpr float G5_QK = -0.4f;
constexpr double G5_QACC = 1.0, G5_QP3 = 1.0, G5_QP4 = 8.0 * (0.1 / (double)(-1.6f));
#endif

__device__ __forceinline__ float4 scale4(float4 v, float f) {
    return make_float4(f * v.x, f * v.y, f * v.z, f * v.w);
}

// One FP32 block sum (a[NAcc]) into the FP64 sums S = (ax, ay, az, pot) -- pot as each kind's
// raw sum (the quadrupole kind's +sum(phi_p + phi_q), which needs no finishing).
template <int KIND>
__device__ __forceinline__ void g5_fold(double (&S)[4], const float* a) {
    if constexpr (KIND == G5_QUAD) {
#pragma unroll
        for (int c = 0; c < 3; c++) S[c] += G5_QACC * (double)a[c];
        S[3] += G5_QP3 * (double)a[3] + G5_QP4 * (double)a[4];
    } else {
#pragma unroll
        for (int c = 0; c < 4; c++) S[c] += (double)a[c];
    }
}

// The same for paired sums: lane k of each a2[c] (k < 0: both lanes, x then y).
template <int KIND>
__device__ __forceinline__ void g5_fold2(double (&S)[4], const float2* a2, int k) {
    float a[2][NAcc<KIND>::n];
#pragma unroll
    for (int c = 0; c < NAcc<KIND>::n; c++) {
        a[0][c] = k == 1 ? a2[c].y : a2[c].x;
        a[1][c] = a2[c].y;
    }
    if (k < 0) {
        if constexpr (KIND == G5_QUAD) {
#pragma unroll
            for (int c = 0; c < 3; c++) S[c] += G5_QACC * ((double)a[0][c] + (double)a[1][c]);
            S[3] += G5_QP3 * ((double)a[0][3] + (double)a[1][3]) + G5_QP4 * ((double)a[0][4] + (double)a[1][4]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++) S[c] = S[c] + (double)a[0][c] + (double)a[1][c];
        }
    } else {
        g5_fold<KIND>(S, a[0]);
    }
}

// A cell's two moment words into shared memory (word 1 at sq[0], word 2 at sq[1]), scaled.
__device__ __forceinline__ void g5_stage_quad(float4* sq, const float4* jaux, int jj) {
    sq[0] = scale4(jaux[2 * jj], G5_QSCALE);
    sq[1] = scale4(jaux[2 * jj + 1], G5_QSCALE);
}

// Table lookup of the cutoff force (PG5/table/libpg5/gravity_kernel_avx2.c:70-124):
// s = min(2 + |dx'|^2, r2cut); the table bin is the float bit pattern of s shifted right by
// 23-FRC_BIT (the exponent and FRC_BIT leading mantissa bits); the bin's node is s with its
// low bits cleared; f = T[bin].x + (s - node) T[bin].y.  `tab` is pre-offset by the bin of 2.0
// so that it can be indexed by the shifted bits directly.  s >= 2 and the clamp (fminf returns
// r2cut for a NaN s) keep every index inside the table.
__device__ __forceinline__ void g5_table_pair(float4 J, float xi, float yi, float zi, const float2* tab,
                                              int shift, float r2cut, float (&a)[4]) {
    float dx = J.x - xi, dy = J.y - yi, dz = J.z - zi;
    float s = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, 2.0f)));
    s = fminf(s, r2cut);
    unsigned u = __float_as_uint(s);
    float node = __uint_as_float((u >> shift) << shift);
    float2 T = tab[u >> shift];
    float f = __fmaf_rn(s - node, T.y, T.x);
    float mf = J.w * f;
    a[0] = __fmaf_rn(mf, dx, a[0]);
    a[1] = __fmaf_rn(mf, dy, a[1]);
    a[2] = __fmaf_rn(mf, dz, a[2]);
}

// The quadrupole cell (c_GravityKernel, PG5/newton_quad/quad/quad_avx2.c:35-149; FP64 form
// source.cpp:1160-1184): with the pair scale s (below q; 1/r by default) and the moments staged
// as Q' = G5_QSCALE Q,
//   v = Q' dr,  D = dr . v,  w = s^3 (m + D s^4),  p = K s^5
//   acc = dr (m r^-3 + (5/2) (dr.Q.dr) r^-7) - (Q dr) r^-5 = G5_QACC (w dr + p v)
//   phi_p + phi_q = m r^-1 + (1/2) (dr.Q.dr) r^-5 = G5_QP3 (m s) + G5_QP4 (p D)
// (s = 1/r: Q' = (5/2) Q, K = -2/5, G5_QACC = 1, G5_QP3 = 1, G5_QP4 = -1/2; s = -2/r: (5/32) Q,
// -8/5, -1/8, -1/2, -1/(10 K)).  34 FP32 operations per pair with s = 1/r (36 with the Newton
// step; the r^-1, r^-2, r^-5 form takes 38); the block sums of w dr + p v, m s and p D are
// scaled and combined in FP64 by g5_fold.  K rounded to FP32 weighs the (Q dr) term 1.5e-8
// (relative) heavier.
__device__ __forceinline__ void g5_quad_pair(float dx, float dy, float dz, float m, float4 Q0, float4 Q1,
                                             float e, float (&a)[5]) {
    // Q0 = q00 q01 q02 q11, Q1 = q12 q22 - -
    const float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, e)));
    const float q = pair_scale(r2);
    const float vx = __fmaf_rn(Q0.z, dz, __fmaf_rn(Q0.y, dy, Q0.x * dx));
    const float vy = __fmaf_rn(Q1.x, dz, __fmaf_rn(Q0.w, dy, Q0.y * dx));
    const float vz = __fmaf_rn(Q1.y, dz, __fmaf_rn(Q1.x, dy, Q0.z * dx));
    const float D = __fmaf_rn(dz, vz, __fmaf_rn(dy, vy, dx * vx));
    const float q2 = q * q, q3 = q2 * q, q4 = q2 * q2, p = q4 * (G5_QK * q);
    const float w = q3 * __fmaf_rn(D, q4, m);
    a[0] = __fmaf_rn(w, dx, __fmaf_rn(p, vx, a[0]));
    a[1] = __fmaf_rn(w, dy, __fmaf_rn(p, vy, a[1]));
    a[2] = __fmaf_rn(w, dz, __fmaf_rn(p, vz, a[2]));
    a[3] = __fmaf_rn(m, q, a[3]);
    a[4] = __fmaf_rn(p, D, a[4]);
}

template <int KIND, int NT>
__device__ __forceinline__ void g5_interact(const float4* sj, int j, float xi, float yi, float zi,
                                            float ei, float (&a)[NAcc<KIND>::n]) {
    float4 J = sj[j];
    float dx = J.x - xi, dy = J.y - yi, dz = J.z - zi;
    if constexpr (KIND == G5_QUAD) {
        g5_quad_pair(dx, dy, dz, J.w, sj[NT + 2 * j], sj[NT + 2 * j + 1], ei, a);
    } else {
        float e = ei;
        if constexpr (KIND == G5_SYMMETRIC) e += sj[NT + j].x;  // GravityKernel0
        float r2 = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, e)));
        float q = pair_scale(r2);
        float mq = J.w * q;
        float q2 = q * q;
        float mq3 = mq * q2;
        a[3] += mq;
        a[0] = __fmaf_rn(mq3, dx, a[0]);
        a[1] = __fmaf_rn(mq3, dy, a[1]);
        a[2] = __fmaf_rn(mq3, dz, a[2]);
    }
}

__device__ __forceinline__ float& lane_of(float2& v, int k) { return k ? v.y : v.x; }

// Two i-particles of a thread (configurations with IPT >= 2) against one j record: the per-i chains exactly as g5_interact / g5_table_pair, the
// accumulations of the two i issued as paired FP32 instructions (FFMA2 / FADD2, each lane rounded
// as the scalar instruction: results bit-identical to two g5_interact calls), except the
// quadrupole kind's, whose sums stay scalar (g5_quad_pair per i: its many other FMAs already
// load the FMA pipe's heavy half, which alone executes paired instructions; paired sums measured
// 2 % slower).  a2[c] holds component c of both i.
template <int KIND, int NT>
__device__ __forceinline__ void g5_interact2(const float4* sj, int j, const float* xi, const float* yi,
                                             const float* zi, const float* ei, const float2* tab, int shift,
                                             float r2cut, float2 (&a2)[NAcc<KIND>::n]) {
    const float4 J = sj[j];
    if constexpr (KIND == G5_QUAD) {
        const float4 Q0 = sj[NT + 2 * j];
        const float4 Q1 = sj[NT + 2 * j + 1];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            float a[5];
#pragma unroll
            for (int c = 0; c < 5; c++) a[c] = lane_of(a2[c], k);
            g5_quad_pair(J.x - xi[k], J.y - yi[k], J.z - zi[k], J.w, Q0, Q1, ei[k], a);
#pragma unroll
            for (int c = 0; c < 5; c++) lane_of(a2[c], k) = a[c];
        }
    } else {
        float dx[2], dy[2], dz[2], s0[2], s3[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            dx[k] = J.x - xi[k];
            dy[k] = J.y - yi[k];
            dz[k] = J.z - zi[k];
            if constexpr (KIND == G5_TABLE) {
                float s = __fmaf_rn(dz[k], dz[k], __fmaf_rn(dy[k], dy[k], __fmaf_rn(dx[k], dx[k], 2.0f)));
                s = fminf(s, r2cut);
                unsigned u = __float_as_uint(s);
                float node = __uint_as_float((u >> shift) << shift);
                float2 T = tab[u >> shift];
                float f = __fmaf_rn(s - node, T.y, T.x);
                s0[k] = J.w * f;
            } else {
                float e = ei[k];
                if constexpr (KIND == G5_SYMMETRIC) e += sj[NT + j].x;
                float r2 = __fmaf_rn(dz[k], dz[k], __fmaf_rn(dy[k], dy[k], __fmaf_rn(dx[k], dx[k], e)));
                float q = pair_scale(r2);
                float mq = J.w * q;
                float q2 = q * q;
                s3[k] = mq;
                s0[k] = mq * q2;
            }
        }
        const float2 M = make_float2(s0[0], s0[1]);
        a2[0] = __ffma2_rn(M, make_float2(dx[0], dx[1]), a2[0]);
        a2[1] = __ffma2_rn(M, make_float2(dy[0], dy[1]), a2[1]);
        a2[2] = __ffma2_rn(M, make_float2(dz[0], dz[1]), a2[2]);
        if constexpr (KIND != G5_TABLE) a2[3] = __fadd2_rn(a2[3], make_float2(s3[0], s3[1]));
    }
}

// ---- j-paired forms -------------------------------------------------------------------------
// One i-particle against two consecutive j records (a "j-pair"), the j-tile held in shared memory
// as one array per field, so that a 16-byte shared load returns a field of four consecutive j and
// every paired FP32 operand is a natural register pair: (j, j+1) for the j fields, a
// loop-invariant (v, v) for the i position.  Every FP32 operation issues paired (FADD2 / FMUL2 /
// FFMA2: two lanes an instruction, each rounded as the scalar one); only the rsqrt, the table
// look-up and the clamp run per lane.  Per pair the arithmetic is g5_interact's / g5_table_pair's,
// operation for operation: the two lanes of an accumulator sum the even and the odd j.
__device__ __forceinline__ void g5_newton_jpair(float2 X, float2 Y, float2 Z, float2 M, float2 nx, float2 ny,
                                                float2 nz, float2 e, float2 (&a)[4]) {
    const float2 dx = __fadd2_rn(X, nx), dy = __fadd2_rn(Y, ny), dz = __fadd2_rn(Z, nz);
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, e)));
    const float2 q = make_float2(pair_scale(r2.x), pair_scale(r2.y));
    const float2 mq = __fmul2_rn(M, q);
    const float2 mq3 = __fmul2_rn(mq, __fmul2_rn(q, q));
    a[3] = __fadd2_rn(a[3], mq);
    a[0] = __ffma2_rn(mq3, dx, a[0]);
    a[1] = __ffma2_rn(mq3, dy, a[1]);
    a[2] = __ffma2_rn(mq3, dz, a[2]);
}

// The cutoff force (g5_table_pair): `tab` is the shared-memory address of the table less the byte
// offset of the entry of 2.0, so that the node's bits shifted right by shift - 3 are the entry's
// byte offset (an entry is 8 bytes).  s - node is formed as node * (-1) + s, which is exact.
__device__ __forceinline__ void g5_table_jpair(float2 X, float2 Y, float2 Z, float2 M, float2 nx, float2 ny,
                                               float2 nz, unsigned tab, int shift3, unsigned nodemask, float r2cut,
                                               float2 (&a)[4]) {
    const float2 dx = __fadd2_rn(X, nx), dy = __fadd2_rn(Y, ny), dz = __fadd2_rn(Z, nz);
    float2 s = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, make_float2(2.0f, 2.0f))));
    s = make_float2(fminf(s.x, r2cut), fminf(s.y, r2cut));
    const unsigned u0 = __float_as_uint(s.x) & nodemask, u1 = __float_as_uint(s.y) & nodemask;
    float2 t0, t1;
    asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(t0.x), "=f"(t0.y) : "r"(tab + (u0 >> shift3)));
    asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(t1.x), "=f"(t1.y) : "r"(tab + (u1 >> shift3)));
    const float2 d = __ffma2_rn(make_float2(__uint_as_float(u0), __uint_as_float(u1)), make_float2(-1.0f, -1.0f), s);
    // per lane: an entry's (f, df/ds) arrive as a register pair, which a paired FMA over the two
    // entries would first have to be transposed
    const float2 mf = __fmul2_rn(M, make_float2(__fmaf_rn(d.x, t0.y, t0.x), __fmaf_rn(d.y, t1.y, t1.x)));
    a[0] = __ffma2_rn(mf, dx, a[0]);
    a[1] = __ffma2_rn(mf, dy, a[1]);
    a[2] = __ffma2_rn(mf, dz, a[2]);
}

// Q = (q00 q01 q02 q11 q12 q22) of the two cells, as pairs, staged as Q' = G5_QSCALE Q: the
// arithmetic of g5_quad_pair with every FP32 operation paired (the moment products, D, r^2, the
// factors q^2 .. w and the sums; only the rsqrt runs per lane), each lane rounded as the scalar
// operation.  An earlier form computed r^2 and the factors per lane (23 paired + 2 x 10 scalar
// instructions per j-pair); pairing them as well (33 paired) follows the Hermite j-paired forms,
// where the same move made the largest call 5 % faster.
__device__ __forceinline__ void g5_quad_jpair(float2 X, float2 Y, float2 Z, float2 M, const float2 (&Q)[6], float2 nx,
                                              float2 ny, float2 nz, float2 e, float2 (&a)[5]) {
    const float2 dx = __fadd2_rn(X, nx), dy = __fadd2_rn(Y, ny), dz = __fadd2_rn(Z, nz);
    const float2 vx = __ffma2_rn(Q[2], dz, __ffma2_rn(Q[1], dy, __fmul2_rn(Q[0], dx)));
    const float2 vy = __ffma2_rn(Q[4], dz, __ffma2_rn(Q[3], dy, __fmul2_rn(Q[1], dx)));
    const float2 vz = __ffma2_rn(Q[5], dz, __ffma2_rn(Q[4], dy, __fmul2_rn(Q[2], dx)));
    const float2 D = __ffma2_rn(dz, vz, __ffma2_rn(dy, vy, __fmul2_rn(dx, vx)));
    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, e)));
    const float2 q = make_float2(pair_scale(r2.x), pair_scale(r2.y));
    const float2 q2 = __fmul2_rn(q, q), q3 = __fmul2_rn(q2, q), q4 = __fmul2_rn(q2, q2);
    const float2 p = __fmul2_rn(q4, __fmul2_rn(make_float2(G5_QK, G5_QK), q));
    const float2 w = __fmul2_rn(q3, __ffma2_rn(D, q4, M));
    a[0] = __ffma2_rn(w, dx, __ffma2_rn(p, vx, a[0]));
    a[1] = __ffma2_rn(w, dy, __ffma2_rn(p, vy, a[1]));
    a[2] = __ffma2_rn(w, dz, __ffma2_rn(p, vz, a[2]));
    a[3] = __ffma2_rn(M, q, a[3]);
    a[4] = __ffma2_rn(p, D, a[4]);
}

// Half `second` of the sums t into a.
template <int N>
__device__ __forceinline__ void g5_half(float2 (&a)[N], const float2 (&t)[N], int second) {
#pragma unroll
    for (int c = 0; c < N; c++) a[c] = second ? make_float2(a[c].x, t[c].y) : make_float2(t[c].x, a[c].y);
}

// Final scaling of the FP64 sums into (acc, pot_raw).
template <int KIND>
__device__ __forceinline__ double4 g5_finish(double4 s, double ascale) {
    if constexpr (KIND == G5_QUAD) return s;  // quad sums are already (acc, +sum(phi_p+phi_q))
    if constexpr (KIND == G5_TABLE)           // acc *= 1/xscale (gravity_kernel_avx2.c:127-129)
        return make_double4(ascale * s.x, ascale * s.y, ascale * s.z, 0.0);
    return make_double4(S_ACC * s.x, S_ACC * s.y, S_ACC * s.z, S_POT * s.w);
}

__device__ __forceinline__ double4 add4(double4 a, double4 b) {
    return make_double4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

// The result of i-particle i.  In host words every 8 bytes carry the call's number themselves: the
// host takes them as they arrive, without a copy, a fence or a synchronisation.
__device__ __forceinline__ void g5_word(const G5Args& A, size_t w, double d) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(d);
    __stwt(A.words + w, make_uint4((unsigned)x, A.seq, (unsigned)(x >> 32), A.seq));
}
__device__ __forceinline__ void g5_result(const G5Args& A, int i, const double4& v) {
    if (!A.words) {
        A.out[i] = v;
        return;
    }
    g5_word(A, 4 * (size_t)i, v.x);
    g5_word(A, 4 * (size_t)i + 1, v.y);
    g5_word(A, 4 * (size_t)i + 2, v.z);
    g5_word(A, 4 * (size_t)i + 3, v.w);
}

// After a task of a split group: the last CTA to finish one of the group's tasks reduces the
// group's partial rows (every thread of the CTA calls this).
template <int KIND, int NT, bool WORDS = false>
__device__ __forceinline__ void g5_group_done(const G5Args& A, const Task& T, double4* red, int* s_flag) {
    const Group G = A.groups[T.group];
    if (group_arrive(A.group_counters, T.group, G.nchunk, s_flag)) {
        // Cooperative reduction of the group's partial rows: P threads per i, each summing a
        // fixed strided subset of the rows, then the P sums in thread order (deterministic
        // for a given group shape).  `red`: NT double4 of shared memory.
        int P = 1;
        while (P * 2 * G.ni <= NT) P *= 2;
        const int per = NT / P;
        for (int base = 0; base < G.ni; base += per) {
            const int li = base + threadIdx.x / P, p = threadIdx.x % P;
            double4 s = make_double4(0, 0, 0, 0);
            if (li < G.ni) {
                // four independent partial sums keep four rows' loads in flight; combined in
                // a fixed order (deterministic)
                const double4* col = A.partial + (size_t)G.slot0 * A.itile + li;
                auto ld = [&](int c) {
                    const double4* r = col + (size_t)c * A.itile;
                    return make_double4(__ldcg(&r->x), __ldcg(&r->y), __ldcg(&r->z), __ldcg(&r->w));
                };
                double4 s1 = s, s2 = s, s3 = s;
                int c = p;
                for (; c + 3 * P < G.nchunk; c += 4 * P) {
                    double4 v0 = ld(c), v1 = ld(c + P), v2 = ld(c + 2 * P), v3 = ld(c + 3 * P);
                    s = add4(s, v0);
                    s1 = add4(s1, v1);
                    s2 = add4(s2, v2);
                    s3 = add4(s3, v3);
                }
                for (; c < G.nchunk; c += P) s = add4(s, ld(c));
                s = add4(add4(s, s1), add4(s2, s3));
            }
            __syncthreads();
            red[threadIdx.x] = s;
            __syncthreads();
            if (p == 0 && li < G.ni) {
                for (int q = 1; q < P; q++) s = add4(s, red[threadIdx.x + q]);
                s = g5_finish<KIND>(s, A.ascale);
                if (!WORDS || !A.words) A.out[G.i0 + li] = s;
            }
            if (WORDS && A.words) {
                // to the host in whole lines: consecutive threads, consecutive words (a thread's own four
                // words each: the 999 x 999 kernel took 15 us instead of 9)
                __syncthreads();
                if (p == 0 && li < G.ni) red[li - base] = s;
                __syncthreads();
                const double* d = reinterpret_cast<const double*>(red);
                const int n = 4 * min(per, G.ni - base);
                for (int w = threadIdx.x; w < n; w += NT) g5_word(A, 4 * (size_t)(G.i0 + base) + w, d[w]);
            }
        }
    }
}

// The kernel of the CTAs of 128 threads and more: IPT i per thread.  JP: the j-paired form (point
// masses and cells, one i per thread), else records of one float4 word each (W words).
template <int NT>
struct G5TileSoA {
    float x[NT], y[NT], z[NT], m[NT];
    float q[6][NT];   // cells: G5_QSCALE (q00 q01 q02 q11 q12 q22)
};

template <int KIND, int NT, int IPT, bool JP = false>
__global__ void __launch_bounds__(NT) g5_kernel(G5Args A) {
    constexpr int W = JWords<KIND>::n;   // 16-byte words per j record
    constexpr bool USE_JP = JP && IPT == 1 && (KIND == G5_NEWTON || KIND == G5_QUAD);
    constexpr int SJ_RECS = NT * (W > 2 ? W : 2);
    constexpr int SJ_SOA = USE_JP ? (int)((sizeof(G5TileSoA<NT>) + 15) / 16) : 0;
    __shared__ float4 sj[SJ_RECS > SJ_SOA ? SJ_RECS : SJ_SOA];  // also the reduction buffer (double4 x NT)
    __shared__ int s_task, s_flag;
    // table kind: the force table in dynamic shared memory sized to the table (A.tbl_size
    // entries, 8 KB for 1024) for the lifetime of the CTA; the other kinds launch without any
    extern __shared__ float2 g5_dyn_tab[];
    const float2* tab = g5_dyn_tab;
    int shift = 0;
    if constexpr (KIND == G5_TABLE) {
        for (int k = threadIdx.x; k < A.tbl_size; k += NT) g5_dyn_tab[k] = A.table[k];
        shift = A.tbl_shift;
        tab = g5_dyn_tab - (0x40000000u >> shift);  // index by (bits of s) >> shift directly
        __syncthreads();
    }
    const int tid = (int)threadIdx.x;

    // The j-paired task: one i per thread.  The tile is staged as field arrays, whose whole quads are
    // taken two j-pairs at a time and the records of a last, partial quad one by one, in both halves
    // of sums of which one counts (padded with massless copies of a record instead, an unsoftened
    // i on that record got 0 * inf).  FP32 sums are folded into FP64 every G5_FOLD j.
    auto jp_task = [&](const Task& T, double (&S)[4]) {
        G5TileSoA<NT>* sa = reinterpret_cast<G5TileSoA<NT>*>(sj);
        const float4 p = A.ipos[T.i0 + (tid < T.ni ? tid : 0)];
        const float2 nx = make_float2(-p.x, -p.x), ny = make_float2(-p.y, -p.y), nz = make_float2(-p.z, -p.z);
        const float2 ei = make_float2(p.w, p.w);
        for (int jt = 0; jt < T.nj; jt += NT) {
            const int nt = min(NT, T.nj - jt);
            __syncthreads();
            if (tid < nt) {
                const int jk = T.j0 + jt + tid;
                const int jj = A.jidx ? __ldg(A.jidx + jk) : jk;
                const float4 J = A.jpos[jj];
                sa->x[tid] = J.x;
                sa->y[tid] = J.y;
                sa->z[tid] = J.z;
                sa->m[tid] = J.w;
                if constexpr (KIND == G5_QUAD) {
                    const float4 Q0 = A.jaux[2 * jj], Q1 = A.jaux[2 * jj + 1];
                    sa->q[0][tid] = G5_QSCALE * Q0.x;
                    sa->q[1][tid] = G5_QSCALE * Q0.y;
                    sa->q[2][tid] = G5_QSCALE * Q0.z;
                    sa->q[3][tid] = G5_QSCALE * Q0.w;
                    sa->q[4][tid] = G5_QSCALE * Q1.x;
                    sa->q[5][tid] = G5_QSCALE * Q1.y;
                }
            }
            __syncthreads();
            const int ntf = nt & ~3;
            for (int jb = 0; jb < ntf; jb += G5_FOLD) {
                const int je = min(jb + G5_FOLD, ntf);
                float2 a2[NAcc<KIND>::n];
#pragma unroll
                for (int c = 0; c < NAcc<KIND>::n; c++) a2[c] = make_float2(0.f, 0.f);
                for (int j = jb; j < je; j += 4) {
                    const float4 X = *reinterpret_cast<const float4*>(&sa->x[j]);
                    const float4 Y = *reinterpret_cast<const float4*>(&sa->y[j]);
                    const float4 Z = *reinterpret_cast<const float4*>(&sa->z[j]);
                    const float4 M = *reinterpret_cast<const float4*>(&sa->m[j]);
                    const float2 xa = make_float2(X.x, X.y), xb = make_float2(X.z, X.w);
                    const float2 ya = make_float2(Y.x, Y.y), yb = make_float2(Y.z, Y.w);
                    const float2 za = make_float2(Z.x, Z.y), zb = make_float2(Z.z, Z.w);
                    const float2 ma = make_float2(M.x, M.y), mb = make_float2(M.z, M.w);
                    if constexpr (KIND == G5_QUAD) {
                        float2 Qa[6], Qb[6];
#pragma unroll
                        for (int c = 0; c < 6; c++) {
                            const float4 v = *reinterpret_cast<const float4*>(&sa->q[c][j]);
                            Qa[c] = make_float2(v.x, v.y);
                            Qb[c] = make_float2(v.z, v.w);
                        }
                        g5_quad_jpair(xa, ya, za, ma, Qa, nx, ny, nz, ei, a2);
                        g5_quad_jpair(xb, yb, zb, mb, Qb, nx, ny, nz, ei, a2);
                    } else {
                        g5_newton_jpair(xa, ya, za, ma, nx, ny, nz, ei, a2);
                        g5_newton_jpair(xb, yb, zb, mb, nx, ny, nz, ei, a2);
                    }
                }
                g5_fold2<KIND>(S, a2, -1);
            }
            if (ntf < nt) {
                float2 a2[NAcc<KIND>::n];
#pragma unroll
                for (int c = 0; c < NAcc<KIND>::n; c++) a2[c] = make_float2(0.f, 0.f);
#pragma unroll 1
                for (int j = ntf; j < nt; j++) {
                    auto both = [&](const float* f) { return make_float2(f[j], f[j]); };
                    if constexpr (KIND == G5_QUAD) {
                        float2 Q[6];
#pragma unroll
                        for (int c = 0; c < 6; c++) Q[c] = both(sa->q[c]);
                        g5_quad_jpair(both(sa->x), both(sa->y), both(sa->z), both(sa->m), Q, nx, ny, nz, ei, a2);
                    } else {
                        g5_newton_jpair(both(sa->x), both(sa->y), both(sa->z), both(sa->m), nx, ny, nz, ei, a2);
                    }
                }
                g5_fold2<KIND>(S, a2, 0);
            }
        }
    };

    for (bool first = true;; first = false) {
        int t = next_task(A.task_counter, &s_task, A.ntasks, first);
        if (t >= A.ntasks) break;
        const Task T = A.tasks[t];
        double S[IPT][4];
#pragma unroll
        for (int k = 0; k < IPT; k++) S[k][0] = S[k][1] = S[k][2] = S[k][3] = 0.0;
        if constexpr (USE_JP) {
            jp_task(T, S[0]);
        } else {
            float xi[IPT], yi[IPT], zi[IPT], ei[IPT];
#pragma unroll
            for (int k = 0; k < IPT; k++) {
                int li = tid + k * NT;
                int ii = T.i0 + (li < T.ni ? li : 0);
                float4 p = A.ipos[ii];
                xi[k] = p.x; yi[k] = p.y; zi[k] = p.z; ei[k] = p.w;
            }
            for (int jt = 0; jt < T.nj; jt += NT) {
                const int nt = min(NT, T.nj - jt);
                __syncthreads();
                if (tid < nt) {
                    const int jk = T.j0 + jt + tid;
                    const int jj = A.jidx ? __ldg(A.jidx + jk) : jk;
                    sj[tid] = A.jpos[jj];
                    if constexpr (W == 2) sj[NT + tid] = A.jaux[jj];
                    if constexpr (W == 3) g5_stage_quad(sj + NT + 2 * tid, A.jaux, jj);
                }
                __syncthreads();
                for (int j0 = 0; j0 < nt; j0 += G5_FOLD) {
                    const int j1 = min(j0 + G5_FOLD, nt);
                    if constexpr (IPT % 2 == 0) {
                        float2 a2[IPT / 2][NAcc<KIND>::n];
#pragma unroll
                        for (int p = 0; p < IPT / 2; p++)
#pragma unroll
                            for (int c = 0; c < NAcc<KIND>::n; c++) a2[p][c] = make_float2(0.f, 0.f);
#pragma unroll 4
                        for (int j = j0; j < j1; j++) {
#pragma unroll
                            for (int p = 0; p < IPT / 2; p++)
                                g5_interact2<KIND, NT>(sj, j, xi + 2 * p, yi + 2 * p, zi + 2 * p, ei + 2 * p, tab, shift,
                                                       A.r2cut, a2[p]);
                        }
#pragma unroll
                        for (int k = 0; k < IPT; k++) g5_fold2<KIND>(S[k], a2[k / 2], k % 2);
                    } else {
                        float a[IPT][NAcc<KIND>::n];
#pragma unroll
                        for (int k = 0; k < IPT; k++)
#pragma unroll
                            for (int c = 0; c < NAcc<KIND>::n; c++) a[k][c] = 0.f;
#pragma unroll 4
                        for (int j = j0; j < j1; j++) {
#pragma unroll
                            for (int k = 0; k < IPT; k++) {
                                if constexpr (KIND == G5_TABLE)
                                    g5_table_pair(sj[j], xi[k], yi[k], zi[k], tab, shift, A.r2cut, a[k]);
                                else
                                    g5_interact<KIND, NT>(sj, j, xi[k], yi[k], zi[k], ei[k], a[k]);
                            }
                        }
#pragma unroll
                        for (int k = 0; k < IPT; k++) g5_fold<KIND>(S[k], a[k]);
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const int li = tid + k * NT;
            if (li >= T.ni) continue;
            const double4 v = make_double4(S[k][0], S[k][1], S[k][2], S[k][3]);
            if (T.group < 0) A.out[T.i0 + li] = g5_finish<KIND>(v, A.ascale);
            else A.partial[(size_t)T.slot * A.itile + li] = v;
        }
        if (T.group >= 0) g5_group_done<KIND, NT>(A, T, reinterpret_cast<double4*>(sj), &s_flag);
    }
}

// ---- the 64-thread kernel: i-slots x j-lanes ------------------------------------------------
// Every task of a 64-thread CTA runs as 16 i-slots over four j-lanes, IPT = ceil(ni / 16) i per
// thread (slot, slot + 16, ...), j-paired.  It is built for batches of small, uneven groups (tree
// and TreePM groups of a few tens to a few hundred i), which the FMA pipe bounds:
//  * a task leaves at most 15 of its slots idle, whatever its size (a 75-particle group runs as
//    64 + 11: 80 slots; 9.6 % of the slots of an N = 2^20 tree's cell pairs are idle);
//  * the j records read from shared memory serve IPT i: a full task reads a 16-byte word per 4
//    pairs (point masses) or 1.6 pairs (cells);
//  * every FP32 operation is paired: a cell pair takes 16.5 + 1 (rsqrt) instructions instead of 34.
// Against the one-record-per-load form it replaces (one to three i per thread, two to four lanes,
// scalar chains): cells of an N = 2^20 tree 4156 -> 3563 us (799 Gint/s: with the idle slots 79 %
// of the FMA rate), its point masses 974 -> 831 us (1930 Gint/s), the 4096 TreePM groups of 2^20
// particles 2906 -> 2282 us (1955 Gint/s; 12 FMA operations, 4 integer ones and a table look-up of
// 2.2 shared wavefronts a pair: FMA heavy half 65 %, shared wavefronts 70 %, issue 65 % busy).
// A j-tile is G5S_NJ records as field arrays; lane l takes the tile's j-quads l, l + 4, ....  The
// tile is padded to a multiple of 4 with massless records far away (G5S_FAR), which add exact
// zeros to any finite sum: where r^2 overflows, 1/r is 0.  The Newton-refined rsqrt of an overflowed
// r^2 is NaN, so with it the records of a last, partial quad are taken one by one instead
// (G5S_TAIL; in the default build that made launches of 5 to 15 us 0.6 to 1 us longer).
// FP32 sums cover a tile (32 terms a lane half and i at most), then go
// into the FP64 sums; the lanes' sums are added in lane order at the end of the task.
constexpr int G5S_NT = 64, G5S_SLOTS = 16, G5S_LANES = 4, G5S_IPT = 4;
constexpr int G5S_NJ = 256;   // records a tile: 64 a lane between two folds into FP64 (128: cells 3 % slower)
// Resident CTAs asked of the compiler: cells 5 (167 registers, 10 warps an SM: 3563 us; 8 CTAs of 128
// registers, which reload the j fields per pair, 3639), point masses and the table 10 (95 registers)
template <int KIND>
constexpr int g5s_min_ctas() { return KIND == G5_QUAD ? 5 : 10; }

constexpr float G5S_FAR = 1e18f;   // its square times three is finite
#ifdef PGB_RSQRT_NEWTON
constexpr bool G5S_TAIL = true;
#else
constexpr bool G5S_TAIL = false;
#endif

template <int KIND>
struct G5STile {
    static constexpr int NQ = KIND == G5_QUAD ? 6 : (KIND == G5_SYMMETRIC ? 1 : 0);   // extra fields
    float f[4 + NQ][G5S_NJ];   // x y z m, then the moments (G5_QSCALE q00 q01 q02 q11 q12 q22) or eps2_j
};

template <int KIND>
struct G5SShared {
    G5STile<KIND> t;
    double S[G5S_IPT][4][G5S_NT];   // the FP64 sums: i k, component c of thread t at S[k][c][t]
};

template <int KIND, int IPT>
__device__ __forceinline__ void g5_slots_task(const G5Args& A, const Task& T, G5SShared<KIND>& sh, unsigned tab) {
    constexpr int NJ = G5S_NJ, R = NJ / G5S_NT;
    constexpr int NC = KIND == G5_TABLE ? 3 : 4;   // components that are summed
    const int tid = (int)threadIdx.x, slot = tid % G5S_SLOTS, lane = tid / G5S_SLOTS;
    float2 nx[IPT], ny[IPT], nz[IPT], ei[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const int li = slot + k * G5S_SLOTS;
        const float4 p = A.ipos[T.i0 + (li < T.ni ? li : 0)];
        nx[k] = make_float2(-p.x, -p.x);
        ny[k] = make_float2(-p.y, -p.y);
        nz[k] = make_float2(-p.z, -p.z);
        ei[k] = make_float2(p.w, p.w);
#pragma unroll
        for (int c = 0; c < 4; c++) sh.S[k][c][tid] = 0.0;
    }
    const int shift3 = A.tbl_shift - 3;
    const unsigned nodemask = ~0u << (A.tbl_shift & 31);
    int jn[R];
    auto load_idx = [&](int j0) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int q = j0 + tid + r * G5S_NT;
            jn[r] = T.j0 + q;
            if (A.jidx && q < T.nj) jn[r] = __ldg(A.jidx + T.j0 + q);
        }
    };
    load_idx(0);
    for (int jt = 0; jt < T.nj; jt += NJ) {
        const int nt = min(NJ, T.nj - jt), nq = G5S_TAIL ? nt >> 2 : (nt + 3) >> 2;
        float4 J[R];
        float4 Q0[R], Q1[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int q = tid + r * G5S_NT;
            J[r] = make_float4(G5S_FAR, G5S_FAR, G5S_FAR, 0.f);
            Q0[r] = Q1[r] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q < nt) {
                const int jj = jn[r];
                J[r] = A.jpos[jj];
                if constexpr (KIND == G5_QUAD) {
                    Q0[r] = scale4(A.jaux[2 * (size_t)jj], G5_QSCALE);
                    Q1[r] = scale4(A.jaux[2 * (size_t)jj + 1], G5_QSCALE);
                }
                if constexpr (KIND == G5_SYMMETRIC) Q0[r].x = A.jaux[jj].x;
            }
        }
        __syncthreads();   // the tile before has been read
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int q = tid + r * G5S_NT;
            if (q < (G5S_TAIL ? nt : 4 * nq)) {
                float(*f)[NJ] = sh.t.f;
                f[0][q] = J[r].x;
                f[1][q] = J[r].y;
                f[2][q] = J[r].z;
                f[3][q] = J[r].w;
                if constexpr (KIND == G5_QUAD) {
                    f[4][q] = Q0[r].x;
                    f[5][q] = Q0[r].y;
                    f[6][q] = Q0[r].z;
                    f[7][q] = Q0[r].w;
                    f[8][q] = Q1[r].x;
                    f[9][q] = Q1[r].y;
                }
                if constexpr (KIND == G5_SYMMETRIC) f[4][q] = Q0[r].x;
            }
        }
        __syncthreads();
        load_idx(jt + NJ);   // the next tile's indices: its records are then one load away
        float2 a[IPT][NAcc<KIND>::n];
#pragma unroll
        for (int k = 0; k < IPT; k++)
#pragma unroll
            for (int c = 0; c < NAcc<KIND>::n; c++) a[k][c] = make_float2(0.f, 0.f);
        // the pair terms of i k and the two records w
        auto add = [&](int k, const float2 (&w)[4 + G5STile<KIND>::NQ], float2 (&s)[NAcc<KIND>::n]) {
            if constexpr (KIND == G5_QUAD) {
                const float2 q[6] = {w[4], w[5], w[6], w[7], w[8], w[9]};
                g5_quad_jpair(w[0], w[1], w[2], w[3], q, nx[k], ny[k], nz[k], ei[k], s);
            } else if constexpr (KIND == G5_TABLE) {
                g5_table_jpair(w[0], w[1], w[2], w[3], nx[k], ny[k], nz[k], tab, shift3, nodemask, A.r2cut, s);
            } else if constexpr (KIND == G5_SYMMETRIC) {
                g5_newton_jpair(w[0], w[1], w[2], w[3], nx[k], ny[k], nz[k], __fadd2_rn(ei[k], w[4]), s);
            } else {
                g5_newton_jpair(w[0], w[1], w[2], w[3], nx[k], ny[k], nz[k], ei[k], s);
            }
        };
#pragma unroll 1
        for (int jq = lane; jq < nq; jq += G5S_LANES) {
            float4 v[4 + G5STile<KIND>::NQ];
#pragma unroll
            for (int c = 0; c < 4 + G5STile<KIND>::NQ; c++) v[c] = *reinterpret_cast<const float4*>(&sh.t.f[c][4 * jq]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float2 w[4 + G5STile<KIND>::NQ];
#pragma unroll
                for (int c = 0; c < 4 + G5STile<KIND>::NQ; c++)
                    w[c] = h ? make_float2(v[c].z, v[c].w) : make_float2(v[c].x, v[c].y);
#pragma unroll
                for (int k = 0; k < IPT; k++) add(k, w, a[k]);
            }
        }
        if (G5S_TAIL && lane == nq % G5S_LANES) {
#pragma unroll 1
            for (int j = 4 * nq; j < nt; j++) {
                float2 w[4 + G5STile<KIND>::NQ];
#pragma unroll
                for (int c = 0; c < 4 + G5STile<KIND>::NQ; c++) w[c] = make_float2(sh.t.f[c][j], sh.t.f[c][j]);
#pragma unroll
                for (int k = 0; k < IPT; k++) {
                    float2 t[NAcc<KIND>::n];
#pragma unroll
                    for (int c = 0; c < NAcc<KIND>::n; c++) t[c] = a[k][c];
                    add(k, w, t);
                    g5_half(a[k], t, j & 1);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            double S[4];
#pragma unroll
            for (int c = 0; c < NC; c++) S[c] = sh.S[k][c][tid];
            S[3] = NC > 3 ? S[3] : 0.0;
            g5_fold2<KIND>(S, a[k], -1);
#pragma unroll
            for (int c = 0; c < NC; c++) sh.S[k][c][tid] = S[c];
        }
    }
    // the lanes' sums in lane order: thread t sums i-particle t
    __syncthreads();
    if (tid < T.ni) {
        const int k = tid / G5S_SLOTS, s0 = tid % G5S_SLOTS;
        double S[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            S[c] = sh.S[k][c][s0];
#pragma unroll
            for (int l = 1; l < G5S_LANES; l++) S[c] += sh.S[k][c][s0 + l * G5S_SLOTS];
        }
        const double4 v = make_double4(S[0], S[1], S[2], S[3]);
        if (T.group < 0) g5_result(A, T.i0 + tid, g5_finish<KIND>(v, A.ascale));
        else A.partial[(size_t)T.slot * A.itile + tid] = v;
    }
    __syncthreads();   // before the sums' or the tile's memory is used again
}

template <int KIND>
__global__ void __launch_bounds__(G5S_NT, g5s_min_ctas<KIND>()) g5_slots_kernel(G5Args A) {
    __shared__ __align__(16) G5SShared<KIND> sh;
    __shared__ int s_task, s_flag;
    extern __shared__ float2 g5_dyn_tab[];   // the table kind's force table, for the CTA's lifetime
    unsigned tab = 0;
    if constexpr (KIND == G5_TABLE) {
        for (int k = threadIdx.x; k < A.tbl_size; k += G5S_NT) g5_dyn_tab[k] = A.table[k];
        tab = (unsigned)__cvta_generic_to_shared(g5_dyn_tab) - (0x40000000u >> (A.tbl_shift - 3));
        __syncthreads();
    }
    for (bool first = true;; first = false) {
        const int t = next_task(A.task_counter, &s_task, A.ntasks, first);
        if (t >= A.ntasks) break;
        const Task T = A.tasks[t];
        if (T.ni > 3 * G5S_SLOTS) g5_slots_task<KIND, 4>(A, T, sh, tab);
        else if (T.ni > 2 * G5S_SLOTS) g5_slots_task<KIND, 3>(A, T, sh, tab);
        else if (T.ni > G5S_SLOTS) g5_slots_task<KIND, 2>(A, T, sh, tab);
        else g5_slots_task<KIND, 1>(A, T, sh, tab);
        if (T.group >= 0) g5_group_done<KIND, G5S_NT, true>(A, T, reinterpret_cast<double4*>(&sh), &s_flag);
    }
}

}  // namespace pgb
