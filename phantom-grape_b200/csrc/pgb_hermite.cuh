// pgb_hermite.cuh -- the PG6 sample integrator's 4th-order Hermite block-time-step scheme on
// the device: block selection, i- and j-prediction, force, corrector and new step, start-up
// step, time reset -- one persistent kernel runs whole block steps back to back.
//
// Reference: PG6/banana (built with -DNORMAL, its setting): timestep.c:87-98 global_time
// (block time and active set), hermite.c:39-63 predict_exmotion (i predictor), hermite.c:67-108
// correct + 143-205 correct_sgmotion (corrector, new state), timestep.c:53-85 dt_criterion
// (Aarseth criterion, step halved or doubled on the power-of-two grid), hermite.c:110-141
// startup_sgmotion + timestep.c:24-51 dt_startup, timestep.c:127-135 reset_time,
// timestep.c:137-150 calc_modulus, banana01.c:119-179 the main loop.  The j-memory that the
// reference re-sends with g6_set_j_particle after every step (hermite.c:240-265: pos, vel,
// acc/2, jerk/6, mass, t) is the particle state itself here: the j predictor reads the state
// arrays, so nothing is re-sent.
//
// State in HBM, one array per field of struct Particle (PG6/banana/particle.h): t, dt, pot,
// mass [n] and pos, vel, acc, jrk [n][3], all FP64 (jrk and pot hold float values: the
// reference stores them as float).
//
// hm_run_kernel is a cooperative launch (every CTA resident) that loops over block steps until
// the global time reaches tend.  Segments of HM_SEG particles belong to CTAs (segment s to CTA
// s mod grid) in every phase.  No barrier separates the steps: a CTA waits only for the data it
// reads, published with the step number as its tag.
//   A  (once per launch, then at the end of every step) per segment: the minimum of t_i + dt_i, how
//      many particles sit at it and which, as a 16-byte record tagged with the next step's number;
//   B  every CTA waits for every segment's record and derives the block time t_gl, the offsets of the
//      segments' active particles and the step's decomposition from them; CTA 0 advances the clock.
// A small step (at most HM_SMALL active particles, most steps of an integration) is a chain of
// latencies, so it hands data over as few times as it can:
//   C  the CTA of a j-chunk predicts its own j and the active i from the particle state, straight
//      into shared memory, evaluates the GRAPE-6 pair terms and writes the chunk's sums as 16-byte
//      words that carry the tag themselves (no fence, no separate flag);
//   D  the owner of an active particle, one warp per particle, reads those words until all are
//      tagged, sums them in chunk order, runs the corrector (or the start-up step), then A.
// A large step goes through memory instead:
//   B' owners predict their segments' particles to t_gl (the library's FP64 j predictor,
//      gravity.c:149-193) and write their active ones, in index order, to the active list with
//      predicted i-records (published per segment);
//   C' the force: the GRAPE-6 pair kernel's tasks (pgb_g6_kernels.cuh g6_task) over an
//      i-tile x j-chunk decomposition of the ni x n pairs, each task once the segments of its
//      i- and j-ranges are built; split j-ranges left as partial rows (published per task);
//   D' per own segment, once the tasks of its active particles' i-tiles are done, as D; reset_time if
//      the step ended on a multiple of dtmax.
// What keeps a fast CTA from overwriting what a slow one still reads: every force task belongs to an
// i-tile with an active particle, whose owner waits for the task before it publishes its record, and
// nobody starts the next step without all records.  So state, predictions, partial sums and flags
// of a step are never written before everybody has read those of the step before.  The records
// themselves are kept for HM_RSLOTS steps, and a record is written over one that every CTA has
// acknowledged (CTAs without work in a step may lag behind the others).
// Every CTA derives the step's decisions (block time, ni, decomposition, end of the run) from
// the same data, so they agree without further communication.  The waits are bounded: one that
// lasts longer than about a second (a limit the host may lower) sets an error word and the kernel
// returns.
// Most steps move fewer than 16 particles, so latencies bound a run: the chain record -> small task ->
// sums -> corrector -> record.  Measured, a Plummer sphere advanced to t = 0.125 (B200): 6.70 / 13.1 /
// 47.0 ms for n = 1000 / 4096 / 16384 (354 / 679 / 2082 steps) against 7.92 / 16.6 / 58.0 ms with a
// grid barrier between the phases and the j predicted through memory.  At 16384 the halved tail tasks
// give 1.1 of the 11 ms.
// The i-predictor and the corrector use the reference's formulas and constants in the order
// its C source evaluates them, with every FP64 multiply and add rounded separately (no fused
// multiply-add): given the same forces the new state equals a plain C evaluation bit for bit.
#pragma once

#include "pgb_g6_kernels.cuh"

namespace pgb {

constexpr int HM_NT = 256;       // threads per CTA
constexpr int HM_SEG = 256;      // particles per segment of the selection (one per thread)
constexpr int HM_MAXSEG = 4096;  // segments at most: n <= 2^20
constexpr int HM_OWN = HM_MAXSEG / 64;   // segments of one CTA at most: the grid has at least 64 CTAs
constexpr int HM_NEXT = 2;       // own segments whose t + dt a CTA keeps in shared memory

struct HmState {
    double *t, *dt, *pos, *vel, *acc, *jrk, *pot, *mass;
    int n;
};

// The integrator's clock and counters in device memory (banana01.c:119-179 bookkeeping): the
// last step's block time and active count, the global time after it (t_mod * dtmax + t_gl, or
// t_mod * dtmax after a reset), the completed dtmax intervals, the particle / block steps, the
// pair interactions and the steps by force decomposition.
struct HmClock {
    double t_gl;
    double time;
    long long psteps, bsteps;
    long long force_pairs;
    long long variant_steps[5];   // steps by force decomposition (i-tile 16, 32, 64, 128, 512)
    long long spin_limit;         // SM cycles a wait may last (0: HM_SPIN_LIMIT)
    int t_mod;
    int ni;       // the last step's active count
    int nch;      // its force decomposition: j-chunks and i-tile
    int itile;
    int bad;      // start-up steps below dtmin
    int err;      // a wait gave up
    int exits;    // CTAs that have returned from the step kernel (all launches)
    int pad;
};

// Default limit of every wait of the step kernel: about a second of SM clock.
constexpr long long HM_SPIN_LIMIT = 2000000000LL;

constexpr int HM_SMALL = 128;   // active particles of a small step at most (one i-tile)
constexpr int HM_RSLOTS = 4;    // steps for which a segment's records are kept

// Published words: read and written as one 16-byte access.
struct __align__(16) HmWord {
    unsigned long long lo, hi;
};
__device__ __forceinline__ HmWord hm_ld(const HmWord* p) {
    HmWord v;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(v.lo), "=l"(v.hi) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void hm_st(HmWord* p, HmWord v) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}"
                 :: "l"(p), "l"(v.lo), "l"(v.hi) : "memory");
}
__device__ __forceinline__ unsigned hm_tag(const HmWord& v) { return (unsigned)(v.hi >> 32); }

// A segment's record: lo = the minimum of t + dt (bits), hi = the tag (high half) | the count (9 bits),
// the local indices of the first two particles at it (8 bits each, from bit 9) and the slot of the
// list of them all (from bit 25).  One chunk's sums for one active particle of a small step: 14 words
// of FP64 halves, three to an HmWord with the tag.
constexpr int HM_SUMW = 5;

struct HmWork {
    HmWord* rec;               // [HM_RSLOTS][nseg] segment records of step T in slot T mod HM_RSLOTS
    unsigned char* seg_list;   // [HM_RSLOTS][nseg][HM_SEG] local indices of the particles at the minimum
                               // (a segment's next list goes to the next slot)
    unsigned* ack;             // [grid] the last step whose records the CTA has read
    HmWord* sums;              // [HM_SMALL][chunks][HM_SUMW] small steps' chunk sums
    int chunks;
    unsigned* seg_flag;        // [nseg] step number of the segment's last build (large steps)
    unsigned* task_flag;       // [task_cap] step number of the force task's last completion, then [grid]
                               // of the second halves of halved tasks
    int task_cap;
    HmClock* clk;
    int* active;               // [n] active particles in index order
    G6I* irec;                 // [n] their predicted i-records (large steps)
    G6PredJ* jpred;            // [n] every particle predicted to t_gl (large steps)
    G6Out* out;                // [n] force, jerk, potential of the active particles (final)
    G6Out* partial;            // partial rows of split j-ranges, part_cap entries
    long long part_cap;
};

struct HmRun {
    HmState P;
    HmWork W;
    float eps2;
    double eta, eta_s, dtmax, tend;
    // the clock as the last launch left it (from the host, so that no CTA reads what CTA 0 stores):
    // the number of the first step, the global time and the completed dtmax intervals
    unsigned step0;
    double time0;
    int t_mod0;
    int startup;     // take the start-up step only
    int max_steps;   // block steps of this launch at most
    int nseg;
    int minj;        // j per chunk at least
    int nch1;        // j-chunks of a step of one i-tile of at most HM_SMALL (hm_shape's, from the host)
    double dtinv;    // 1 / dtmax
};

// A bounded wait: `more` returns true while the caller has to look again.  It gives up after about a
// second of SM clock (C->spin_limit cycles when set), or when another wait has (the error word).
template <class More>
__device__ __forceinline__ bool hm_wait(HmClock* C, More more) {
    if (!more()) return true;
    const long long t0 = clock64();
    const long long lim = C->spin_limit > 0 ? C->spin_limit : HM_SPIN_LIMIT;
    for (unsigned it = 1; more(); it++) {
        if (clock64() - t0 > lim || ((it & 255) == 0 && *(volatile int*)&C->err)) {
            atomicExch(&C->err, 1);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ bool hm_spin_until(volatile unsigned* w, unsigned target, HmClock* C) {
    return hm_wait(C, [&] { return *w != target; });
}

__device__ __forceinline__ double hm_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double hm_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double hm_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double hm_float(double a) { return (double)__double2float_rn(a); }

// predict_exmotion's constants as its source spells them (hermite.h)
constexpr double HM_SECOND = 5e-1;
constexpr double HM_THIRD = 1.666666666666667e-1;
constexpr double HM_FOURTH = 4.166666666666667e-2;
constexpr double HM_FIFTH = 8.333333333333333e-3;

// i predictor (hermite.c:47-56): x + v d + a d^2 (1/2) + j d^3 (1/6), v + a d + j d^2 (1/2)
__device__ __forceinline__ void hm_predict_i(const HmState& P, int i, double t_gl, double xp[3], double vp[3]) {
    const double d = hm_sub(t_gl, __ldcg(P.t + i));
    const double d2 = hm_mul(d, d), d3 = hm_mul(d, d2);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double x = __ldcg(P.pos + 3 * i + c), v = __ldcg(P.vel + 3 * i + c), a = __ldcg(P.acc + 3 * i + c),
                     j = __ldcg(P.jrk + 3 * i + c);
        xp[c] = hm_add(hm_add(hm_add(x, hm_mul(v, d)), hm_mul(hm_mul(a, d2), HM_SECOND)),
                       hm_mul(hm_mul(j, d3), HM_THIRD));
        vp[c] = hm_add(hm_add(v, hm_mul(a, d)), hm_mul(hm_mul(j, d2), HM_SECOND));
    }
}

// calc_modulus (timestep.c:137-150): what is left of num after removing the largest
// power-of-two multiples down to mod; zero when num is a multiple of mod on dtmax's grid.
__device__ __forceinline__ double hm_modulus(double num, double mod, double modmax) {
    double tmpmod = modmax;
    for (int it = 0; num > 0.0 && it < 4096; it++) {
        for (int k = 0; tmpmod > num && k < 2048; k++) tmpmod *= 0.5;
        if (tmpmod < mod) break;
        num = hm_sub(num, tmpmod);
    }
    return num;
}

// The minimum over the CTA (any 64-bit pattern, unsigned); sm: NT / 32 words, free again after the
// caller's next barrier.
__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
    const unsigned full = 0xffffffffu;
    const unsigned hi = __reduce_min_sync(full, (unsigned)(v >> 32));
    const unsigned lo = __reduce_min_sync(full, (unsigned)(v >> 32) == hi ? (unsigned)v : ~0u);
    return (unsigned long long)hi << 32 | lo;
}
template <int NT>
__device__ __forceinline__ unsigned long long block_min_u64(unsigned long long v, unsigned long long* sm) {
    v = warp_min_u64(v);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
    __syncthreads();
    v = sm[0];
#pragma unroll
    for (int w = 1; w < NT / 32; w++) v = sm[w] < v ? sm[w] : v;
    return v;
}

// Inclusive scan of v over the CTA (warp shuffles, then the warp totals); *total = the sum.
template <int NT>
__device__ __forceinline__ int block_scan(int v, int* sw, int* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    __syncthreads();
    if (lane == 31) sw[w] = v;
    __syncthreads();
    int base = 0, all = 0;
#pragma unroll
    for (int k = 0; k < NT / 32; k++) {
        base += k < w ? sw[k] : 0;
        all += sw[k];
    }
    *total = all;
    return v + base;
}

// A force from its FP64 sums s (ax, ay, az, jx, jy, jz, pot), scaled as the force kernel's final stage
// does.
__device__ __forceinline__ G6Out hm_scaled(const double (&s)[7]) {
    G6Out F;
    F.ax = S_ACC * s[0]; F.ay = S_ACC * s[1]; F.az = S_ACC * s[2];
    F.jx = S_ACC * s[3]; F.jy = S_ACC * s[4]; F.jz = S_ACC * s[5];
    F.pot = S_POT * s[6];
    F.key = 0.f;
    F.jadr = -1;
    return F;
}

// The warp's lane sums, added by a butterfly; every lane gets lane 0's sums.
__device__ __forceinline__ void hm_warp_sum(double (&s)[7]) {
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < 7; q++) s[q] += __shfl_xor_sync(full, s[q], o);
#pragma unroll
    for (int q = 0; q < 7; q++) s[q] = __shfl_sync(full, s[q], 0);
}

// The force of active particle k of a large step, by the whole warp: with nch > 1 the sum of its nch
// j-chunk partial rows in a fixed order (lane l takes chunks l, l+32, ..., then a butterfly), written
// to out[k]; with nch == 1 the force kernel's final result out[k].
__device__ __forceinline__ G6Out hm_force_of(const HmWork& W, int k, int nch, int itile) {
    const int lane = threadIdx.x & 31;
    if (nch == 1) return W.out[k];
    const int it = k / itile, li = k - it * itile;
    const double2* row = reinterpret_cast<const double2*>(W.partial + (size_t)it * nch * itile + li);
    const size_t stride = (size_t)itile * 4;   // double2 words per partial row
    double s[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int c = lane; c < nch; c += 32) {
        const double2* r = row + (size_t)c * stride;
        const double2 w0 = __ldcg(r), w1 = __ldcg(r + 1), w2 = __ldcg(r + 2), w3 = __ldcg(r + 3);
        s[0] += w0.x; s[1] += w0.y; s[2] += w1.x; s[3] += w1.y; s[4] += w2.x; s[5] += w2.y; s[6] += w3.x;
    }
    hm_warp_sum(s);
    const G6Out F = hm_scaled(s);
    if (lane == 0) W.out[k] = F;
    return F;
}

// The same for a small step: each chunk's tagged words are read until they carry the step's tag.
// False (in every lane) if a wait gave up.
__device__ __forceinline__ bool hm_force_small(const HmWork& W, int k, int nch, unsigned E, G6Out& F) {
    const int lane = threadIdx.x & 31;
    double s[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    bool ok = true;
    for (int c = lane; ok && c < nch; c += 32) {
        const HmWord* p = W.sums + ((size_t)k * W.chunks + c) * HM_SUMW;
        HmWord w[HM_SUMW];
        ok = hm_wait(W.clk, [&] {
            bool all = true;
#pragma unroll
            for (int q = 0; q < HM_SUMW; q++) w[q] = hm_ld(p + q);
#pragma unroll
            for (int q = 0; q < HM_SUMW; q++) all = all && hm_tag(w[q]) == E;
            return !all;
        });
        unsigned u[3 * HM_SUMW];
#pragma unroll
        for (int q = 0; q < HM_SUMW; q++) {
            u[3 * q] = (unsigned)w[q].lo;
            u[3 * q + 1] = (unsigned)(w[q].lo >> 32);
            u[3 * q + 2] = (unsigned)w[q].hi;
        }
#pragma unroll
        for (int q = 0; q < 7; q++)
            s[q] += __longlong_as_double((long long)((unsigned long long)u[2 * q + 1] << 32 | u[2 * q]));
    }
    ok = __all_sync(0xffffffffu, ok);
    hm_warp_sum(s);
    F = hm_scaled(s);
    if (lane == 0) W.out[k] = F;
    return ok;
}

// Corrector and new step of active particle i (hermite.c:67-108, 143-205; timestep.c:53-85), given
// its new acceleration (FP64), jerk and potential (rounded to float as the reference's struct
// NewAccJerk stores them), by a whole warp: lane l works on component l mod 3, and on norm l mod 4
// of the criterion; the operations on each and their order are the reference's.  load() reads the
// state and predicts, which does not need the force.
struct HmOwn {
    double dts, dtsinv, a0, j0, x1, v1;
    __device__ __forceinline__ void load(const HmState& P, int i, double tg) {
        const int c = (int)(threadIdx.x & 31) % 3, k = 3 * i + c;
        const double x = P.pos[k], v = P.vel[k];
        a0 = P.acc[k];
        j0 = P.jrk[k];
        dts = P.dt[i];
        const double d = hm_sub(tg, P.t[i]);
        const double d2 = hm_mul(d, d), d3 = hm_mul(d, d2);
        x1 = hm_add(hm_add(hm_add(x, hm_mul(v, d)), hm_mul(hm_mul(a0, d2), HM_SECOND)), hm_mul(hm_mul(j0, d3), HM_THIRD));
        v1 = hm_add(hm_add(v, hm_mul(a0, d)), hm_mul(hm_mul(j0, d2), HM_SECOND));
        dtsinv = 1.0 / dts;
    }
    // Returns t + dt afterwards (bits).
    __device__ __forceinline__ unsigned long long correct(const HmState& P, int i, double tg, const G6Out& F, double eta,
                                                          double dtmax) {
        const unsigned full = 0xffffffffu;
        const int lane = (int)(threadIdx.x & 31), c = lane % 3;
        const double dtmin = dtmax / 2251799813685248.0;  // dtmax / 2^51
        const double a1 = c == 0 ? F.ax : (c == 1 ? F.ay : F.az);
        const double j1 = hm_float(c == 0 ? F.jx : (c == 1 ? F.jy : F.jz));
        const double da = hm_sub(a0, a1);
        const double s0 = hm_mul(hm_mul(hm_mul(2.0, hm_sub(hm_mul(-3.0, da), hm_mul(hm_add(hm_mul(2.0, j0), j1), dts))),
                                        dtsinv),
                                 dtsinv);
        const double c0 = hm_mul(hm_mul(hm_mul(hm_mul(6.0, hm_add(hm_mul(2.0, da), hm_mul(hm_add(j0, j1), dts))), dtsinv),
                                        dtsinv),
                                 dtsinv);
        const double s1 = hm_add(s0, hm_mul(c0, dts));
        // dt_criterion at t_gl with the old step: |a|, |j|, |s|, |c| on lanes 0 .. 3
        double r = 0.0;
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const double va = __shfl_sync(full, a1, q), vj = __shfl_sync(full, j1, q);
            const double vs = __shfl_sync(full, s1, q), vc = __shfl_sync(full, c0, q);
            const double y = (lane & 2) ? ((lane & 1) ? vc : vs) : ((lane & 1) ? vj : va);
            r = hm_add(r, hm_mul(y, y));
        }
        r = sqrt(r);
        const double a = __shfl_sync(full, r, 0), jj = __shfl_sync(full, r, 1);
        const double sn = __shfl_sync(full, r, 2), cr = __shfl_sync(full, r, 3);
        const double s4 = hm_mul(hm_mul(hm_mul(hm_mul(hm_mul(s0, dts), dts), dts), dts), HM_FOURTH);
        const double c5 = hm_mul(hm_mul(hm_mul(hm_mul(hm_mul(hm_mul(c0, dts), dts), dts), dts), dts), HM_FIFTH);
        const double s3 = hm_mul(hm_mul(hm_mul(hm_mul(s0, dts), dts), dts), HM_THIRD);
        const double c4 = hm_mul(hm_mul(hm_mul(hm_mul(hm_mul(c0, dts), dts), dts), dts), HM_FOURTH);
        if (lane < 3) {
            P.pos[3 * i + c] = hm_add(x1, hm_add(s4, c5));
            P.vel[3 * i + c] = hm_add(v1, hm_add(s3, c4));
            P.acc[3 * i + c] = a1;
            P.jrk[3 * i + c] = j1;
        }
        const double dti =
            hm_mul(eta, sqrt(hm_add(hm_mul(a, sn), hm_mul(jj, jj)) / hm_add(hm_mul(jj, cr), hm_mul(sn, sn))));
        double dnew = dts;
        if (dti < dnew) {
            for (int it = 0; dnew > dti && dnew > dtmin && it < 64; it++) dnew *= 0.5;
        } else if (dti > 2.0 * dnew) {
            if (hm_modulus(tg, 2.0 * dnew, dtmax) == 0.0) dnew = 2.0 * dnew;
        }
        if (lane == 0) {
            P.t[i] = tg;
            P.dt[i] = dnew;
            P.pot[i] = hm_float(F.pot);
        }
        return (unsigned long long)__double_as_longlong(hm_add(tg, dnew));
    }
};

// Start-up step (hermite.c:110-141, timestep.c:24-51): every particle active at t = 0; the new
// force becomes the state and the first step is the largest power-of-two fraction of dtmax
// below eta_s |a|/|j| that divides t.  Counts the steps that fell below dtmin into W.clk->bad.
__device__ __forceinline__ void hm_startup(const HmState& P, const HmWork& W, int i, const G6Out& F, double eta_s,
                                           double dtmax) {
    const double dtmin = dtmax / 2251799813685248.0;
    const double a1[3] = {F.ax, F.ay, F.az};
    const double j1[3] = {hm_float(F.jx), hm_float(F.jy), hm_float(F.jz)};
    double a = 0.0, jj = 0.0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        P.acc[3 * i + c] = a1[c];
        P.jrk[3 * i + c] = j1[c];
        a = hm_add(a, hm_mul(a1[c], a1[c]));
        jj = hm_add(jj, hm_mul(j1[c], j1[c]));
    }
    P.pot[i] = hm_float(F.pot);
    const double dtcrit = hm_mul(eta_s, sqrt(a / jj));
    double d = dtmax;
    for (int it = 0; d > dtcrit && d > dtmin && it < 64; it++) d *= 0.5;
    for (int it = 0; hm_modulus(P.t[i], d, dtmax) != 0.0 && it < 64; it++) {
        d *= 0.5;
        if (d < dtmin) {
            atomicAdd(&W.clk->bad, 1);
            break;
        }
    }
    P.dt[i] = d;
}

// t + dt (bits) of particle tid of a segment, from the state; reset: its time restarts first.
__device__ __forceinline__ unsigned long long hm_next_time(const HmState& P, int seg, int reset) {
    const int i = seg * HM_SEG + (int)threadIdx.x;
    if (i >= P.n) return ~0ull;
    double t = P.t[i];
    if (reset) {
        t = 0.0;
        P.t[i] = 0.0;
    }
    return (unsigned long long)__double_as_longlong(hm_add(t, P.dt[i]));
}

// Phase A for one segment (the whole CTA; b: its particles' t + dt): its record for step `tag`, with
// the particles at the minimum, published after everything the CTA has written before.
__device__ __forceinline__ void hm_segment_min(const HmRun& R, int seg, unsigned long long b, unsigned tag, unsigned slot,
                                               unsigned long long* sm) {
    __shared__ unsigned s_mask[HM_NT / 32];
    const int tid = (int)threadIdx.x;
    const unsigned long long m = block_min_u64<HM_NT>(b, sm);
    const bool at = seg * HM_SEG + tid < R.P.n && b == m;
    const unsigned mask = __ballot_sync(0xffffffffu, at);
    if ((tid & 31) == 0) s_mask[tid >> 5] = mask;
    __syncthreads();
    int c = 0, rank = 0, first = 0, second = 0;
#pragma unroll
    for (int w = 0; w < HM_NT / 32; w++) {
        const unsigned k = s_mask[w];
        if (w == tid >> 5) rank = c + __popc(k & ((1u << (tid & 31)) - 1u));
        if (k) {
            const int f = 32 * w + __ffs(k) - 1;
            const unsigned more = k & (k - 1);
            if (c == 0) {
                first = f;
                if (more) second = 32 * w + __ffs(more) - 1;
            } else if (c == 1) {
                second = f;
            }
        }
        c += __popc(k);
    }
    if (c > 2) {   // more than the record holds: the list
        if (at) R.W.seg_list[((size_t)slot * R.nseg + seg) * HM_SEG + rank] = (unsigned char)tid;
        __syncthreads();
    }
    if (tid == 0) {
        __threadfence();
        const unsigned info = (unsigned)c | (unsigned)first << 9 | (unsigned)second << 17 | slot << 25;
        hm_st(R.W.rec + (size_t)(tag % HM_RSLOTS) * R.nseg + seg, HmWord{m, (unsigned long long)tag << 32 | info});
    }
}

// The j predictor of the library (gravity.c:149-193) on (pos, vel, acc/2, jerk/6, t) of a particle;
// the loads do not need the time that is predicted to.
struct HmJ {
    double t, m, x[3], v[3], a[3], j[3];
    __device__ __forceinline__ void load(const HmState& P, int i) {
        t = __ldcg(P.t + i);
        m = __ldcg(P.mass + i);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            x[c] = __ldcg(P.pos + 3 * i + c);
            v[c] = __ldcg(P.vel + 3 * i + c);
            a[c] = __ldcg(P.acc + 3 * i + c);
            j[c] = __ldcg(P.jrk + 3 * i + c);
        }
    }
    __device__ __forceinline__ G6PredJ predict(int i, double tg, bool ff) const {
        const double d = tg - t, d2 = d * d, d3 = d2 * d;
        double xp[3];
        float vp[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double a2 = a[c] * 0.5, j6 = j[c] * (1.0 / 6.0);
            xp[c] = x[c] + v[c] * d + a2 * d2 + j6 * d3;
            vp[c] = (float)(v[c] + 2.0 * a2 * d + 3.0 * j6 * d2);
        }
        G6PredJ o;
        store_pos(o.p, xp[0], xp[1], xp[2], ff);
        o.m = (float)m;
        o.id = i;
        o.vx = vp[0];
        o.vy = vp[1];
        o.vz = vp[2];
        o.pad = 0.f;
        return o;
    }
};

// Component c of the i-record of active particle i at t_gl.
__device__ __forceinline__ void hm_irecord_c(const HmState& P, int i, int c, double tg, bool ff, G6I& rec) {
    const int k = 3 * i + c;
    const double x = __ldcg(P.pos + k), v = __ldcg(P.vel + k), a = __ldcg(P.acc + k), j = __ldcg(P.jrk + k);
    const double d = hm_sub(tg, __ldcg(P.t + i));
    const double d2 = hm_mul(d, d), d3 = hm_mul(d, d2);
    const double xp = hm_add(hm_add(hm_add(x, hm_mul(v, d)), hm_mul(hm_mul(a, d2), HM_SECOND)),
                             hm_mul(hm_mul(j, d3), HM_THIRD));
    const double vp = hm_add(hm_add(v, hm_mul(a, d)), hm_mul(hm_mul(j, d2), HM_SECOND));
    if (ff) split_ff(xp, (&rec.p.f.xh)[c], (&rec.p.f.xl)[c]);
    else (&rec.p.d.x)[c] = xp;
    (&rec.vx)[c] = (float)vp;
    if (c == 0) rec.id = i;
}

// The i-record of active particle i at t_gl.
__device__ __forceinline__ G6I hm_irecord(const HmState& P, int i, double tg, bool ff) {
    double xp[3], vp[3];
    hm_predict_i(P, i, tg, xp, vp);
    G6I rec;
    store_pos(rec.p, xp[0], xp[1], xp[2], ff);
    rec.vx = (float)vp[0];
    rec.vy = (float)vp[1];
    rec.vz = (float)vp[2];
    rec.id = i;
    rec.h2 = 0.f;
    rec.pad = 0.f;
    return rec;
}

// Phase B' for one segment: j-prediction of its particles; its active ones (in index order from
// offset base) into the active list with their predicted i-records.
__device__ __forceinline__ void hm_segment_build(const HmRun& R, int seg, double tg, int base, bool ff, int* sw) {
    const HmState& P = R.P;
    const HmWork& W = R.W;
    const int i = seg * HM_SEG + (int)threadIdx.x;
    bool act = false;
    if (i < P.n) {
        HmJ J;
        J.load(P, i);
        W.jpred[i] = J.predict(i, tg, ff);
        act = hm_add(P.t[i], P.dt[i]) == tg;
    }
    int tot;
    const int inc = block_scan<HM_NT>(act ? 1 : 0, sw, &tot);
    if (act) {
        const int k = base + inc - 1;
        W.active[k] = i;
        W.irec[k] = hm_irecord(P, i, tg, ff);
    }
}

// The force decomposition of a step with ni active particles (identical in every CTA): the pair
// kernel's shape by ni (i-tile of 16, 32, 64, 128 or 512: j-lanes 16, 8, 4, 2 or two i per
// thread), j-chunks for about one task per CTA, at least minj j per chunk, partial rows and
// task flags within their buffers.
struct HmShape {
    int variant, itile, itiles, nch, ntasks;
};
__device__ __forceinline__ HmShape hm_shape(const HmRun& R, int ni) {
    HmShape h;
    h.variant = ni <= 16 ? 0 : ni <= 32 ? 1 : ni <= 64 ? 2 : ni <= 2048 ? 3 : 4;
    h.itile = h.variant == 4 ? 512 : (16 << h.variant);
    h.itiles = (ni + h.itile - 1) / h.itile;
    const int nj = R.P.n;
    int nch = ((int)gridDim.x + h.itiles - 1) / h.itiles;
    const int by_j = nj / R.minj > 1 ? nj / R.minj : 1;
    nch = nch < by_j ? nch : by_j;
    const long long cap = R.W.part_cap / ((long long)h.itiles * h.itile);
    if (nch > cap) nch = cap > 1 ? (int)cap : 1;
    const int tcap = R.W.task_cap / h.itiles;
    if (nch > tcap) nch = tcap > 1 ? tcap : 1;
    h.nch = nch < 1 ? 1 : nch;
    h.ntasks = h.itiles * h.nch;
    return h;
}

// Wait (all threads of the CTA) until every flag[k] for which need(k) holds equals tag; then the
// data published before those flags is visible to the CTA.  False if a wait gave up.
template <class Need>
__device__ __forceinline__ bool hm_wait_flags(unsigned* flag, int nflag, unsigned tag, HmClock* C, Need need) {
    int ok = 1;
    for (int k = threadIdx.x; k < nflag; k += HM_NT)
        if (need(k)) ok &= hm_spin_until(flag + k, tag, C);
    __threadfence();
    return __syncthreads_and(ok) != 0;
}

// Publish (thread 0, after the CTA's writes): flag = tag.
__device__ __forceinline__ void hm_publish(unsigned* flag, unsigned tag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        *(volatile unsigned*)flag = tag;
    }
}

// The CTA's j-tile of a task over j-lanes: field arrays for the paired form, records otherwise.
__device__ __forceinline__ void hm_stage(unsigned char* smem, int k, const G6PredJ& r, bool ff) {
    if (ff) {
        G6TileSoA<HM_NT>* t = reinterpret_cast<G6TileSoA<HM_NT>*>(smem);
        t->xh[k] = r.p.f.xh;
        t->yh[k] = r.p.f.yh;
        t->zh[k] = r.p.f.zh;
        t->xl[k] = r.p.f.xl;
        t->yl[k] = r.p.f.yl;
        t->zl[k] = r.p.f.zl;
        t->m[k] = r.m;
        t->vx[k] = r.vx;
        t->vy[k] = r.vy;
        t->vz[k] = r.vz;
        t->id[k] = r.id;
    } else {
        reinterpret_cast<G6PredJ*>(smem)[k] = r;
    }
}
// What fills up the last j-pair of an odd paired tile: a massless record far away, whose terms are exact zeros
// (where r^2 overflows, 1/r is 0).  The Newton-refined rsqrt of an overflowed r^2 is NaN: with it the
// tile's last record, whose numbers are in range, and hm_lanes masks that half of the pair (in
// the default build the mask made an interval of 4096 particles 3.81 -> 3.88 ms).
#ifdef PGB_RSQRT_NEWTON
constexpr bool HM_MASK_FILL = true;
#else
constexpr bool HM_MASK_FILL = false;
#endif
__device__ __forceinline__ G6PredJ hm_far() {
    G6PredJ r;
    r.p.f.xh = r.p.f.yh = r.p.f.zh = 1e18f;
    r.p.f.xl = r.p.f.yl = r.p.f.zl = 0.f;
    r.m = r.vx = r.vy = r.vz = r.pad = 0.f;
    r.id = -1;
    return r;
}
__device__ __forceinline__ void hm_stage_tile(unsigned char* smem, int k, int nt, const G6PredJ& r, bool ff) {
    hm_stage(smem, k, r, ff);
    if (HM_MASK_FILL && ff && k == nt - 1 && (nt & 1)) hm_stage(smem, nt, r, ff);
}

// The pair terms of one i-slot and its j-lanes over a tile of nt j, with the arithmetic and the
// summation order of g6_task<HM_NT, 1, JL>: FP32 sums of a lane over the tile, added into the FP64
// sums S.  The paired form (double-float positions) takes two neighbouring lanes a thread, as the two
// halves of paired FP32 instructions (lanes 2p and 2p + 1 of slot tid mod ISL on thread p ISL + slot): half
// of the CTA's threads, half of the instructions and 20 instead of 24 LSU cycles a pair of pairs (N =
// 4096, an interval of 1/8: 13.3 ms against 14.1 with one lane a thread); else one lane a thread.
template <int JL, bool FF>
__device__ __forceinline__ void hm_lanes(const unsigned char* smem, int nt, const G6I& I, float eps2, double (&S)[2][7]) {
    constexpr int ISL = HM_NT / JL;
    const int p = (int)threadIdx.x / ISL;
    if constexpr (FF) {
        if (p >= JL / 2) return;
        const G6TileSoA<HM_NT>* t = reinterpret_cast<const G6TileSoA<HM_NT>*>(smem);
        G6IPair IP;
        IP.nxh = make_float2(-I.p.f.xh, -I.p.f.xh);
        IP.nyh = make_float2(-I.p.f.yh, -I.p.f.yh);
        IP.nzh = make_float2(-I.p.f.zh, -I.p.f.zh);
        IP.nxl = make_float2(-I.p.f.xl, -I.p.f.xl);
        IP.nyl = make_float2(-I.p.f.yl, -I.p.f.yl);
        IP.nzl = make_float2(-I.p.f.zl, -I.p.f.zl);
        IP.vx = I.vx;
        IP.vy = I.vy;
        IP.vz = I.vz;
        IP.id = I.id;
        const float2 z2 = make_float2(0.f, 0.f);
        G6Acc2 a{z2, z2, z2, z2, z2, z2, {0.f, 0.f}};
        float tmin = 0.f;
        auto f2 = [](const float* f) { return *reinterpret_cast<const float2*>(f); };
#pragma unroll 2
        for (int j = 2 * p; j < nt; j += JL)
            g6_jpair<false, true>(f2(t->xh + j), f2(t->yh + j), f2(t->zh + j), f2(t->xl + j), f2(t->yl + j), f2(t->zl + j),
                                  f2(t->m + j), f2(t->vx + j), f2(t->vy + j), f2(t->vz + j),
                                  *reinterpret_cast<const int2*>(t->id + j), HM_MASK_FILL ? nt - j : 2, IP, eps2, a, tmin);
        const float2* v = &a.ax;
#pragma unroll
        for (int q = 0; q < 6; q++) {
            S[0][q] += (double)v[q].x;
            S[1][q] += (double)v[q].y;
        }
        S[0][6] += (double)a.pot[0];
        S[1][6] += (double)a.pot[1];
    } else {
        const G6PredJ* sj = reinterpret_cast<const G6PredJ*>(smem);
        G6Acc a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float kmin = 0.f;
        int kadr = 0;
#pragma unroll 2
        for (int j = p; j < nt; j += JL)
            g6_pair<FF, false, false>(sj[j], 0, I.p, I.vx, I.vy, I.vz, I.id, eps2, 0.f, a, kmin, kadr, nullptr, nullptr, 0);
        S[0][0] += (double)a.ax;
        S[0][1] += (double)a.ay;
        S[0][2] += (double)a.az;
        S[0][3] += (double)a.jx;
        S[0][4] += (double)a.jy;
        S[0][5] += (double)a.jz;
        S[0][6] += (double)a.pot;
    }
}

// The lanes' sums of a task in lane order: component q of slot i ends in red[q * HM_NT + i].
template <int JL, bool FF>
__device__ __forceinline__ void hm_lane_sums(double* red, const double (&S)[2][7]) {
    constexpr int ISL = HM_NT / JL;
    const int tid = (int)threadIdx.x, slot = tid % ISL, p = tid / ISL;
    __syncthreads();
    if (!FF || p < JL / 2) {
#pragma unroll
        for (int q = 0; q < 7; q++) {
            red[q * HM_NT + (FF ? 2 * p : p) * ISL + slot] = S[0][q];
            if (FF) red[q * HM_NT + (2 * p + 1) * ISL + slot] = S[1][q];
        }
    }
    __syncthreads();
    for (int f = tid; f < 7 * ISL; f += HM_NT) {
        double* r = red + (f / ISL) * HM_NT + f % ISL;
        double v = r[0];
#pragma unroll
        for (int l = 1; l < JL; l++) v += r[l * ISL];
        r[0] = v;
    }
    __syncthreads();
}

// Phase C of a small step: the j of the CTA's chunk [j0, j1) against its ni <= ISL i-records in s_i;
// the chunk's first tile is staged.
template <int JL, bool FF>
__device__ __forceinline__ void hm_small_task(const HmRun& R, unsigned char* smem, const G6I* s_i, int ni, int j0, int j1,
                                           double tg, unsigned E) {
    constexpr int ISL = HM_NT / JL;
    const int tid = (int)threadIdx.x, slot = tid % ISL, c = (int)blockIdx.x;
    double S[2][7] = {};
    const G6I I = s_i[slot < ni ? slot : 0];
    for (int jt = j0; jt < j1; jt += HM_NT) {
        const int nt = min(HM_NT, j1 - jt);
        if (jt > j0) {
            HmJ J;
            if (tid < nt) J.load(R.P, jt + tid);
            __syncthreads();
            if (tid < nt) hm_stage_tile(smem, tid, nt, J.predict(jt + tid, tg, FF), FF);
            else if (!HM_MASK_FILL && FF && tid == nt) hm_stage(smem, tid, hm_far(), FF);
            __syncthreads();
        }
        hm_lanes<JL, FF>(smem, nt, I, R.eps2, S);
    }
    double* red = reinterpret_cast<double*>(smem);
    hm_lane_sums<JL, FF>(red, S);
    for (int f = tid; f < HM_SUMW * ni; f += HM_NT) {
        const int k = f / HM_SUMW, w = f % HM_SUMW;
        unsigned u[3];
#pragma unroll
        for (int h = 0; h < 3; h++) {
            const int g = 3 * w + h;   // half g of the seven sums
            u[h] = g < 14 ? reinterpret_cast<const unsigned*>(red + (g / 2) * HM_NT + k)[g % 2] : 0u;
        }
        hm_st(R.W.sums + ((size_t)k * R.W.chunks + c) * HM_SUMW + w,
              HmWord{(unsigned long long)u[1] << 32 | u[0], (unsigned long long)E << 32 | u[2]});
    }
}

// A record of a large step, through L2.
template <class Rec>
__device__ __forceinline__ Rec hm_ldrec(const Rec* p) {
    static_assert(sizeof(Rec) == 48, "three words");
    union {
        uint4 w[3];
        Rec r;
    } u;
#pragma unroll
    for (int q = 0; q < 3; q++) u.w[q] = __ldcg(reinterpret_cast<const uint4*>(p) + q);
    return u.r;
}

// Phase C' of a large step, one i per slot: task T over JL j-lanes; its sums to its partial row, or
// (an unsplit j-range) the finished force to out.
template <int JL, bool FF>
__device__ __forceinline__ void hm_large_task(const HmRun& R, unsigned char* smem, const Task& T, int itile) {
    constexpr int ISL = HM_NT / JL;
    const int tid = (int)threadIdx.x, slot = tid % ISL;
    double S[2][7] = {};
    const G6I I = hm_ldrec(R.W.irec + T.i0 + (slot < T.ni ? slot : 0));
    for (int jt = 0; jt < T.nj; jt += HM_NT) {
        const int nt = min(HM_NT, T.nj - jt);
        __syncthreads();
        if (tid < nt) hm_stage_tile(smem, tid, nt, hm_ldrec(R.W.jpred + T.j0 + jt + tid), FF);
        else if (!HM_MASK_FILL && FF && tid == nt) hm_stage(smem, tid, hm_far(), FF);
        __syncthreads();
        hm_lanes<JL, FF>(smem, nt, I, R.eps2, S);
    }
    double* red = reinterpret_cast<double*>(smem);
    hm_lane_sums<JL, FF>(red, S);
    for (int f = tid; f < 7 * T.ni; f += HM_NT) {
        const int k = f / 7, q = f % 7;
        const double v = red[q * HM_NT + k];
        if (T.group >= 0) (&R.W.partial[(size_t)T.slot * itile + k].ax)[q] = v;
        else (&R.W.out[T.i0 + k].ax)[q] = (q < 6 ? S_ACC : S_POT) * v;
    }
}

// START: the start-up step only, of more than HM_SMALL particles.  It is an instance of its own because the
// small steps' code beside the force loop costs that loop registers (no spills without it, 620 bytes of
// stores with it): 65536 particles 8.1 -> 7.4 ms, 300000 124 -> 111.
template <bool FF, bool START>
__device__ __forceinline__ void hm_run_body(const HmRun& R) {
    const bool startup = START || R.startup;
    __shared__ __align__(16) unsigned char smem[HM_NT * sizeof(G6Out)];
    __shared__ int s_boff[HM_MAXSEG + 1];   // offsets of every segment's active particles (+ ni)
    __shared__ unsigned long long sm[HM_NT / 32];
    __shared__ int sw[HM_NT / 32];
    __shared__ int s_act[HM_SMALL];
    __shared__ G6I s_i[HM_SMALL];
    __shared__ HmWord s_own[HM_OWN];        // this step's records of the CTA's own segments
    __shared__ unsigned s_slot[HM_OWN];     // and the slots of their lists
    __shared__ unsigned long long s_next[HM_NEXT][HM_SEG];   // t + dt of the first own segments' particles
    const HmWork& W = R.W;
    HmClock* C = W.clk;
    const int G = (int)gridDim.x, nseg = R.nseg, tid = (int)threadIdx.x;
    // every CTA carries the clock on by itself, CTA 0 stores it
    unsigned E = R.step0;
    double time = R.time0;
    int t_mod = R.t_mod0;
    // A (once per launch): the segments' records of the current state
    for (int seg = blockIdx.x, own = 0; seg < nseg; seg += G, own++) {
        if (tid == 0) s_slot[own] = 0;
        const unsigned long long b = hm_next_time(R.P, seg, 0);
        if (own < HM_NEXT) s_next[own][tid] = b;
        hm_segment_min(R, seg, b, E, 0, sm);
        __syncthreads();
    }
    __shared__ HmClock k_last;
    if (blockIdx.x == 0 && tid == 0) k_last = *C;
    // the CTA's chunk of a small step, whose first tile's state is read as soon as it is final
    const bool chunk = (int)blockIdx.x < R.nch1;
    const int jc0 = chunk ? (int)((long long)blockIdx.x * R.P.n / R.nch1) : 0;
    const int jc1 = chunk ? (int)((long long)(blockIdx.x + 1) * R.P.n / R.nch1) : 0;
    for (int step = 0;; step++) {
        // the loop condition of banana01.c:146
        if (startup ? step >= 1 : (!(time < R.tend) || step >= R.max_steps)) break;
        // B: every segment's record of this step.  The owners also wait until every CTA has read the
        // records that this step's will replace.
        const HmWord* rec = W.rec + (size_t)(E % HM_RSLOTS) * nseg;
        unsigned long long lo = ~0ull;
        HmWord mine{~0ull, 0ull};   // the record of segment tid
        int ok = 1;
        if (!chunk && (int)blockIdx.x >= nseg) {
            // a CTA without a segment or a chunk of a small step looks at one record until that is there:
            // 296 CTAs reading all of them over and over keep the few L2 slices that hold them busy
            if (tid == 0) ok = hm_wait(C, [&] { return hm_tag(hm_ld(rec + (int)blockIdx.x % nseg)) != E; });
            if (!__syncthreads_and(ok)) return;
        }
        for (int k = tid; k < nseg; k += HM_NT) {
            HmWord v;
            ok &= hm_wait(C, [&] {
                v = hm_ld(rec + k);
                return hm_tag(v) != E;
            });
            lo = v.lo < lo ? v.lo : lo;
            if (k == tid) mine = v;
            if (k % G == (int)blockIdx.x) s_own[k / G] = v;
        }
        const bool has_j = jc0 + tid < jc1;
        if (has_j) ok &= hm_wait(C, [&] { return hm_tag(hm_ld(rec + (jc0 + tid) / HM_SEG)) != E; });
        __threadfence();   // the state behind the records
        // in flight while the step is worked out (in a large step unused, and then perhaps torn: its
        // owners may already be correcting)
        HmJ J;
        if (has_j) J.load(R.P, jc0 + tid);
        if (!__syncthreads_and(ok)) return;
        // the block time, the offsets of the segments' active particles, and the particles of a small step
        const unsigned long long g = block_min_u64<HM_NT>(lo, sm);
        int ni = 0;
        for (int b0 = 0; b0 < nseg; b0 += HM_NT) {
            const int k = b0 + tid;
            HmWord v = mine;
            if (b0 > 0 && k < nseg) v = hm_ld(rec + k);
            const int cnt = (k < nseg && v.lo == g) ? (int)(v.hi & 511) : 0;
            int sum;
            const int first = ni + block_scan<HM_NT>(cnt, sw, &sum) - cnt;
            if (k < nseg) s_boff[k] = first;
            if (cnt > 0 && first + cnt <= HM_SMALL) {
                const unsigned char* list = W.seg_list + ((size_t)((unsigned)v.hi >> 25) * nseg + k) * HM_SEG;
                for (int q = 0; q < cnt; q++) {
                    const int l = cnt <= 2 ? (int)(v.hi >> (9 + 8 * q)) & 255 : (int)__ldcg(list + q);
                    s_act[first + q] = k * HM_SEG + l;
                }
            }
            ni += sum;
        }
        const double tg = __longlong_as_double((long long)g);
        if (tid == 0) s_boff[nseg] = ni;
        __syncthreads();
        if (tid == 0) *(volatile unsigned*)(W.ack + blockIdx.x) = E;   // the records have been read
        // banana01.c:161-179: after a step that ends on a multiple of dtmax the times restart
        // (reset_time, applied with the corrector below) and t_mod counts the interval
        int rs = 0;
        if (!startup) {
            const double q = (double)__double2int_rz(hm_mul(tg, R.dtinv));
            rs = hm_sub(tg, hm_mul(q, R.dtmax)) == 0.0;
        }
        // (a step that resets every particle's time writes state that small steps' tasks read)
        const bool small = !START && ni <= HM_SMALL && !rs;
        HmShape sh;
        if (small) {
            sh.variant = ni <= 16 ? 0 : ni <= 32 ? 1 : ni <= 64 ? 2 : 3;
            sh.itile = 16 << sh.variant;
            sh.itiles = 1;
            sh.nch = sh.ntasks = R.nch1;
        } else {
            sh = hm_shape(R, ni);
        }
        if (blockIdx.x == 0 && tid == 0) {   // the clock's counters, stored when the launch ends
            k_last.t_gl = tg;
            k_last.ni = ni;
            k_last.nch = sh.nch;
            k_last.itile = sh.itile;
            k_last.psteps += ni;
            k_last.bsteps += 1;
            k_last.force_pairs += (long long)ni * R.P.n;
            k_last.variant_steps[sh.variant] += 1;
        }
        // of a large step of two i per thread: the tasks of the last, part-filled round are halved by
        // their i (one per thread), so that the round ends sooner (16384 active particles: 320 tasks on
        // 296 CTAs)
        const int ntail = !small && sh.variant == 4 && 2 * (sh.ntasks % G) <= G ? sh.ntasks % G : 0;
        const int nfull = sh.ntasks - ntail;
        if (small) {
            // C
            if (chunk) {
                for (int f = tid; f < 3 * ni; f += HM_NT) hm_irecord_c(R.P, s_act[f / 3], f % 3, tg, FF, s_i[f / 3]);
                if (has_j) hm_stage_tile(smem, tid, min(HM_NT, jc1 - jc0), J.predict(jc0 + tid, tg, FF), FF);
                else if (!HM_MASK_FILL && FF && jc0 + tid == jc1) hm_stage(smem, tid, hm_far(), FF);
                __syncthreads();
                if (sh.variant == 0) hm_small_task<16, FF>(R, smem, s_i, ni, jc0, jc1, tg, E);
                else if (sh.variant == 1) hm_small_task<8, FF>(R, smem, s_i, ni, jc0, jc1, tg, E);
                else if (sh.variant == 2) hm_small_task<4, FF>(R, smem, s_i, ni, jc0, jc1, tg, E);
                else hm_small_task<2, FF>(R, smem, s_i, ni, jc0, jc1, tg, E);
            }
        } else {
            // B'
            for (int seg = blockIdx.x; seg < nseg; seg += G) {
                __syncthreads();
                hm_segment_build(R, seg, tg, s_boff[seg], FF, sw);
                hm_publish(W.seg_flag + seg, E);
            }
            __syncthreads();
            // C': force tasks, each after the segments it reads are built
            G6Args a;
            a.ipart = W.irec;
            a.jpred = W.jpred;
            a.eps2 = R.eps2;
            a.tasks = nullptr;
            a.ntasks = sh.ntasks;
            a.task_counter = nullptr;
            a.groups = nullptr;
            a.group_counters = nullptr;
            a.partial = W.partial;
            a.out = W.out;
            a.itile = sh.itile;
            a.nb_count = nullptr;
            a.nb_list = nullptr;
            a.nb_maxlen = 0;
            a.reg_ni = ni;
            a.reg_nj = R.P.n;
            a.reg_nch = sh.nch;
            a.partial_only = true;
            for (int u = blockIdx.x; u < nfull + 2 * ntail; u += G) {
                const int t = u < nfull ? u : nfull + (u - nfull) / 2;
                Task T = regular_task(a, t);
                const int js0 = T.j0 / HM_SEG, js1 = (T.j0 + T.nj - 1) / HM_SEG;
                const int k0 = T.i0, k1 = T.i0 + T.ni;
                if (!hm_wait_flags(W.seg_flag, nseg, E, C, [&](int s) {
                        return (s >= js0 && s <= js1) || (s_boff[s] < k1 && s_boff[s + 1] > k0);
                    })) return;
                if (u >= nfull) {
                    const int h = (u - nfull) & 1;
                    T.i0 += h * HM_NT;
                    T.ni = min(HM_NT, T.ni - h * HM_NT);
                    G6Args b = a;
                    b.partial += h * HM_NT;
                    if (T.ni > 0) g6_task<HM_NT, 1, 1, FF, false, false>(b, T, smem);
                    hm_publish(h ? W.task_flag + W.task_cap + t - nfull : W.task_flag + t, E);
                    continue;
                }
                switch (sh.variant) {
                    case 0: hm_large_task<16, FF>(R, smem, T, sh.itile); break;
                    case 1: hm_large_task<8, FF>(R, smem, T, sh.itile); break;
                    case 2: hm_large_task<4, FF>(R, smem, T, sh.itile); break;
                    case 3: hm_large_task<2, FF>(R, smem, T, sh.itile); break;
                    default: g6_task<HM_NT, 2, 1, FF, false, false>(a, T, smem); break;
                }
                hm_publish(W.task_flag + t, E);
            }
        }
        // D + next A, segment by segment (the CTA that owns it): the force of each active particle
        // once its chunks are done, the corrector (or start-up step) of each, one warp each; the time
        // reset; the segment's new record
        const int wpc = HM_NT / 32;
        // this step's records replace those of step E + 1 - HM_RSLOTS, which every CTA has read when it
        // has acknowledged that step (long ago, but for a CTA that was held up)
        if ((int)blockIdx.x < nseg) {
            ok = 1;
            for (int k = tid; k < G; k += HM_NT)
                ok &= hm_wait(C, [&] { return (int)(*(volatile unsigned*)(W.ack + k) - (E + 1 - HM_RSLOTS)) < 0; });
            if (!__syncthreads_and(ok)) return;
        }
        for (int seg = blockIdx.x, own = 0; seg < nseg; seg += G, own++) {
            const int k0 = s_boff[seg], k1 = s_boff[seg + 1];
            if (small && k1 == k0) {
                // a segment that the step leaves as it is: the same record for the next step
                if (tid == 0) {
                    const HmWord v = s_own[own];
                    hm_st(W.rec + (size_t)((E + 1) % HM_RSLOTS) * nseg + seg,
                          HmWord{v.lo, (unsigned long long)(E + 1) << 32 | (v.hi & 0xffffffffull)});
                }
                continue;
            }
            ok = 1;
            if (!small && k1 > k0) {
                const int it0 = k0 / sh.itile, it1 = (k1 - 1) / sh.itile;
                if (!hm_wait_flags(W.task_flag, sh.ntasks, E, C,
                                   [&](int t) { return t / sh.nch >= it0 && t / sh.nch <= it1; })) return;
                if (ntail > 0 && !hm_wait_flags(W.task_flag + W.task_cap, ntail, E, C, [&](int h) {
                        return (nfull + h) / sh.nch >= it0 && (nfull + h) / sh.nch <= it1;
                    })) return;
            }
            for (int k = k0 + (tid >> 5); k < k1; k += wpc) {
                const int i = small ? s_act[k] : W.active[k];
                HmOwn O;
                if (!startup) O.load(R.P, i, tg);   // before the force is there
                G6Out F;
                if (small) ok &= hm_force_small(W, k, sh.nch, E, F);
                else F = hm_force_of(W, k, sh.nch, sh.itile);
                if (!ok) break;
                if (small && (tid & 31) == 0) W.active[k] = i;
                if (startup) {
                    if ((tid & 31) == 0) hm_startup(R.P, W, i, F, R.eta_s, R.dtmax);
                } else {
                    const unsigned long long b = O.correct(R.P, i, tg, F, R.eta, R.dtmax);
                    if (own < HM_NEXT && (tid & 31) == 0) s_next[own][i - seg * HM_SEG] = b;
                }
            }
            if (!__syncthreads_and(ok)) return;   // and the segment's updated state
            unsigned long long b;
            if (own < HM_NEXT && !rs && !startup) {
                b = s_next[own][tid];
            } else {
                b = hm_next_time(R.P, seg, rs);
                if (own < HM_NEXT) s_next[own][tid] = b;
            }
            const unsigned slot = (s_slot[own] + 1) % HM_RSLOTS;
            hm_segment_min(R, seg, b, E + 1, slot, sm);
            __syncthreads();
            if (tid == 0) s_slot[own] = slot;
        }
        if (!startup) {
            t_mod += rs;
            time = rs ? hm_add(hm_mul((double)t_mod, R.dtmax), 0.0) : hm_add(hm_mul((double)t_mod, R.dtmax), tg);
        }
        E++;
    }
    if (blockIdx.x == 0 && tid == 0) {
        C->t_gl = k_last.t_gl;
        C->ni = k_last.ni;
        C->nch = k_last.nch;
        C->itile = k_last.itile;
        C->psteps = k_last.psteps;
        C->bsteps = k_last.bsteps;
        C->force_pairs = k_last.force_pairs;
#pragma unroll
        for (int v = 0; v < 5; v++) C->variant_steps[v] = k_last.variant_steps[v];
        if (!startup) {
            C->t_mod = t_mod;
            C->time = time;
        }
    }
}

// The step kernel: the body above, then every CTA counts its return (on every path, the early
// returns of a wait that gave up included), so the host can tell that the whole grid has left.
template <bool FF, bool START>
__global__ void __launch_bounds__(HM_NT, 2) hm_run_kernel(const __grid_constant__ HmRun R) {
    hm_run_body<FF, START>(R);
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(&R.W.clk->exits, 1);
}

// Kinetic and potential energy (calc_energy.c:9-33): ek = sum m v^2 / 2, ew = sum m pot / 2.
// One CTA, fixed summation order: the result does not depend on the launch.
__global__ void __launch_bounds__(1024) hm_energy_kernel(HmState P, double* out) {
    __shared__ double sk[1024], sp[1024];
    double k = 0.0, w = 0.0;
    for (int i = threadIdx.x; i < P.n; i += 1024) {
        const double vx = P.vel[3 * i], vy = P.vel[3 * i + 1], vz = P.vel[3 * i + 2];
        k += P.mass[i] * (vx * vx + vy * vy + vz * vz);
        w += P.mass[i] * P.pot[i];
    }
    sk[threadIdx.x] = k;
    sp[threadIdx.x] = w;
    __syncthreads();
    for (int o = 512; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sk[threadIdx.x] += sk[threadIdx.x + o];
            sp[threadIdx.x] += sp[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = 0.5 * sk[0];
        out[1] = 0.5 * sp[0];
    }
}

}  // namespace pgb
