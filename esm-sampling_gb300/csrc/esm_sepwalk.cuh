// The walk of the separable storage moves (the state-of-charge atoms of a storage field: storage
// units at distinct nodes and nothing else) by blocks of warps, a batch of (step, replica) tasks at
// a time.
//
// The line potential of such a move is a sum of one-dimensional piecewise-linear unit functions,
// each with at most ten kinks in a walking direction: its clamps (0 and 1 of the state of charge,
// the primary breakpoints of walk!, src/local.jl:1294), its storage thresholds and the zero
// crossings of its two node balances (the secondary roots of piece_roots!, :1267). The walk visits
// the union of those points in walking order, stops at the first clamp where the potential stands
// more than maxnats above its minimum, and takes ray steps once every clamp is behind.
//
// A list holds one direction of one task's walk. Its work splits into parts of different width:
//   1. events, one lane per (list, unit): the unit's pieces up to the window end, the nearest clamp
//      of the list (98 % of the walks of a production chain stop there);
//   2. order, one warp per list (bitonic, in shared memory) or, for a short list, its scan lane;
//   3. scan, one lane per list: the summed slope, the potential and the stop test, event by event
//      in double, in the order of the one-lane walk, so that every sum has the same bits;
//   4. segment masses, one warp per task (a lane per segment);
//   5. draw, one lane per task: the sums over the segments are again taken in order;
//   6. commit, one lane per (task, unit).
// A list that its window does not end gets the next clamp's window (every event made again: 2 % of
// the lists at 40 nodes), at last one without an end, in which the ray steps follow.
//
// Why this split: the one-lane walk (Lane::walk_sep) runs a heap of units per lane; its lanes sit
// in different units and pieces, and its unit and heap state, several KB a lane, goes through L2.
// Here the events, which are nearly all of the arithmetic, are made by lanes in step, with the
// unit in registers, and the lists stay in shared memory. What bounds it now: the latency of the
// events' dependent arithmetic and of the scan, at 16 warps per SM in FP32 (four blocks by registers and
// by shared memory) and 8 in FP64 (two, by registers); the warps of a batch of few long lists wait for its
// scan. Measured for one move at T = 2920, 64 replicas (93440 tasks), FP32, one-lane walk
// and block walk: 40 units 16.4 and 3.2 ms, 20 units 5.7 and 1.8 ms, 10 units 2.1 and 1.2 ms, 7 units
// 1.4 and 0.7 ms.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "esm_common.cuh"

namespace esm {

#define ESM_SEP_WARPS 4           // warps of a block
#define ESM_SEP_LISTS 128         // lists of a batch at most: one scan thread each
#define ESM_SEP_EV 12             // events of one unit in one direction, at most (ten by the unit's shape)
#define ESM_SEP_SHORT 8           // lists up to this length are sorted by their scan lane
// Moves up to this many units keep what the round-off scales and the ray steps need (18 bytes an entry
// in FP32, and room for ray points). Larger moves do without (14 bytes): of their draws 0.3 % (7 units)
// to 0.01 % (40 units) need the scales and run again, alone; of those of 2 units 27 % would.
#define ESM_SEP_FULL 4

// The FP32 potential of a unit decides which way a draw on an almost flat segment goes, so the block
// walk gives every value the rounding that the one-lane walk (Lane::unit_val, Lane::commit) gives it:
// the contractions of the FP32 build are written out here (fma_rn; in the FP64 build, which has none,
// a product and a sum) instead of left to the compiler, which chooses them per function.
__device__ inline float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ inline double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ inline float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ inline double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ inline float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ inline double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ inline float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ inline double fma_rn(double a, double b, double c) { return __dadd_rn(__dmul_rn(a, b), c); }

// FP32 to FP64 and back (to nearest even) with integer instructions where the value is normal: a
// conversion, like every FP64 instruction, holds a scheduler's FP64 unit for 64 cycles whatever the
// number of active lanes (measured; 16 to 19 cycles per SM), and the scan lanes convert at every event.
// (the other values in calls of their own, so that they are not converted on every lane)
static __device__ __noinline__ double sep_widen_any(float x) { return (double)x; }
static __device__ __noinline__ float sep_narrow_any(double x) { return (float)x; }
__device__ __forceinline__ double sep_widen(float x) {
    unsigned u = __float_as_uint(x), m = u & 0x7fffffffu;
    if (m != 0 && m - 0x00800000u >= 0x7f000000u) return sep_widen_any(x);
    unsigned h = m == 0 ? 0u : (m >> 3) + 0x38000000u;
    return __hiloint2double((int)((u & 0x80000000u) | h), (int)(u << 29));
}
__device__ inline double sep_widen(double x) { return x; }
__device__ __forceinline__ float sep_narrow(double x, float) {
    unsigned h = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x), m = h & 0x7fffffffu;
    if (m - 0x38100000u >= 0x0fd00000u) return (m | l) == 0 ? __uint_as_float(h) : sep_narrow_any(x);
    unsigned f = ((m - 0x38000000u) << 3) | (l >> 29);
    unsigned rem = l & 0x1fffffffu;
    f += rem > 0x10000000u || (rem == 0x10000000u && (f & 1u));
    return __uint_as_float((h & 0x80000000u) | f);
}
__device__ inline double sep_narrow(double x, double) { return x; }
// the sums over a list, in double in both builds
template <class real>
__device__ __forceinline__ double sep_fma(double a, double b, double c) {
    return sizeof(real) == 4 ? __fma_rn(a, b, c) : __dadd_rn(__dmul_rn(a, b), c);
}
// the double of a high word in integer order (and a low word of zeros)
__device__ __forceinline__ double sep_word(int w) {
    return __hiloint2double(w ^ ((w >> 31) & 0x7fffffff), w < 0 ? -1 : 0);
}
// a float at least |x| (of FP32 size) and no more than 2^-19 above it
__device__ __forceinline__ float sep_above(double x) {
    unsigned m = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return __uint_as_float(m < 0x38000000u ? 8u : ((m - 0x38000000u) << 3) + 8u);
}

// The draw inside a segment (sample_line!, src/local.jl:1501; a function of its own, so that its
// contractions depend on nothing around it).
template <class real>
__device__ __noinline__ real sep_pick(real p0, real p1, real g, real L, real uoff, real flat) {
    return (g >= 0 || fabs(g * L) < flat) ? p0 + Lane<real>::trexp_offset(uoff, g, L, flat)
                                          : p1 - Lane<real>::trexp_offset(uoff, -g, L, flat);
}

// How a list is laid out: the entries of a batch's list, those of a small move's, and those of a task
// that runs alone, with room for the events beyond the last clamp (two a unit) and for every ray point.
enum { SEP_BATCH = 0, SEP_SMALL = 1, SEP_SOLE = 2 };
__host__ __device__ inline int sep_kind(int nu, bool alone) { return alone ? SEP_SOLE : nu <= ESM_SEP_FULL ? SEP_SMALL : SEP_BATCH; }
__host__ __device__ inline int sep_events(int nu, int maxpts, int kind) {
    int e = ESM_SEP_EV * nu;
    return (e < maxpts ? e : maxpts) + (kind == SEP_BATCH ? 1 : 2 * nu);
}
__host__ __device__ inline int sep_entries(int nu, int maxpts, int kind) {
    int more = kind == SEP_BATCH ? 0 : 2 * nu + (kind == SEP_SMALL ? 8 : 84);
    return (sep_events(nu, maxpts, kind) + more + 1) & ~1;
}
// The longest list that is sorted in registers; a longer one takes a buffer in global memory.
template <class real>
__host__ __device__ constexpr int sep_regs() {
    return sizeof(real) == 4 ? 256 : 128;
}
// Shared memory of one list (SepList).
template <class real>
__host__ __device__ inline int sep_list_bytes(int nu, int maxpts, int kind) {
    int n = sep_entries(nu, maxpts, kind);
    return (((int)sizeof(real) * ((kind == SEP_BATCH ? 3 : 4) * n + nu) + (int)sizeof(real) / 2 * n) + 15) & ~15;
}
// shared memory of the move's units
template <class real>
__host__ __device__ inline int sep_unit_bytes(int nu) {
    return ((2 * (int)sizeof(int) + 7 * (int)sizeof(real)) * nu + 15) & ~15;
}

template <class real>
struct SepUnits {  // the move's storage units (shared memory)
    int *j, *n;
    real *a, *k, *h, *qt, *ein, *eout, *mc;
    __device__ SepUnits(char *p, int nu) {
        a = (real *)p;
        k = a + nu;
        h = k + nu;
        qt = h + nu;
        ein = qt + nu;
        eout = ein + nu;
        mc = eout + nu;
        j = (int *)(mc + nu);
        n = j + nu;
    }
};

// One direction of one task (shared memory). An event comes with its key (sgn * t), its slot and the
// unit's slopes before and after it (x, y of its pair). In order, an entry of a batch's list has the key,
// negative for a clamp, and the change of the summed slope in double over x and y; the scan leaves the
// potential there, which masses() rounds into x, and the segment masses go to y. The other lists keep the pairs by slot; the scan leaves the
// potential and its round-off scale in x and y, the masses have an array.
template <class real>
struct SepPair {
    real x, y;
};
// a slot with the event's clamp flag (bit 15); in the FP64 build, whose sums have other last bits in
// another order, also the unit (bits 16 ..), by which events of one time are ordered
template <class real>
struct SepSlot {
    using type = unsigned short;
};
template <>
struct SepSlot<double> {
    using type = unsigned int;
};
template <class real>
struct SepList {
    using slot_t = typename SepSlot<real>::type;
    SepPair<real> *pair;
    real *key, *sl, *m;
    slot_t *slot;
    __device__ __forceinline__ SepList(char *p, int n, int nu, bool full) {
        pair = (SepPair<real> *)p;
        key = (real *)(pair + n);
        sl = key + n;
        m = sl + nu;
        slot = (slot_t *)(full ? m + n : m);
    }
};
template <class real>
__device__ __forceinline__ void sep_put(SepPair<real> &p, double v) {
    if constexpr (sizeof(real) == 4)
        *(double *)&p = v;
    else
        p.x = v;
}
template <class real>
__device__ __forceinline__ double sep_get(const SepPair<real> &p) {
    if constexpr (sizeof(real) == 4)
        return *(const double *)&p;
    else
        return p.x;
}

// SEP_REDO: left to the one-lane walk. In FP32 a list's events of one time stand in an order of the list's
// own, which depends on the lists beside it; the one-lane walk's comes from its heap. Neither the points'
// times and potentials nor the stop tests depend on it, but two things do: which of the group's events come
// before a point cap that cuts it, and the round-off scale of the group's last point. A walk that they
// decide is walked again by k_move.
enum { SEP_OPEN = 2, SEP_PROPER = 1, SEP_IMPROPER = 0, SEP_GUARD = -1, SEP_ALONE = -2, SEP_REDO = -3 };

// One storage term of a unit (its step tau or its step tau - 1) at the start: d0, its piece, the
// linear coefficients there and its parts.
template <class real>
struct SepTerm {
    real d0, si, sr, sp, inj, run, pen;
    int piece;
};
// A unit in the walk: its constants and its two terms.
template <class real>
struct SepUnit {
    real a, k, h, ein, eout, qt, e0, s0w, s0a;
    real A, P, X;  // cost per unit of running part, penalty part and box excess
    SepTerm<real> w, t;
    int pos, posa;  // the unit's node slots at tau and tau - 1 (LineWalk)

    // soc_parts at d, whose charging part pc = d / ein the caller has
    __device__ __forceinline__ void parts(real d, real pc, real *inj, real *run, real *pen) const {
        real x = mul_rn(-d, eout), m = fmin(x, real(1)), y = sub_rn(x, real(1));
        bool up = d >= 0;
        real c = ein > 0 ? pc : real(0);
        *inj = up ? c : -m;
        *run = up ? c : m;
        real pu = add_rn(c > 1 ? sub_rn(c, real(1)) : real(0), ein <= 0 ? d : real(0));
        real pd = (qt <= 0 && y > 0) ? y : real(0);
        *pen = up ? pu : pd;
    }
    __device__ __forceinline__ int piece(real d, real pc) const {
        return d >= 0 ? ((ein > 0 && pc > 1) ? 1 : 0) : (mul_rn(-d, eout) >= 1 ? 3 : 2);
    }
    __device__ __forceinline__ void start(SepTerm<real> &T, real d0) const {
        T.d0 = d0;
        real pc = d0 / ein;
        T.piece = piece(d0, pc);
        real r = real(1) / ein;
        T.si = T.piece == 0 ? (ein > 0 ? r : real(0)) : T.piece == 1 ? r : T.piece == 2 ? eout : real(0);
        T.sr = T.piece <= 1 ? T.si : T.piece == 2 ? -eout : real(0);
        T.sp = T.piece == 0 ? (ein <= 0 ? real(1) : real(0))
               : T.piece == 1 ? T.si
               : T.piece == 2 ? real(0)
                              : (qt <= 0 ? -eout : real(0));
        parts(d0, pc, &T.inj, &T.run, &T.pen);
    }
    // soc_diff of a term whose d0 changes by dd and whose box excess changes by dex; *di the injection
    // change per unit capacity, *d1 the new d
    __device__ __forceinline__ real cost(const SepTerm<real> &T, real dd, real dex, real *di, real *d1) const {
        real dn = add_rn(T.d0, dd);
        *d1 = dn;
        real pc = dn / ein;
        bool same = piece(dn, pc) == T.piece;
        real inj, run, pen;
        parts(dn, pc, &inj, &run, &pen);
        real dinj = same ? mul_rn(T.si, dd) : sub_rn(inj, T.inj);
        real drun = same ? mul_rn(T.sr, dd) : sub_rn(run, T.run);
        real dpen = same ? mul_rn(T.sp, dd) : sub_rn(pen, T.pen);
        *di = dinj;
        return fma_rn(X, dex, fma_rn(A, drun, mul_rn(P, dpen)));
    }
    __device__ __forceinline__ real soc(const SepTerm<real> &T, real dd, real dex, real *dj) const {
        real di, d1;
        real c = cost(T, dd, dex, &di, &d1);
        *dj = mul_rn(k, di);
        return c;
    }
    // the unit of slot q from its table and state
    __device__ __forceinline__ void load(const DevModel<real> &M, const SepUnits<real> &U, int q, real e0_, real e1c,
                                         real emc) {
        load(M, U.k[q], U.h[q], U.qt[q], U.ein[q], U.eout[q], U.mc[q], U.a[q], e0_, e1c, emc);
    }
    __device__ __forceinline__ void load(const DevModel<real> &M, real k_, real h_, real qt_, real ein_, real eout_,
                                         real mc, real a_, real e0_, real e1c, real emc) {
        a = a_;
        k = k_;
        h = h_;
        qt = qt_;
        ein = ein_;
        eout = eout_;
        e0 = e0_;
        real wt = add_rn(k, M.kappa0), dt = M.dt, cv = M.c_viol;
        A = mul_rn(mul_rn(dt, mc), k);
        P = mul_rn(mul_rn(cv, dt), wt);
        X = mul_rn(mul_rn(cv, wt), h);
        real ec = clampr<real>(e0, 0, 1);
        start(w, sub_rn(mul_rn(h, sub_rn(e1c, ec)) / dt, qt));
        start(t, sub_rn(mul_rn(h, sub_rn(ec, emc)) / dt, qt));
    }
    // the cost and injection changes of step tau and step tau - 1 when the state of charge moves by x
    __device__ __forceinline__ void move(const DevModel<real> &M, real x, real *cw, real *ca, real *djw,
                                         real *dja) const {
        // clamp_diff
        real y1 = add_rn(e0, x);
        real c0 = clampr<real>(e0, 0, 1), c1 = clampr<real>(y1, 0, 1);
        bool in = e0 > 0 && e0 < 1 && y1 > 0 && y1 < 1, above = e0 >= 1 && y1 >= 1, below = e0 <= 0 && y1 <= 0;
        real dc = in ? x : (above || below) ? real(0) : sub_rn(c1, c0);
        real dex = in ? real(0) : above ? x : below ? -x : sub_rn(fabs(sub_rn(y1, c1)), fabs(sub_rn(e0, c0)));
        real dd = mul_rn(h, dc) / M.dt;
        *cw = soc(w, -dd, dex, djw);
        *ca = soc(t, dd, real(0), dja);
    }
    __device__ __forceinline__ static real phi(real S0, real dS, real cs, real cd) {  // phibal_diff
        real S1 = add_rn(S0, dS);
        real lin = S0 > 0 ? mul_rn(cs, dS) : mul_rn(-cd, dS);
        real far = fma_rn(S1 > 0 ? cs : -cd, S1, -mul_rn(S0 > 0 ? cs : -cd, S0));
        return (S0 > 0 && S1 > 0) || (S0 < 0 && S1 < 0) ? lin : far;
    }
    // beta * (cost change) at t, with the two node balances (Lane::unit_val)
    __device__ __forceinline__ real val(const DevModel<real> &M, real tt, real *Sw, real *Sa) const {
        real cw, ca, djw, dja;
        move(M, mul_rn(tt, a), &cw, &ca, &djw, &dja);
        *Sw = add_rn(s0w, djw);
        *Sa = add_rn(s0a, dja);
        real pw = phi(s0w, djw, M.c_shed, M.c_dump), pa = phi(s0a, dja, M.c_shed, M.c_dump);
        return mul_rn(M.beta_v, fma_rn(M.dt, pa, add_rn(fma_rn(M.dt, pw, cw), ca)));
    }
};

template <class real>
__device__ __forceinline__ bool sep_root(real a, real b, real lo, real hi, real sgn, real *x) {
    if ((a < 0) != (b < 0) && a != b) {
        real xx = lo + (hi - lo) * a / (a - b);
        if (sgn * (xx - lo) > 0 && sgn * (hi - xx) > 0) {
            *x = xx;
            return true;
        }
    }
    return false;
}

// The block's shared state of a batch.
template <class real>
struct SepBlock {
    real W[ESM_SEP_LISTS];       // window end (sgn * t; infinite: none)
    int n[ESM_SEP_LISTS];        // events of the list
    int before[ESM_SEP_LISTS];   // those before the window end
    int ncl[ESM_SEP_LISTS];      // clamps ahead of the start
    int st[ESM_SEP_LISTS];       // SEP_*
    int np[ESM_SEP_LISTS];       // points
    int ray[ESM_SEP_LISTS];      // first point of the ray phase, whose points follow the events
    float ab[ESM_SEP_LISTS];     // the summed magnitudes of the units' slopes (an upper bound, FP32)
    real t[ESM_SEP_LISTS / 2];   // the task's draw
    int alone[ESM_SEP_LISTS / 2];
    int nalone, batch;
};

template <class real>
struct SepWalk {
    const DevModel<real> &M;
    const SepUnits<real> &U;
    SepBlock<real> &B;
    char *lists;
    int nu, maxe, maxent, lbytes;  // units, events and entries per list, bytes of a list
    bool full, alone;              // the pairs by slot (not SEP_BATCH); SEP_SOLE
    int lane;

    __device__ __forceinline__ SepList<real> list(int l) const {
        return SepList<real>(lists + (size_t)l * lbytes, maxent, nu, full);
    }
    __device__ __forceinline__ size_t ix(int x, int t, int rep) const { return sidx(x, t, rep, M.T, M.R); }

    // The window end of list l, of which this lane holds the units q0, q0 + qstep, ...: the nearest
    // clamp beyond `after` (sgn * t), over the lanes of the list (those nl apart); and the count of
    // the clamps ahead of the start.
    __device__ __forceinline__ real next_clamp(int q0, int qstep, int nl, int tau, int rep, real sgn, real after,
                                               int *ncl) const {
        real best = real(INFINITY);
        int cnt = 0;
        for (int q = q0; q < nu; q += qstep) {
            real a = U.a[q], e0 = M.e[ix(U.j[q], tau, rep)];
            real c0 = (real(0) - e0) / a, c1 = (real(1) - e0) / a;
            if (isfinite(c0) && sgn * c0 > 0) {
                ++cnt;
                if (sgn * c0 > after) best = fmin(best, sgn * c0);
            }
            if (isfinite(c1) && sgn * c1 > 0) {
                ++cnt;
                if (sgn * c1 > after) best = fmin(best, sgn * c1);
            }
        }
        for (int o = nl; o < 32; o <<= 1) {
            best = fmin(best, __shfl_xor_sync(0xffffffffu, best, o));
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        }
        *ncl = cnt;
        return best;
    }

    // The events of a warp's nl lists (a power of two; this lane's list is l, its units q0, q0 +
    // qstep, ...) up to the window end Wk, appended to the lists in lane order, and every unit's
    // slope at the start; *before the events before the window end. Each round takes one unit per lane through its pieces (unit_piece and
    // unit_next of the one-lane walk): an iteration has one evaluation and gives at most one event,
    // the previous one, whose outgoing slope the evaluation tells. Returns the list's event count.
    __device__ __forceinline__ int events(int l, bool on, int q0, int qstep, int nl, int tau, int taum, int tau1,
                                          int rep, real sgn, real Wk, int *before) const {
        // what a lane evaluates next: the end of the piece at t, a node-balance root inside it, its
        // end again (known), the slope beyond the last root; or it hands out its last event; or nothing
        enum { PIECE, ROOT, END, TAIL, FLUSH, DONE };
        const real INF = real(INFINITY);
        SepList<real> A = list(l);
        unsigned mine = 0;  // the lanes of this list
        for (int i = lane & (nl - 1); i < 32; i += nl) mine |= 1u << i;
        unsigned below = mine & ((1u << lane) - 1u);
        int cnt = 0, last = 0;
        int rounds = (nu + qstep - 1) / qstep;
        for (int rd = 0; rd < rounds; ++rd) {
            int q = q0 + rd * qstep;
            int st = on && q < nu ? PIECE : DONE;
            SepUnit<real> u{};
            real ck[8];  // the unit's clamps (0, 1) and thresholds as sgn * t (infinite: none)
#pragma unroll
            for (int i = 0; i < 8; ++i) ck[i] = INF;
            if (st == PIECE) {
                int j = U.j[q], n = U.n[q];
                real e0 = M.e[ix(j, tau, rep)], e1 = M.e[ix(j, tau1, rep)], em = M.e[ix(j, taum, rep)];
                u.s0w = M.r[ix(n, tau, rep)];
                u.s0a = M.r[ix(n, taum, rep)];
                real e1c = clampr<real>(e1, 0, 1), emc = clampr<real>(em, 0, 1);
                u.load(M, U, q, e0, e1c, emc);
                real h = u.h, qt = u.qt, dt = M.dt;
                auto cand = [&](real x) -> real {
                    real tc = x / u.a;
                    return isfinite(tc) ? sgn * tc : INF;
                };
                ck[0] = cand(real(0) - e0);
                ck[1] = cand(real(1) - e0);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    real th = i == 0 ? real(0) : i == 1 ? u.ein : real(-1) / u.eout;
                    if (i == 1 && !(u.ein > 0)) continue;
                    if (i == 2 && !(u.eout > 0)) continue;
                    real xw = e1c - e0 - (th + qt) * dt / h;
                    if (e0 + xw >= 0 && e0 + xw <= 1) ck[2 + 2 * i] = cand(xw);
                    real xa = emc - e0 + (th + qt) * dt / h;
                    if (e0 + xa >= 0 && e0 + xa <= 1) ck[3 + 2 * i] = cand(xa);
                }
            }
            real t = 0, f = 0, sw0 = u.s0w, sa0 = u.s0a;            // the position; the balances at its piece's start
            real tE = 0, fE = 0, swE = 0, saE = 0, r0 = 0, r1 = 0;  // the piece's end and roots
            int nr = 0;
            bool have = false, prim = false, first = true;
            bool pend = false, pcl = false;  // the event at the position, not yet handed out
            real psl = 0;                    // the slope up to it
            while (__any_sync(0xffffffffu, st != DONE)) {
                bool emit = false, xcl = false, flush = st == FLUSH;
                real xt = 0, xlo = 0, xhi = 0;
                if (flush) {
                    emit = true;
                    xt = t;
                    xlo = xhi = psl;
                    xcl = pcl;
                    st = DONE;
                } else if (st != DONE) {
                    real te;
                    if (st == PIECE) {
                        real tk = sgn * t, best = INF;
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            if (ck[i] > tk) best = fmin(best, ck[i]);
                        have = best < INF;
                        prim = best == ck[0] || best == ck[1];
                        tE = have ? sgn * best : t + sgn * fmax(real(1), fabs(t));
                        te = tE;
                    } else {
                        te = st == ROOT ? r0 : st == END ? tE : t + sgn * fmax(real(1), fabs(t));
                    }
                    real v = fE, Sw = swE, Sa = saE;
                    if (st != END) v = u.val(M, te, &Sw, &Sa);
                    bool ev = true;     // an event at te (else only the slope to infinity)
                    bool known = true;  // the slope up to te
                    bool cl = false;
                    if (st == PIECE) {
                        fE = v;
                        swE = Sw;
                        saE = Sa;
                        nr = 0;
                        real x;
                        bool hit;
                        if (have) {
                            hit = sep_root<real>(sw0, Sw, t, tE, sgn, &x);
                        } else {  // linear to infinity: a crossing anywhere ahead
                            x = t + (tE - t) * sw0 / (sw0 - Sw);
                            hit = sw0 != Sw && isfinite(x) && sgn * (x - t) > 0;
                        }
                        if (hit) {
                            r0 = x;
                            nr = 1;
                        }
                        if (have) {
                            hit = sep_root<real>(sa0, Sa, t, tE, sgn, &x);
                        } else {
                            x = t + (tE - t) * sa0 / (sa0 - Sa);
                            hit = sa0 != Sa && isfinite(x) && sgn * (x - t) > 0;
                        }
                        if (hit) {
                            r1 = x;
                            if (nr == 0) {
                                r0 = x;
                            } else if (sgn * (r1 - r0) < 0) {
                                r1 = r0;
                                r0 = x;
                            }
                            ++nr;
                        }
                        if (nr > 0) {
                            st = ROOT;
                            known = false;
                        } else if (have) {
                            cl = prim;
                            sw0 = Sw;
                            sa0 = Sa;
                        } else {
                            ev = false;
                        }
                    } else if (st == ROOT) {
                        r0 = r1;
                        --nr;
                        st = nr > 0 ? ROOT : have ? END : TAIL;
                    } else if (st == END) {
                        cl = prim;
                        sw0 = swE;
                        sa0 = saE;
                        st = PIECE;
                    } else {
                        ev = false;
                    }
                    if (known) {
                        real sl = te != t ? (v - f) / (te - t) : real(0);
                        if (first) A.sl[q] = sl;
                        first = false;
                        emit = pend;
                        xt = t;
                        xlo = psl;
                        xhi = sl;
                        xcl = pcl;
                        t = te;
                        f = v;
                        psl = sl;
                        pcl = cl;
                        pend = ev && sgn * te <= Wk;
                        if (!pend) st = DONE;
                        else if (sgn * te == Wk) st = FLUSH;
                    }
                }
                unsigned em = __ballot_sync(0xffffffffu, emit);
                if (em == 0) continue;
                if (emit) {
                    int p = cnt + __popc(em & below);
                    if (p < maxe) {
                        A.key[p] = sgn * xt;
                        A.pair[p] = SepPair<real>{xlo, xhi};
                        A.slot[p] = (typename SepList<real>::slot_t)(((unsigned)q << 16) | p | (xcl ? 0x8000 : 0));
                    }
                }
                cnt += __popc(em & mine);
                if (flush) ++last;
            }
        }
        for (int o = nl; o < 32; o <<= 1) last += __shfl_xor_sync(0xffffffffu, last, o);
        *before = cnt - last;
        return cnt;
    }

    // The entries of a list in order, the pairs of a batch's list with them.
    __device__ __forceinline__ static real signed_key(real k, unsigned p) { return (p & 0x8000u) ? -k : k; }
    __device__ __forceinline__ static double slope_change(const SepPair<real> &p) {
        return sep_widen(p.y) - sep_widen(p.x);
    }
    // The first n <= 32 E entries of a list in order, by the warp, E consecutive entries a lane in
    // registers: a bitonic network whose comparisons all point upward (each merge starts with mirrored
    // pairs); strides below E stay in the lane.
    // (FP32 entries of one time keep the order that the network gives them: SEP_REDO.)
    __device__ __forceinline__ static bool after(real ka, unsigned pa, real kb, unsigned pb) {
        if constexpr (sizeof(real) == 8) return ka > kb || (ka == kb && pa > pb);
        return ka > kb;
    }
    template <int E>
    __device__ __forceinline__ void sort_regs(const SepList<real> &A, int n) const {
        real k[E];
        unsigned p[E];
#pragma unroll
        for (int r = 0; r < E; ++r) {
            int i = lane * E + r;
            k[r] = i < n ? A.key[i] : real(INFINITY);
            p[r] = i < n ? A.slot[i] : 0xffffffffu;
        }
#pragma unroll
        for (int lk = 1; (1 << lk) <= 32 * E; ++lk) {
#pragma unroll
            for (int lj = lk - 1; lj >= 0; --lj) {
                const int kk = 1 << lk, j = 1 << lj;
                const bool mirror = lj == lk - 1;
                if (j < E) {
#pragma unroll
                    for (int r = 0; r < E; ++r) {
                        const int o = mirror ? r ^ ((kk - 1) & (E - 1)) : r ^ j;
                        if (o > r) {
                            bool sw = after(k[r], p[r], k[o], p[o]);
                            real a = sw ? k[o] : k[r], b = sw ? k[r] : k[o];
                            unsigned pa = sw ? p[o] : p[r], pb = sw ? p[r] : p[o];
                            k[r] = a;
                            k[o] = b;
                            p[r] = pa;
                            p[o] = pb;
                        }
                    }
                } else {
                    const int x = mirror ? (kk - 1) / E : j / E;
                    bool low = (lane & (j / E)) == 0;
                    real ok[E];
                    unsigned op[E];
#pragma unroll
                    for (int r = 0; r < E; ++r) {
                        ok[r] = __shfl_xor_sync(0xffffffffu, k[mirror ? E - 1 - r : r], x);
                        op[r] = __shfl_xor_sync(0xffffffffu, p[mirror ? E - 1 - r : r], x);
                    }
#pragma unroll
                    for (int r = 0; r < E; ++r) {
                        if constexpr (sizeof(real) == 8) {
                            bool sw = low ? after(k[r], p[r], ok[r], op[r]) : after(ok[r], op[r], k[r], p[r]);
                            k[r] = sw ? ok[r] : k[r];
                            p[r] = sw ? op[r] : p[r];
                        } else {
                            real nk = low ? fmin(k[r], ok[r]) : fmax(k[r], ok[r]);
                            p[r] = nk == k[r] ? p[r] : op[r];  // (equal keys: each lane keeps its own)
                            k[r] = nk;
                        }
                    }
                }
            }
        }
        double ds[E];
        if (!full)
#pragma unroll
            for (int r = 0; r < E; ++r)
                if (lane * E + r < n) ds[r] = slope_change(A.pair[p[r] & 0x7fffu]);
        __syncwarp();
#pragma unroll
        for (int r = 0; r < E; ++r) {
            int i = lane * E + r;
            if (i < n) {
                A.key[i] = full ? k[r] : signed_key(k[r], p[r]);
                A.slot[i] = (typename SepList<real>::slot_t)p[r];
                if (!full) sep_put<real>(A.pair[i], ds[r]);
            }
        }
        __syncwarp();
    }
    // the same in shared memory, for lists of any length; tmp: n doubles
    __device__ __noinline__ void sort_mem(const SepList<real> &A, int n, double *tmp) const {
        int n2 = 32;
        while (n2 < n) n2 <<= 1;
        for (int k = 2; k <= n2; k <<= 1) {
            for (int j = k >> 1; j > 0; j >>= 1) {
                bool mirror = j == (k >> 1);
                for (int i = lane; i < (n2 >> 1); i += 32) {
                    int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1));
                    int hi = mirror ? lo ^ (k - 1) : lo + j;
                    if (hi < n) {
                        real ka = A.key[lo], kb = A.key[hi];
                        auto pa = A.slot[lo], pb = A.slot[hi];
                        if (after(ka, pa, kb, pb)) {
                            A.key[lo] = kb;
                            A.key[hi] = ka;
                            A.slot[lo] = pb;
                            A.slot[hi] = pa;
                        }
                    }
                }
                __syncwarp();
            }
        }
        if (full) return;
        for (int i = lane; i < n; i += 32) {
            unsigned p = A.slot[i];
            tmp[i] = slope_change(A.pair[p & 0x7fffu]);
            A.key[i] = signed_key(A.key[i], p);
        }
        __syncwarp();
        for (int i = lane; i < n; i += 32) sep_put<real>(A.pair[i], tmp[i]);
        __syncwarp();
    }
    __device__ __forceinline__ void sort(const SepList<real> &A, int n, double *tmp) const {
        if (n <= 32)
            sort_regs<1>(A, n);
        else if (n <= 64)
            sort_regs<2>(A, n);
        else if (n <= 128)
            sort_regs<4>(A, n);
        else if (n <= sep_regs<real>())
            sort_regs<sep_regs<real>() / 32>(A, n);
        else
            sort_mem(A, n, tmp);
    }
    // a short list, by one lane
    __device__ __forceinline__ void sort_short(const SepList<real> &A, int n) const {
        for (int i = 0; i < n; ++i) {
            real k = A.key[i];
            unsigned p = A.slot[i];
            SepPair<real> v = A.pair[i];
            if (!full) {
                double ds = slope_change(v);
                sep_put<real>(v, ds);
                if (p & 0x8000u) k = -k;
            }
            int j = i - 1;
            for (; j >= 0 && after(fabs(A.key[j]), A.slot[j], fabs(k), p); --j) {
                A.key[j + 1] = A.key[j];
                A.slot[j + 1] = A.slot[j];
                if (!full) A.pair[j + 1] = A.pair[j];
            }
            A.key[j + 1] = k;
            A.slot[j + 1] = (typename SepList<real>::slot_t)p;
            if (!full) A.pair[j + 1] = v;
        }
    }

    // One direction of walk! over list l of a batch, whose window ends at a clamp: the potential at
    // every event and the stop test at the clamps. Sets the list's state: SEP_OPEN when the window
    // does not end it.
    __device__ __forceinline__ void scan(int l, real sgn) const {
        SepList<real> A = list(l);
        int n = B.n[l];
        if (n > maxe) {  // more events before the window end than points; else many at the end itself
            B.st[l] = B.before[l] >= M.maxpts ? SEP_GUARD : SEP_ALONE;
            return;
        }
        if (n <= ESM_SEP_SHORT) sort_short(A, n);
        double b = 0, c = 0;
        float abf = 0;
        for (int q = 0; q < nu; ++q) {
            real x = A.sl[q];
            b += sep_widen(x);
            abf += fabsf((float)x);
        }
        const double maxnats = (double)M.maxnats;
        const int last = n < M.maxpts ? n : M.maxpts;
        int i = 0, st = SEP_OPEN, low = 0;  // the high word of the least potential so far (ordered as an integer)
        // Two FP64 instructions an event, 64 cycles each, up to the next clamp: the potentials are kept in
        // double (masses() rounds them), the minimum by its high word, and the stop test stands outside the
        // loop (395 cycles an event with the rounding and the exact minimum in it, 635 with the test too).
        real kn = A.key[0];
        double dn = sep_get<real>(A.pair[0]);
        real kc = 0;
        while (i < last) {
            bool clamp = false;
#pragma unroll 2
            do {
                const real ka = fabs(kn);
                const double wn = sep_widen(sgn * (ka - kc));
                clamp = kn < 0;
                kc = ka;
                c = sep_fma<real>(b, wn, c);
                b += dn;
                abf += sep_above(dn);
                if (i + 1 < last) {
                    kn = A.key[i + 1];
                    dn = sep_get<real>(A.pair[i + 1]);
                }
                sep_put<real>(A.pair[i], c);
                const int h = __double2hiint(c);
                low = min(low, h ^ ((h >> 31) & 0x7fffffff));
                ++i;
            } while (!clamp && i < last);
            if (clamp) {
                // the least potential lies between this word and the next: where that does not decide, it
                // is taken from the potentials
                const double m0 = sep_word(low), m1 = sep_word(low + 1);
                bool stop = c - m1 > maxnats;
                if (!stop && c - m0 > maxnats) {
                    double cmin = 0;
                    for (int j = 0; j < i; ++j) cmin = fmin(cmin, sep_get<real>(A.pair[j]));
                    stop = c - cmin > maxnats;
                }
                if (stop) {
                    st = SEP_PROPER;
                    break;
                }
            }
        }
        if (st == SEP_OPEN && i < n) st = SEP_GUARD;  // more points than the cap
        // the cap cuts the group of events that the walk ends in
        if (sizeof(real) == 4 && n > M.maxpts && st != SEP_OPEN && kc == fabs(A.key[M.maxpts])) st = SEP_REDO;
        B.np[l] = i;
        B.ab[l] = abf;
        B.st[l] = st;
    }

    // The same for any window, with the ray steps after the last clamp and the round-off scale of every
    // point. SEP_ALONE when the list has not the room.
    __device__ __forceinline__ void scan_full(int l, real sgn) const {
        const real INF = real(INFINITY);
        SepList<real> A = list(l);
        int n = B.n[l], ncl = B.ncl[l];
        bool inf = !(B.W[l] < INF);
        if (n > maxe) {
            B.st[l] = B.before[l] >= M.maxpts || alone ? SEP_GUARD : SEP_ALONE;
            return;
        }
        if (n <= ESM_SEP_SHORT) sort_short(A, n);
        double b = 0, ab = 0, c = 0, cmin = 0;
        for (int q = 0; q < nu; ++q) {
            double x = sep_widen(A.sl[q]);
            b += x;
            ab += fabs(x);
        }
        const double maxnats = (double)M.maxnats;
        const int maxpts = M.maxpts;
        real tcur = 0;
        int i = 0, np = 0, ray = 0x7fffffff, st = SEP_OPEN;
        auto advance = [&](real t) {
            c = sep_fma<real>(b, sep_widen((real)(t - tcur)), c);
            tcur = t;
        };
        auto pass = [&](const SepPair<real> &v) {  // an event's slopes
            b += slope_change(v);
            ab = fmax(ab, ab + fabs(sep_widen(v.y)) - fabs(sep_widen(v.x)));
        };
        auto point = [&](real t) -> bool {
            int e = np < ray ? np : n + np - ray;
            if (np >= maxpts || e >= maxent) {
                st = np >= maxpts || alone ? SEP_GUARD : SEP_ALONE;
                return false;
            }
            if (e >= n) {
                A.key[e] = sgn * t;
                A.slot[e] = (typename SepList<real>::slot_t)e;
            }
            SepPair<real> v;
            v.x = sep_narrow(c, real(0));
            v.y = 0;
            if constexpr (sizeof(real) == 4)
                v.y = real(4.8e-7) * sep_narrow(sep_fma<real>(ab, fabs(sep_widen(t)), fabs(c)), real(0));
            A.pair[A.slot[e] & 0x7fffu] = v;
            cmin = fmin(cmin, c);
            ++np;
            return true;
        };
        while (st == SEP_OPEN && ncl > 0 && i < n) {
            unsigned p = A.slot[i];
            SepPair<real> v = A.pair[p & 0x7fffu];
            advance(sgn * A.key[i]);
            if (!point(tcur)) break;
            pass(v);
            if (p & 0x8000u) {
                --ncl;
                if (c - cmin > maxnats) st = SEP_PROPER;
            }
            ++i;
        }
        if (st == SEP_OPEN && inf) {  // (no event left before the clamps the count expects: as behind them)
            ray = np;
            real delta = 0;
            int nx = 0;
            while (st == SEP_OPEN) {
                double sl = (double)sgn * b;
                if (sl > 0)
                    delta = fmin(real(2) * M.maxnats / (real)sl, real(1e3) * fmax(fabs(tcur), real(1e-3)));
                else
                    delta = delta == 0 ? fmax(fabs(tcur), real(1e-6)) : real(2) * delta;
                real target = tcur + sgn * delta;
                if (++nx > 80) {
                    st = SEP_IMPROPER;
                    break;
                }
                bool ok = true;
                while (ok && i < n) {  // the events before the target
                    real t = sgn * A.key[i];
                    if (!(sgn * (target - t) > 0)) break;
                    SepPair<real> v = A.pair[A.slot[i] & 0x7fffu];
                    advance(t);
                    ok = point(t);
                    if (ok) pass(v);
                    ++i;
                }
                if (ok) {
                    advance(target);
                    ok = point(target);
                }
                if (!ok) break;
                while (i < n && sgn * A.key[i] == target) pass(A.pair[A.slot[i++] & 0x7fffu]);
                if (c - cmin > maxnats) st = SEP_PROPER;
            }
        }
        // (as in scan; no event ends a walk in the ray phase)
        if (sizeof(real) == 4 && n > maxpts && ray == 0x7fffffff && (st == SEP_PROPER || st == SEP_GUARD))
            if (A.key[np - 1] == A.key[maxpts]) st = SEP_REDO;
        B.np[l] = np;
        B.ray[l] = ray;
        B.st[l] = st;
    }

    // The points of a list, and the segments: segment k ends at point k and starts at point k - 1 (at
    // 0 for k = 0).
    struct Points {
        SepList<real> A;
        int ray, n;
        bool full;
        __device__ __forceinline__ int entry(int k) const { return k < ray ? k : n + k - ray; }
        __device__ __forceinline__ real key(int k) const { return k < 0 ? real(0) : fabs(A.key[entry(k)]); }
        __device__ __forceinline__ int at(int k) const { return full ? A.slot[entry(k)] & 0x7fff : k; }
        __device__ __forceinline__ real c(int k) const { return k < 0 ? real(0) : A.pair[at(k)].x; }
        __device__ __forceinline__ real z(int k) const { return k < 0 ? real(0) : A.pair[at(k)].y; }
        __device__ __forceinline__ real &m(int k) const { return full ? A.m[entry(k)] : A.pair[k].y; }
    };
    __device__ __forceinline__ Points points(int l) const {
        return Points{list(l), full ? B.ray[l] : 0x7fffffff, B.n[l], full};
    }

    // the masses of the segments of tasks k0 .. k0 + nt - 1 relative to each task's largest (sample_line!,
    // src/local.jl:1501), by the warp: G lanes a list, two lists a task
    template <int G>
    __device__ __forceinline__ void masses(int k0, int nt) const {
        const int side = (lane / G) & 1, j0 = lane & (G - 1);
        for (int k = k0 + lane / (2 * G); k - lane / (2 * G) < k0 + nt; k += 16 / G) {
            bool on = k < k0 + nt && B.st[2 * k] == SEP_PROPER && B.st[2 * k + 1] == SEP_PROPER;
            const int l = on ? 2 * k + side : 0;
            Points pt = points(l);
            int np = on ? B.np[l] : 0;
            real mx = -INFINITY;
            if (!full) {  // the potentials of the scan, rounded
                for (int j = j0; j < np; j += G) pt.A.pair[j].x = sep_narrow(sep_get<real>(pt.A.pair[j]), real(0));
                __syncwarp();
            }
            for (int j = j0; j < np; j += G) {
                real L = pt.key(j) - pt.key(j - 1), c0 = pt.c(j - 1), c1 = pt.c(j);
                real lm = L > 0 ? -fmin(c0, c1) + Lane<real>::logseg(L, fabs(c1 - c0)) : real(-INFINITY);
                pt.m(j) = lm;
                mx = fmax(mx, lm);
            }
#pragma unroll
            for (int o = G; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            for (int j = j0; j < np; j += G) {
                real &x = pt.m(j);
                x = exp(x - mx);
            }
        }
    }

    // the draw over the segments of task k; the sums in segment order: the left walk's from its last
    // point inward, then the right walk's. *st: SEP_ALONE where the round-off scales decide, which a batch
    // has not, SEP_REDO where the order of events of one time does.
    __device__ __forceinline__ real draw(int k, real ucat, real uoff, int *st) const {
        const Points R = points(2 * k), Lf = points(2 * k + 1);
        const int nr = B.np[2 * k], nl = B.np[2 * k + 1];
        // masses j of a list, in its order: eight loads, then the sums one after the other
        real tot = 0;
        auto total = [&](int n, auto &&at) {
            for (int j0 = 0; j0 < n; j0 += 8) {
                real s[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] = j0 + i < n ? at(j0 + i) : real(0);
#pragma unroll
                for (int i = 0; i < 8; ++i) tot += s[i];
            }
        };
        real u = 0, acc = 0;
        // the first segment whose sum reaches u, -1 if none
        auto find = [&](int n, auto &&at) -> int {
            for (int j0 = 0; j0 < n; j0 += 8) {
                real s[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] = j0 + i < n ? at(j0 + i) : real(0);
#pragma unroll
                for (int i = 0; i < 8; ++i) s[i] = acc = acc + s[i];
                if (!(u <= acc)) continue;
                int x = -1;
#pragma unroll
                for (int i = 7; i >= 0; --i)
                    if (j0 + i < n && u <= s[i]) x = j0 + i;
                if (x >= 0) return x;
            }
            return -1;
        };
        int m0, mr = -1;
        if (full) {
            total(nl, [&](int j) { return Lf.m(nl - 1 - j); });
            total(nr, [&](int j) { return R.m(j); });
            u = ucat * tot;
            m0 = find(nl, [&](int j) { return Lf.m(nl - 1 - j); });
            if (m0 < 0) mr = find(nr, [&](int j) { return R.m(j); });
        } else {
            const SepPair<real> *pl = Lf.A.pair + (nl - 1), *pr = R.A.pair;
            total(nl, [&](int j) { return pl[-j].y; });
            total(nr, [&](int j) { return pr[j].y; });
            u = ucat * tot;
            m0 = find(nl, [&](int j) { return pl[-j].y; });
            if (m0 < 0) mr = find(nr, [&](int j) { return pr[j].y; });
        }
        // the segment starts at merged point m0 (0: the start, -k the left walk's, k the right walk's)
        if (m0 >= 0)
            m0 -= nl;
        else
            m0 = mr >= 0 ? mr : nr - 1;
        auto P = [&](int m) -> real { return m < 0 ? -Lf.key(-m - 1) : R.key(m - 1); };
        auto C = [&](int m) -> real { return m < 0 ? Lf.c(-m - 1) : R.c(m - 1); };
        real p0 = P(m0), p1 = P(m0 + 1), c0 = C(m0), c1 = C(m0 + 1);
        real L = p1 - p0;
        real g = (c1 - c0) / L;
        real flat = Lane<real>::flat_nats;
        if constexpr (sizeof(real) == 4) {
            auto slope = [&](int m) -> real {
                if (m < -nl || m >= nr) return 0;
                real Lm = P(m + 1) - P(m);
                return Lm > 0 ? fabs((C(m + 1) - C(m)) / Lm) : real(0);
            };
            real gl = slope(m0 - 1), gm = slope(m0), gr = slope(m0 + 1);
            if (full) {
                auto Z = [&](int m) -> real { return m < 0 ? Lf.z(-m - 1) : R.z(m - 1); };
                real z0 = Z(m0) + real(2.4e-7) * fabs(p0) * fmax(gl, gm);
                real z1 = Z(m0 + 1) + real(2.4e-7) * fabs(p1) * fmax(gm, gr);
                // Where the segment's inner end is one of a group, its scale depends on the group's order, by no
                // more than the outer end's (whose slopes are those behind the group): below twice the sum of
                // both, the order decides. Below `flat` alone the draw is uniform in any order.
                const real x = fabs(g * L);
                if (x < real(2.001) * (z0 + z1) && x >= real(0.9999) * flat)
                    if (m0 < 0 ? m0 <= -3 && p1 == P(m0 + 2) : m0 >= 2 && p0 == P(m0 - 1)) {
                        *st = SEP_REDO;
                        return 0;
                    }
                flat = fmax(flat, z0 + z1);
            } else {
                // an upper bound of the two scales: where it leaves no doubt they are not needed
                real a0 = B.ab[2 * k + (m0 < 0)], a1 = B.ab[2 * k + (m0 + 1 < 0)];
                real most = real(4.9e-7) * (fabs(c0) + a0 * fabs(p0) + fabs(c1) + a1 * fabs(p1)) +
                            real(2.5e-7) * (fabs(p0) * fmax(gl, gm) + fabs(p1) * fmax(gm, gr));
                if (!(fabs(g * L) > most && fabs(g * L) > flat)) {
                    *st = SEP_ALONE;
                    return 0;
                }
            }
        }
        return sep_pick<real>(p0, p1, g, L, uoff, flat);
    }

    // the commit of unit q of a task at t (apply_step!, src/local.jl:2507): its state of charge and
    // its two node balances
    __device__ __forceinline__ void commit(int q, real t, int tau, int taum, int tau1, int rep) const {
        int j = U.j[q], n = U.n[q];
        real *pe = &M.e[ix(j, tau, rep)];
        SepUnit<real> u{};
        u.load(M, U, q, *pe, clampr<real>(M.e[ix(j, tau1, rep)], 0, 1), clampr<real>(M.e[ix(j, taum, rep)], 0, 1));
        real cw, ca, djw, dja;
        u.move(M, mul_rn(t, u.a), &cw, &ca, &djw, &dja);
        real *pa = &M.r[ix(n, taum, rep)], *pw = &M.r[ix(n, tau, rep)];
        *pa = add_rn(*pa, dja);
        *pw = add_rn(*pw, djw);
        *pe = fma_rn(t, u.a, u.e0);
    }
};

// The units of a separable move by its header (0: not separable); whether a descriptor's header is of such a
// move with at least sepmin units (the moves of sep_run).
__device__ inline int sep_units(const int *h) {
    bool sep = h[0] == 0 && h[2] == 0 && h[3] == 0 && h[4] == 0 && h[6] == 0 && h[8] == 0 && h[5] == h[1] && h[7] == h[1];
    return sep ? h[1] : 0;
}
__device__ inline bool sep_move(const int *hdr, int sepmin) { return sepmin > 0 && hdr[15] >= sepmin; }

// The walks of separable move mi of one model over a block's tasks, in batches of as many as its shared
// memory (region bytes at smem) holds lists for, but no more than `share`; next(n), called by thread 0,
// gives the first task of a batch of n (none from `end` on). A task whose walk passes every clamp, or
// whose draw needs the round-off scales of its points, runs again, alone, with room for both; redo(task)
// takes those left to the one-lane walk. rot: the warp that the scans start at; tmp: the warp's buffer for
// long sorts.
template <class real, class Next, class Redo>
__device__ __forceinline__ void sep_run(const DevModel<real> &M, const Desc<real> &d, SepBlock<real> &B, char *smem,
                                        int region, int share, int rot, char *tmp, const int *steps, int nsteps,
                                        uint32_t sweep, int mi, int end, unsigned int &tried, unsigned int &moved,
                                        unsigned int &guards, Next next, Redo redo) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nu = d.hdr[1], T = M.T;
    SepUnits<real> U(smem, nu);
    for (int q = threadIdx.x; q < nu; q += 32 * ESM_SEP_WARPS) {
        int j = d.si[q];
        U.j[q] = j;
        U.n[q] = M.s_bus[j];
        U.a[q] = d.sa[q];
        U.k[q] = M.kc_s[j];
        U.h[q] = M.s_hours[j];
        U.qt[q] = M.s_qt[j];
        U.ein[q] = M.s_etain[j];
        U.eout[q] = M.s_etaout[j];
        U.mc[q] = M.s_mc[j];
    }
    const int ub = sep_unit_bytes<real>(nu);
    // tasks of a batch: nw warps of nt tasks (a power of two)
    int fit = (region - ub) / (2 * sep_list_bytes<real>(nu, M.maxpts, sep_kind(nu, false)));
    if (fit > share) fit = share;
    const int nw_batch = fit < ESM_SEP_WARPS ? fit : ESM_SEP_WARPS;
    int nt_batch = 1;
    while (nt_batch < 16 && 2 * nt_batch * ESM_SEP_WARPS <= fit) nt_batch <<= 1;
    const int sl = (threadIdx.x + 32 * rot) & (32 * ESM_SEP_WARPS - 1);  // the list of this thread's scan
    if (threadIdx.x == 0) B.nalone = 0;
    while (true) {
        __syncthreads();
        const bool alone = B.nalone > 0;
        __syncthreads();
        if (threadIdx.x == 0) {
            if (alone)
                B.batch = B.alone[--B.nalone];
            else
                B.batch = next(nw_batch * nt_batch);
        }
        __syncthreads();
        const int nw = alone ? 1 : nw_batch, nt = alone ? 1 : nt_batch;
        const int tb = nw * nt;  // tasks of the batch
        const int task0 = B.batch, ntask = alone ? task0 + 1 : end;
        if (task0 >= ntask) break;
        const int kind = sep_kind(nu, alone);
        const bool full = kind != SEP_BATCH;
        SepWalk<real> S{M, U, B, smem + ub, nu, sep_events(nu, M.maxpts, kind), sep_entries(nu, M.maxpts, kind),
                        sep_list_bytes<real>(nu, M.maxpts, kind), full, alone, lane};
        // this lane's list in the event part: list l (task l / 2, direction l % 2)
        const int nl = 2 * nt;
        const int l = wib * nl + (lane & (nl - 1));
        const int q0 = lane / nl, qstep = 32 / nl;
        const real sgn = (l & 1) ? real(-1) : real(1);
        const int task = task0 + (l >> 1);
        const bool mine = wib < nw && (l >> 1) < tb && task < ntask;
        int rep = 0, tau = 0, taum = 0, tau1 = 0;
        if (mine) {
            rep = task % M.R;
            tau = steps[task / M.R];
            taum = (tau - 1 + T) % T;
            tau1 = (tau + 1) % T;
        }
        if (wib < nw) {
            int ncl;
            real W = S.next_clamp(mine ? q0 : nu, qstep, nl, tau, rep, sgn, real(0), &ncl);
            if (lane < nl) {
                B.W[l] = W;
                B.ncl[l] = ncl;
                B.st[l] = !mine ? SEP_IMPROPER : (full || W < real(INFINITY)) ? SEP_OPEN : SEP_ALONE;
            }
        }
        __syncwarp();
        bool open = true;
        while (open) {
            if (wib < nw) {
                bool on = mine && B.st[l] == SEP_OPEN;
                if (__any_sync(0xffffffffu, on)) {
                    int before;
                    int n = S.events(l, on, q0, qstep, nl, tau, taum, tau1, rep, sgn, B.W[l], &before);
                    if (on && lane < nl) {
                        B.n[l] = n;
                        B.before[l] = before;
                    }
                    __syncwarp();
                    unsigned todo = __ballot_sync(0xffffffffu, on && lane < nl && n > ESM_SEP_SHORT && n <= S.maxe);
                    while (todo) {
                        int x = __ffs(todo) - 1;
                        todo &= todo - 1;
                        S.sort(S.list(wib * nl + x), __shfl_sync(0xffffffffu, n, x),
                               (double *)tmp);
                    }
                }
            }
            __syncthreads();
            bool again = false;
            if (sl < 2 * tb && B.st[sl] == SEP_OPEN) {
                real dir = (sl & 1) ? real(-1) : real(1);
                if (full)
                    S.scan_full(sl, dir);
                else
                    S.scan(sl, dir);
                again = B.st[sl] == SEP_OPEN;
            }
            open = __syncthreads_or(again);
            if (open && wib < nw) {  // the open lists' windows end at the next clamp
                bool on = mine && B.st[l] == SEP_OPEN;
                int ncl;
                real W = S.next_clamp(on ? q0 : nu, qstep, nl, tau, rep, sgn, B.W[l], &ncl);
                __syncwarp();
                if (on && lane < nl) {
                    B.W[l] = W;
                    if (!full && !(W < real(INFINITY))) B.st[l] = SEP_ALONE;
                }
                __syncwarp();
            }
        }
        if (wib < nw)
            if (nu <= ESM_SEP_FULL)
                S.template masses<8>(wib * nt, nt);
            else
                S.template masses<16>(wib * nt, nt);
        __syncthreads();
        if (sl < tb) {
            int k = sl, tk = task0 + k;
            real t = 0;
            if (tk < ntask) {
                int r = tk % M.R, qs = tk / M.R, ts = steps[qs];
                int a = B.st[2 * k], b = B.st[2 * k + 1];
                // the right walk's outcome counts first, as in the one-lane walk
                int w = a != SEP_PROPER ? a : b;
                if (w == SEP_PROPER) {
                    double uc, uo;
                    uniform2(M.seed, ESM_TAG_LANE, 2 * (uint32_t)mi, (uint32_t)ts, (uint32_t)r, sweep, &uc, &uo);
                    t = S.draw(k, unit_uniform<real>(uc), unit_uniform<real>(uo), &w);
                }
                if (w == SEP_ALONE) {
                    B.alone[atomicAdd(&B.nalone, 1)] = tk;
                } else if (sizeof(real) == 4 && w == SEP_REDO) {
                    redo(tk);
                } else {
                    ++tried;
                    if (w == SEP_GUARD) ++guards;
                    if (t != 0) ++moved;
                    if (M.mlog && r < M.mlog_nrep) M.mlog[((size_t)mi * nsteps + qs) * M.mlog_nrep + r] = (double)t;
                }
            }
            B.t[k] = t;
        }
        __syncthreads();
        if (wib < nw) {  // lanes: the warp's tasks, then its units
            int k = wib * nt + (lane & (nt - 1)), tk = task0 + k;
            if (k < tb && tk < ntask) {
                real t = B.t[k];
                if (t != 0) {
                    int r = tk % M.R, ts = steps[tk / M.R];
                    for (int q = lane / nt; q < nu; q += 32 / nt) S.commit(q, t, ts, (ts - 1 + T) % T, (ts + 1) % T, r);
                }
            }
        }
    }
}

}  // namespace esm
