// Storage multiscale sweep on the device: the plateau moves of storage_ms_sweep!
// (src/flowmoves.jl:255, prep_storage_ms! :187 without a shape). A move raises the state of charge
// of its units (one storage unit, or the units of one carrier in one country cell) by t at the
// instants b0+1 .. b0+L of a dyadic block, i.e. moves energy from step b0 to step b0+L; the power
// changes only at those two end steps, where the dispatch at the units' nodes follows pro rata
// (prorata!, src/local.jl:1782, with the requirement adjustment soc_qadj, :1826), with the Jacobian
// of logjac (:1871). Every step of the block has the units' storage terms and node balances.
//
// Mapping. The blocks of one length and parity are independent (they share no step); a class pass
// is one launch in which tasks (block, replica), replica fastest (neighbouring state access), run
// the class's 8 moves in order. The move selections are state-independent and drawn on the host
// from the class stream, as the local sweep's move list is. Blocks below 32 steps take one thread
// a task where there are thousands of tasks, whose walks go through one state machine so that the threads of a
// warp evaluate together. Longer blocks, and few tasks, take one warp a task and the long-range moves one block of 8
// warps, with the move's states, units and ends in shared memory: the threads take one (unit, end),
// one interior step or one segment each, the sums are formed in a fixed order, and what the walk
// decides every thread decides alike. Bound by the latency and the instructions of the evaluations'
// chains, not by memory. 40 nodes, T=2920, 64 replicas, one pass: 27.7 -> 12.0 ms for blocks of 2 steps
// and 14.9 -> 6.4 ms for 16 (threads that part at every root and come together late -> one evaluation
// site that they reach together), 8.2 -> 3.6 ms for 64 (every lane of a warp doing all of the ends ->
// shared).
//
// Interior steps. At an interior step both state-of-charge values of a unit's storage term move by
// t, so while every moved value stays strictly inside (0, 1) the term's cost, injection and
// secondaries are exactly unchanged (clamp_diff keeps the change, d does not move). A unit's
// interior steps are therefore evaluated only outside that interval, whose ends are also the first
// primary breakpoints (the state-of-charge clamps) of the unit; the walk visits the same points
// as walk! over the whole block.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "esm_common.cuh"
#include "esm_linemove.cuh"

namespace esm {

#define ESM_PLAT_RB 256   // roots between two walk points (beyond: the move is left, a guard event)
#define ESM_PLAT_NACT 8   // listed steps per unit whose state lies outside the box (more: the unit is evaluated whole)
#define ESM_PLAT_LOCAL 4096  // reals of a thread's local array, if a task has one thread (larger layouts: the global slab)
#define ESM_PLAT_PTS 48   // walk points per direction a warp's shared memory holds (beyond: the global slab)
#define ESM_PLAT_ROOTS 32 // roots of either kind it holds (beyond: the global slab)
#define ESM_PLAT_SHORT 32 // blocks below this length: at most a warp's interior steps, summed in order
#define ESM_PLAT_LONG 256 // threads of a long-range task
#define ESM_PLAT_STAGE (110 << 10)  // its shared memory with the year's states and terms in it (two blocks an SM)

// a task's layout (reals): a thread's array or a warp's shared memory, and the warp's global slab for what
// that does not hold
struct PlatLayout {
    int K;                               // kinked units per node
    int npt, nrt;                        // walk points per direction, roots of a kind
    int pt;                              // [6 * npt] walk points: position, cost, round-off bound, to the right and left
    int ro;                              // [2 * nrt] node-balance and storage roots; then the segment masses
    int cnt;                             // two root counters (integers)
    int slo, shi;                        // [U] clamp-free interval of the moved states inside the box
    int na, act;                         // [U] count, [U * NACT] interior steps touching a state outside the box
    int par;                             // [U * 7] capacity, hours, inflow, efficiencies, marginal cost, node
    int Di, Ai;                          // [U] interior sums
    int kv, kq, kg, kp, ke, knm, kph;    // [2U] compensation kink per (unit, end)
    int ka;                              // [2U * K * 5] per (unit, end, disp unit): kinked coefficient, state, unit data
    int dr, r0;                          // [2U] node-balance change and value per (unit, end)
    int s3, p3;                          // [2U * 3] end storage secondaries, current / previous
    int sb, pb;                          // [2U] end node balances, current / previous
    int w;                               // [2U * (K + 2)] an evaluation's terms, in the order of their sum
    int ys, ny;                          // [U * ny] the states at the block's positions (ny 0: not staged)
    int tc, nt;                          // [6 * nt] a long-range move's terms: cost and size in the sum, injection
                                         // and d of the two last points kept (nt 0: in the global slab)
    int red;                             // [ESM_PLAT_LONG / 32] a long-range task's reductions
    int total;
    int gp, gr, gl, gc, gtotal;          // global slab: points, roots, masses, terms
};

// U units, K kinked units per node, ny staged positions; wide: of a warp or block; nt, ng: terms of a
// long-range move kept in shared memory, in the global slab
__host__ __device__ inline PlatLayout plat_layout(int maxpts, int U, int K, int ny, bool wide, int nt = 0, int ng = 0) {
    PlatLayout L;
    int o = 0;
    L.K = K;
    L.npt = wide && maxpts > ESM_PLAT_PTS ? ESM_PLAT_PTS : maxpts;
    L.nrt = wide ? ESM_PLAT_ROOTS : ESM_PLAT_RB > maxpts + 1 ? ESM_PLAT_RB : maxpts + 1;
    L.ny = ny;
    L.w = o; o += 2 * U * (K + 2);  // (first: also read as doubles)
    L.pt = o; o += 6 * L.npt;
    L.ro = o; o += 2 * L.nrt;
    L.cnt = o; o += 2;
    L.slo = o; o += U;
    L.shi = o; o += U;
    L.na = o; o += U;
    L.act = o; o += U * ESM_PLAT_NACT;
    L.par = o; o += 7 * U;
    L.Di = o; o += U;
    L.Ai = o; o += U;
    L.kv = o; o += 2 * U;
    L.kq = o; o += 2 * U;
    L.kg = o; o += 2 * U;
    L.kp = o; o += 2 * U;
    L.ke = o; o += 2 * U;
    L.knm = o; o += 2 * U;
    L.kph = o; o += 2 * U;
    L.ka = o; o += 2 * U * K * 5;
    L.dr = o; o += 2 * U;
    L.r0 = o; o += 2 * U;
    L.s3 = o; o += 6 * U;
    L.p3 = o; o += 6 * U;
    L.sb = o; o += 2 * U;
    L.pb = o; o += 2 * U;
    L.ys = o; o += U * ny;
    L.nt = nt;
    L.tc = o; o += 6 * nt;
    L.red = o; o += ESM_PLAT_LONG / 32;
    L.total = (o + 3) & ~3;
    L.gp = 0;
    L.gr = 6 * maxpts;
    L.gl = L.gr + 2 * ESM_PLAT_RB;
    L.gc = L.gl + 2 * maxpts + 1;
    L.gtotal = (L.gc + 6 * ng + 3) & ~3;
    return L;
}

// One move at a time of a task of G lanes (a thread, a warp, or the ESM_PLAT_LONG threads of a block). The (unit, end) pair i = 2 u + s belongs to lane
// i % G, which alone writes and reads its entries; what the walk needs of them goes through sums,
// minima and the root buffers that every lane of the task receives.
template <class real, int G>
struct PLane {
    const DevModel<real> &M;
    const PlatLayout &LL;
    real *sm, *gm;  // the task's layout, the warp's global slab
    int sstride;    // between reals of a thread's layout in global memory (else 1)
    int lane;       // within the task
    bool on = true; // the thread has a task (G 1: the threads of a warp walk together)
    int L, b0, rep, U;
    bool lvl = false;  // the level move of the long-range sweep: every instant of the year rises, no end steps
    bool dup = false;  // two units at one node
    bool inorder = false;  // a short block's: interior sums in step order, whatever G
    const int *uj;  // the move's storage units
    mutable real nzs = 0;
    mutable int buf = 0;  // the kept terms that the next evaluation writes (the other: those at the last point saved)

    __device__ PLane(const DevModel<real> &M_, const PlatLayout &LL_, real *sm_, int sstride_, real *gm_)
        : M(M_), LL(LL_), sm(sm_), gm(gm_), sstride(sstride_), lane(G == 1 ? 0 : threadIdx.x) {}
    __device__ inline void sync() const {
        if constexpr (G == 32) __syncwarp();
        if constexpr (G > 32) __syncthreads();
    }
    // within a warp
    __device__ inline real wsum(real v) const {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        return __shfl_sync(0xffffffffu, v, 0);
    }
    __device__ inline real wmin(real v) const {
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    }
    __device__ inline real wmax(real v) const { return -wmin(-v); }
    // over the task, on every lane
    __device__ inline real tmin(real v) const {
        if constexpr (G > 1) v = wmin(v);
        if constexpr (G > 32) {
            sync();
            if (lane % 32 == 0) S(LL.red, lane / 32) = v;
            sync();
            for (int w = 0; w < G / 32; ++w) v = fmin(v, S(LL.red, w));
        }
        return v;
    }
    __device__ inline real tmax(real v) const { return -tmin(-v); }

    __device__ inline real &S(int off, int i) const {
        return G > 1 ? sm[off + i] : sm[(size_t)(off + i) * sstride];
    }
    // walk point i of array a (0 position, 1 cost, 2 round-off bound to the right; 3, 4, 5 to the left)
    __device__ inline real &pt(int a, int i) const {
        return G == 1 || i < LL.npt ? S(LL.pt, a * LL.npt + i) : gm[LL.gp + a * M.maxpts + i];
    }
    // root i of kind h (0 node balances, 1 storage); mass j
    __device__ inline real &rt(int h, int i) const {
        return G == 1 || i < LL.nrt ? S(LL.ro, h * LL.nrt + i) : gm[LL.gr + h * ESM_PLAT_RB + i];
    }
    __device__ inline real &lm(int j) const { return G == 1 || j < 2 * LL.nrt ? S(LL.ro, j) : gm[LL.gl + j]; }
    // kept term array a (0 cost, 1 size; 2, 3 injection and 4, 5 d of either buffer), term i
    __device__ inline real &tc(int a, int i) const { return LL.nt ? sm[LL.tc + a * LL.nt + i] : gm[LL.gc + a * M.T + i]; }
    __device__ inline int &cnt(int h) const { return reinterpret_cast<int *>(sm + LL.cnt)[h]; }
    __device__ inline size_t ix(int x, int t) const { return sidx(x, t, rep, M.T, M.R); }
    // unit data: 0 capacity, 1 hours, 2 inflow, 3 and 4 efficiencies, 5 marginal cost (a thread's task reads
    // the model, at the same address as its warp's others)
    __device__ inline real par(int u, int k) const {
        if constexpr (G > 1) return S(LL.par, 7 * u + k);
        const int j = uj[u];
        const real *const f[6] = {M.kc_s, M.s_hours, M.s_qt, M.s_etain, M.s_etaout, M.s_mc};
        return f[k][j];
    }
    __device__ inline int node(int u) const { return G > 1 ? (int)S(LL.par, 7 * u + 6) : M.s_bus[uj[u]]; }
    // block positions: step b0 + q, cyclic (the long-range plateaus wrap); the interior terms (both
    // states raised) are q0() .. q0() + nq() - 1, the raised states q0() .. q0() + ns() - 1
    __device__ inline int cyc(int x) const { return x >= M.T ? x - M.T : x; }
    __device__ inline int stp(int q) const { return cyc(b0 + q); }
    __device__ inline int q0() const { return lvl ? 0 : 1; }
    __device__ inline int nq() const { return lvl ? M.T : L - 1; }
    __device__ inline int ns() const { return lvl ? M.T : L; }
    __device__ inline int tau_end(int s) const { return s == 0 ? stp(0) : stp(L); }
    // the state of unit u at position q, and at the one after it
    __device__ inline real Y(int u, int q) const { return G > 1 && LL.ny ? S(LL.ys, u * LL.ny + q) : M.e[ix(uj[u], stp(q))]; }
    __device__ inline real Y1(int u, int q) const {
        return G > 1 && LL.ny ? S(LL.ys, u * LL.ny + (lvl && q + 1 == M.T ? 0 : q + 1)) : M.e[ix(uj[u], cyc(stp(q) + 1))];
    }
    // an interior term whose two states stay strictly inside (0, 1) at t is exactly unchanged
    __device__ inline bool quiet(int u, int q, real t) const {
        real y0 = Y(u, q), y1 = Y1(u, q);
        return y0 > 0 && y0 < 1 && y1 > 0 && y1 < 1 && y0 + t > 0 && y0 + t < 1 && y1 + t > 0 && y1 + t < 1;
    }
    __device__ inline bool inside(int u, real t) const { return t > S(LL.slo, u) && t < S(LL.shi, u); }

    // the move's units and their states into shared memory
    __device__ __noinline__ void load() {
        sync();
        if constexpr (G == 1) {
            dup = true;  // (one lane: always in order)
            return;
        }
        for (int u = lane; u < U; u += G) {
            const int j = uj[u];
            const real q[7] = {M.kc_s[j], M.s_hours[j], M.s_qt[j], M.s_etain[j], M.s_etaout[j], M.s_mc[j], real(M.s_bus[j])};
            for (int k = 0; k < 7; ++k) S(LL.par, 7 * u + k) = q[k];
        }
        if (LL.ny) {
            const int np = lvl ? M.T : L + 2;
            for (int u = 0; u < U; ++u)
                for (int q = lane; q < np; q += G) S(LL.ys, u * LL.ny + q) = M.e[ix(uj[u], cyc(stp(q)))];
        }
        sync();
        bool d = false;
        for (int u = lane; u < U; u += G)
            for (int v = 0; v < u; ++v) d = d || node(v) == node(u);
        dup = __any_sync(0xffffffffu, d);
    }

    // storage term of unit u at block step q (0..L): the change of its cost; *dj the injection
    // change, *d1 the new d (src/energy.jl:448 soc_cost in difference form)
    __device__ __noinline__ real sterm(int u, int q, real t, real *dj, real *d1) const {
        real k = par(u, 0);
        return soc_diff<real>(par(u, 1), par(u, 2), par(u, 3), par(u, 4), par(u, 5), k, k + M.kappa0, M.dt, M.c_viol, Y(u, q), Y1(u, q),
                              (lvl || q >= 1) ? t : real(0), (lvl || q + 1 <= L) ? t : real(0), dj, d1);
    }
    __device__ inline void sec3(int u, real d, real out[3]) const {
        real ein = par(u, 3);
        out[0] = d;
        out[1] = ein > 0 ? d - ein : real(1);
        out[2] = -d * par(u, 4) - real(1);
    }

    // the compensation at the end steps (prorata! with soc_qadj), per (unit, end)
    __device__ __noinline__ void kinks() const {
        for (int i = lane; i < 2 * U; i += G) {
            const int u = i >> 1, s = i & 1;
            int tau = tau_end(s);
            int n = node(u);
            real ks = par(u, 0) * par(u, 1) / M.dt;
            real g = s == 0 ? ks : -ks;
            real Pm = 0, Qs = 0;
            int nv = 0, c = 0;
            for (int p = M.up[n]; p < M.up[n + 1] && c < LL.K; ++p, ++c) {
                int d = M.ua[p];
                real kap = M.d_avail[d] * M.kc_d[d];
                if (!(fabs(kap) >= M.kmin)) continue;
                real om = M.g[ix(d, tau)];
                Pm += kap * om;
                Qs += kap * clampr<real>(om, 0, 1);
                nv += 1;
            }
            bool valid = g != 0 && nv > 0 && !(fabs(Pm) < real(1e-6));
            // soc_qadj: nominal minus actual injection of the unit at its node
            real ye = Y(u, s == 0 ? 0 : L), ye1 = Y1(u, s == 0 ? 0 : L);
            real ec = clampr<real>(ye, 0, 1), ec1 = clampr<real>(ye1, 0, 1);
            real dd = par(u, 1) * (ec1 - ec) / M.dt - par(u, 2);
            real pc = 0, mcx = 0;
            if (dd >= 0)
                pc = par(u, 3) > 0 ? dd / par(u, 3) : real(0);
            else
                mcx = fmin(-dd * par(u, 4), real(1));
            real qadj = par(u, 0) * par(u, 1) * (ye1 - ye) / M.dt - par(u, 0) * (pc - mcx);
            real r0 = M.r[ix(n, tau)];
            real Q = r0 + Qs + qadj;
            S(LL.r0, i) = r0;
            S(LL.kv, i) = valid ? real(1) : real(0);
            S(LL.kq, i) = Q;
            S(LL.kg, i) = g;
            S(LL.kp, i) = valid ? Pm : real(1);
            S(LL.ke, i) = Pm - fmax(Q, real(0));
            S(LL.knm, i) = real(nv - 1);
            c = 0;
            for (int p = M.up[n]; c < LL.K; ++p, ++c) {
                const int ka = 5 * (i * LL.K + c);
                real ak = 0;
                if (p < M.up[n + 1]) {
                    int d = M.ua[p];
                    real kap = M.d_avail[d] * M.kc_d[d];
                    if (valid && fabs(kap) >= M.kmin) {
                        real sigma = kap * M.g[ix(d, tau)] / Pm;
                        if (sigma != 0) ak = sigma / kap;
                    }
                    S(LL.ka, ka + 1) = M.g[ix(d, tau)];
                    S(LL.ka, ka + 2) = M.kc_d[d];
                    S(LL.ka, ka + 3) = M.d_avail[d];
                    S(LL.ka, ka + 4) = M.d_mc[d];
                }
                S(LL.ka, ka + 0) = ak;
            }
        }
    }

    // Per unit: the interval of t over which every moved state that lies strictly inside (0, 1)
    // stays inside, and the list of interior steps whose storage term involves a moved state outside
    // the box (a state of charge at or beyond a bound moves the term for every t). While t is in the
    // interval, the other interior terms are exactly unchanged. A unit with more than NACT such
    // steps gets an empty interval (evaluated whole).
    __device__ __noinline__ void intervals() const {
        constexpr int W = G > 1 ? 32 : 1;  // (a block's first warp)
        for (int u = 0; u < (lane < W ? U : 0); ++u) {
            real mn = 2, mx = -1;
            int na = 0;
            bool over = false;
            auto list = [&](int qt) {  // an interior term involving a state outside the box
                for (int i = 0; i < na; ++i)
                    if (S(LL.act, u * ESM_PLAT_NACT + i) == real(qt)) return;
                if (na < ESM_PLAT_NACT) {
                    S(LL.act, u * ESM_PLAT_NACT + na++) = real(qt);  // (every lane writes the same value)
                    if constexpr (G > 1) __syncwarp();
                } else {
                    over = true;
                }
            };
            auto out_state = [&](int q) {  // state q is the end value of term q - 1 and the start of term q
                if (lvl) {
                    list(q == 0 ? M.T - 1 : q - 1);
                    list(q);
                } else {
                    if (q - 1 >= 1) list(q - 1);
                    if (q <= L - 1) list(q);
                }
            };
            for (int base = 0; base < ns(); base += W) {
                int p = base + lane, qo = -1;
                if (p < ns()) {
                    int q = q0() + p;
                    real y = Y(u, q);
                    if (y > 0 && y < 1) {
                        mn = fmin(mn, y);
                        mx = fmax(mx, y);
                    } else {
                        qo = q;
                    }
                }
                // the states outside the box, in step order, listed alike on every lane
                if constexpr (G > 1) {
                    unsigned bal = over ? 0u : __ballot_sync(0xffffffffu, qo >= 0);
                    while (bal && !over) {
                        int l = __ffs(bal) - 1;
                        bal &= bal - 1;
                        out_state(__shfl_sync(0xffffffffu, qo, l));
                    }
                } else if (qo >= 0) {
                    out_state(qo);
                }
            }
            if constexpr (G > 1) {
                mn = wmin(mn);
                mx = wmax(mx);
            }
            bool ok = !over && mn <= mx;
            if (lane == 0) {
                if (!over && mn > mx) {  // every raised state outside the box: no interval, terms listed
                    S(LL.slo, u) = real(-INFINITY);
                    S(LL.shi, u) = real(INFINITY);
                } else {
                    S(LL.slo, u) = ok ? -mn : real(0);
                    S(LL.shi, u) = ok ? real(1) - mx : real(0);
                }
                S(LL.na, u) = real(over ? 0 : na);
            }
        }
        sync();
    }

    // the interior step terms of unit u to evaluate at t: every one outside its interval, else the listed
    __device__ inline int nterms(int u, bool in) const { return in ? (int)S(LL.na, u) : nq(); }
    __device__ inline int term_q(int u, bool in, int i) const {
        return in ? (int)S(LL.act, u * ESM_PLAT_NACT + i) : q0() + i;
    }
    // f(u, in, q) for the terms of all units, split over the lanes in the order of unit and step; the
    // number of the terms of unit u and whether they are its listed ones from nt(u, &in)
    template <class N, class F>
    __device__ inline void each_term(N nt, F f) const {
        int u = 0, i = lane;
        while (u < U) {
            bool in;
            const int n = nt(u, &in);
            if (i >= n) {
                i -= n;
                ++u;
                continue;
            }
            f(u, in, term_q(u, in, i));
            i += G;
        }
    }

    // mv_eval! of the block (src/local.jl:1219): beta * DeltaC(t); the end steps' secondaries into
    // s3/sb (the interior ones are evaluated where they change, in collect)
    __device__ __noinline__ real eval(real t) const {
        const real dt = M.dt, cv = M.c_viol, k0 = M.kappa0;
        real D = 0, A = 0;
        // interior steps of a unit: storage term and node balance; the listed terms and those of a short
        // block in order, the terms of a longer one outside the unit's interval by lanes of a warp, each
        // on to its next term that changes. (The warps
        // of a long-range task take every 8th round and keep the terms, which its first warp sums as if
        // it had made them, and from which collect takes the secondaries.)
        auto inner = [&](int u) {
            const bool in = inside(u, t);
            const int nt = nterms(u, in);
            real Di = 0, Ai = 0;
            auto term = [&](int q, real *v, real *a, real *dj, real *d1) {
                real cs = sterm(u, q, t, dj, d1);
                real cb = dt * phibal_diff<real>(M.r[ix(node(u), stp(q))], *dj, M.c_shed, M.c_dump);
                *v = cs + cb;
                *a = fabs(cs) + fabs(cb);
            };
            real v = 0, a = 0, dj, d1;
            if (G > 1 && (in || (G == 32 && inorder))) {  // (no more than a warp's lanes)
                const int q = lane < nt ? term_q(u, in, lane) : 0;
                if (lane < nt && (in || !quiet(u, q, t))) term(q, &v, &a, &dj, &d1);
                if (lane < 32)
                    for (int l = 0; l < nt; ++l) {
                        Di += __shfl_sync(0xffffffffu, v, l);
                        Ai += __shfl_sync(0xffffffffu, a, l);
                    }
            } else if constexpr (G > 32) {
                for (int i = lane; i < nt; i += G) {
                    v = a = 0;
                    if (!quiet(u, q0() + i, t)) {
                        term(q0() + i, &v, &a, &dj, &d1);
                        tc(2 + buf, i) = dj;
                        tc(4 + buf, i) = d1;
                    }
                    tc(0, i) = v;
                    tc(1, i) = a;
                }
                sync();
                if (lane < 32) {
#pragma unroll 8
                    for (int i = lane; i < nt; i += 32) {
                        Di += tc(0, i);
                        Ai += tc(1, i);
                    }
                    Di = wsum(Di);
                    Ai = wsum(Ai);
                }
            } else {
                int i = lane;
                while (true) {
                    while (i < nt && !in && quiet(u, q0() + i, t)) i += G;
                    if (i >= nt) break;
                    term(term_q(u, in, i), &v, &a, &dj, &d1);
                    Di += v;
                    Ai += a;
                    i += G;
                }
                if constexpr (G == 32) {
                    sync();
                    Di = wsum(Di);
                    Ai = wsum(Ai);
                }
            }
            if constexpr (G == 1) {
                D += Di;
                A += Ai;
            } else if (lane == 0) {
                S(LL.Di, u) = Di;
                S(LL.Ai, u) = Ai;
            }
        };
        sync();
        for (int i = lane; i < (lvl ? 0 : 2 * U); i += G) {  // end steps: storage term, kinked dispatch, node balance
            const int u = i >> 1, s = i & 1, q = s == 0 ? 0 : L;
            const int w = i * (LL.K + 2);
            auto add = [&](int h, real v) {  // a term of the sum
                if constexpr (G > 1) {
                    S(LL.w, w + h) = v;
                } else {
                    D += v;
                    A += fabs(v);
                }
            };
            real Q = S(LL.kq, i);
            real ph = S(LL.kv, i) != 0 ? fmax(Q + S(LL.kg, i) * t, real(0)) - fmax(Q, real(0)) : real(0);
            S(LL.kph, i) = ph;
            real dj, d1;
            add(0, sterm(u, q, t, &dj, &d1));
            real sc[3];
            sec3(u, d1, sc);
            for (int h = 0; h < 3; ++h) S(LL.s3, 3 * i + h) = sc[h];
            real dr = dj;
            for (int c = 0; c < LL.K; ++c) {
                const int ka = 5 * (i * LL.K + c);
                real ak = S(LL.ka, ka), cg = 0;
                if (ak != 0) {
                    real k = S(LL.ka, ka + 2), Av = S(LL.ka, ka + 3);
                    real dyc, dex;
                    clamp_diff<real>(S(LL.ka, ka + 1), ak * ph, &dyc, &dex);
                    real dp = Av * k * dyc;
                    cg = dt * S(LL.ka, ka + 4) * dp + cv * dt * (k + k0) * dex;
                    dr -= dp;
                }
                add(1 + c, cg);
            }
            S(LL.dr, i) = dr;
            real r0 = S(LL.r0, i);
            add(1 + LL.K, dt * phibal_diff<real>(r0, dr, M.c_shed, M.c_dump));
            S(LL.sb, i) = r0 + dr;
            if (G == 1 && s == 1) inner(u);
        }
        if constexpr (G > 1) {
            for (int u = 0; u < U; ++u) inner(u);
            sync();
            for (int u = 0; u < U; ++u) {
                const int w = 2 * u * (LL.K + 2);
                for (int h = 0; h < (lvl ? 0 : 2 * (LL.K + 2)); ++h) {
                    D += S(LL.w, w + h);
                    A += fabs(S(LL.w, w + h));
                }
                D += S(LL.Di, u);
                A += S(LL.Ai, u);
            }
        }
        if constexpr (sizeof(real) == 4) nzs = M.beta_v * A * real(4.8e-7);
        return M.beta_v * D;
    }

    __device__ inline void save_prev() const {
        for (int i = lane; i < 2 * U; i += G) {
            for (int h = 0; h < 3; ++h) S(LL.p3, 3 * i + h) = S(LL.s3, 3 * i + h);
            S(LL.pb, i) = S(LL.sb, i);
        }
        buf ^= 1;
    }

    __device__ static inline bool root_of(real a, real b, real lo, real hi, real sgn, real *x) {
        if ((a < 0) != (b < 0) && a != b) {
            real xx = lo + (hi - lo) * a / (a - b);
            if (sgn * (xx - lo) > 0 && sgn * (hi - xx) > 0) {
                *x = xx;
                return true;
            }
        }
        return false;
    }
    __device__ inline void add_root(int h, real x, int *n) const {  // n: a thread's counts
        const int i = G == 1 ? n[h]++ : atomicAdd(&cnt(h), 1);
        if (i < ESM_PLAT_RB) rt(h, i) = x;
    }

    // sign changes of the secondaries between prev (at lo) and cur (at hi): storage ones (want_stor)
    // and node balances into their buffers, in any order (they are sorted); interior steps of the
    // units whose states leave their interval in [lo, hi]
    __device__ __noinline__ void collect(real lo, real hi, real sgn, bool want_stor, int *nro, int *ngro) const {
        int n[2] = {0, 0};
        if constexpr (G > 1) {
            sync();
            if (lane < 2) cnt(lane) = 0;
            sync();
        }
        real x;
        for (int i = lane; i < (lvl ? 0 : 2 * U); i += G) {
            if (want_stor)
                for (int h = 0; h < 3; ++h)
                    if (root_of(S(LL.p3, 3 * i + h), S(LL.s3, 3 * i + h), lo, hi, sgn, &x)) add_root(1, x, n);
            if (root_of(S(LL.pb, i), S(LL.sb, i), lo, hi, sgn, &x)) add_root(0, x, n);
        }
        each_term(
            [&](int u, bool *in) {
                *in = inside(u, lo) && inside(u, hi);
                return nterms(u, *in);
            },
            [&](int u, bool in, int q) {
                if (!in && quiet(u, q, lo) && quiet(u, q, hi)) return;
                real dja, d1a, djb, d1b;
                if (G > 32 && !inside(u, lo) && !quiet(u, q, lo)) {  // (as the evaluation at lo kept it)
                    dja = tc(2 + (buf ^ 1), q - q0());
                    d1a = tc(4 + (buf ^ 1), q - q0());
                } else {
                    sterm(u, q, lo, &dja, &d1a);
                }
                if (G > 32 && !inside(u, hi) && !quiet(u, q, hi)) {
                    djb = tc(2 + buf, q - q0());
                    d1b = tc(4 + buf, q - q0());
                } else {
                    sterm(u, q, hi, &djb, &d1b);
                }
                if (want_stor) {
                    real a3[3], b3[3];
                    sec3(u, d1a, a3);
                    sec3(u, d1b, b3);
                    for (int h = 0; h < 3; ++h)
                        if (root_of(a3[h], b3[h], lo, hi, sgn, &x)) add_root(1, x, n);
                }
                real r0 = M.r[ix(node(u), stp(q))];
                if (root_of(r0 + dja, r0 + djb, lo, hi, sgn, &x)) add_root(0, x, n);
            });
        if constexpr (G > 1) {
            sync();
            n[0] = cnt(0);
            n[1] = cnt(1);
        }
        *nro = n[0];
        *ngro = n[1];
    }

    __device__ __noinline__ void sort_buf(int h, int n, real sgn) const {
        if (n > 1 && lane == 0)
            for (int i = 1; i < n; ++i) {
                real x = rt(h, i);
                int j = i - 1;
                while (j >= 0 && (sgn > 0 ? x < rt(h, j) : x > rt(h, j))) {
                    rt(h, j + 1) = rt(h, j);
                    --j;
                }
                rt(h, j + 1) = x;
            }
        sync();
    }

    // next primary breakpoint beyond tp (finalize! of every step, scanned): the kink points, the
    // clamps of the kinked dispatch, the clamps of the moved states of charge
    __device__ __noinline__ bool next_bp(real tp, real sgn, real *out) const {
        bool have = false;
        real best = 0;
        auto consider = [&](real x) {
            if (!isfinite(x)) return;
            if (!(sgn * x > 0)) return;
            if (!(sgn * (x - tp) > 0)) return;
            if (!have || sgn * (x - best) < 0) {
                best = x;
                have = true;
            }
        };
        for (int i = lane; i < (lvl ? 0 : 2 * U); i += G) {
            if (S(LL.kv, i) == 0) continue;
            real g = S(LL.kg, i), Q = S(LL.kq, i);
            consider(-Q / g);
            for (int c = 0; c < LL.K; ++c) {
                const int ka = 5 * (i * LL.K + c);
                real ak = S(LL.ka, ka);
                if (ak == 0) continue;
                real y0 = S(LL.ka, ka + 1);
                real offs[4] = {real(0), real(0), -ak * Q, ak * Q};
                real sls[4] = {ak * g, real(0), real(0), ak * g};
                for (int h = 0; h < 4; ++h) {
                    if (sls[h] == 0) continue;
                    consider((real(0) - y0 - offs[h]) / sls[h]);
                    consider((real(1) - y0 - offs[h]) / sls[h]);
                }
            }
        }
        // a unit inside its interval: the nearest clamp of the states inside the box, then the clamps of
        // the states outside it (each a state of a listed term); another: the clamps of all its states
        auto in_box = [&](int u) { return tp > S(LL.slo, u) && tp < S(LL.shi, u) && S(LL.slo, u) < S(LL.shi, u); };
        for (int u = lane; u < U; u += G) {
            if (!in_box(u)) continue;
            consider(sgn > 0 ? S(LL.shi, u) : S(LL.slo, u));
            int na = (int)S(LL.na, u);
            for (int i = 0; i < na; ++i) {
                int q = (int)S(LL.act, u * ESM_PLAT_NACT + i);
                for (int h = 0; h < 2; ++h) {
                    real y0 = h == 0 ? Y(u, q) : Y1(u, q);
                    if (y0 > 0 && y0 < 1) continue;
                    consider(real(0) - y0);
                    consider(real(1) - y0);
                }
            }
        }
        int u = 0, i = lane;
        while (u < U) {
            const int n = in_box(u) ? 0 : ns();
            if (i >= n) {
                i -= n;
                ++u;
                continue;
            }
            real y0 = Y(u, q0() + i);
            consider(real(0) - y0);
            consider(real(1) - y0);
            i += G;
        }
        sync();
        real key = tmin(have ? sgn * best : real(INFINITY));  // the nearest over the lanes (a sign flip is exact)
        have = key < real(INFINITY);
        *out = have ? sgn * key : real(0);
        return have;
    }

    // walk! (src/local.jl:1294) with storage splitting, to the right and then to the left; 1 both proper, 0
    // one improper, -1 buffer overflow (the first walk that is not proper counts). A state machine: each
    // iteration evaluates the move once, at whatever point the walk needs next, so the threads of a warp,
    // whose walks differ in length and in roots, stay together over the evaluation; the secondaries at a
    // point are saved before the roots of its segment are evaluated, so that none is evaluated again only to
    // restore them. The roots of both kinds come from one pass over the segment; those of the node balances
    // are taken again, piece by piece, only where the segment has storage roots. One
    // multiscale and one long-range sweep of 40 nodes, T=2920, 16 replicas: 193 ms with the evaluation called
    // from nine places of two walks; with this walk and the kernels below 53 to 74 ms, by the state.
    __device__ __noinline__ int walks(int *nr, int *nl) const {
        // the point evaluated next: 0; a breakpoint (chosen first); the slope probe of a ray step; the
        // segment's end; a storage root; the segment's end again; a node-balance root
        enum { START, NEXT, PROBE, END, STAT, BACK, ROOT, DONE };
        const int maxpts = M.maxpts;
        int st = START, after = END, rc = 1;
        real sgn = 1, tp = 0, t = 0, lo = 0, c = 0, zc = 0, cmin = 0, cprev = 0, delta = 0, hp = 0;
        real xs = 0, cs = 0, zs = 0;  // a storage root's point
        int np = 0, nx = 0, nro = 0, ri = 0, ngro = 0, gi = 0;
        *nr = *nl = 0;
        auto put = [&](real x, real v, real z) -> bool {
            if (np >= maxpts) {
                rc = -1;
                st = DONE;
                return false;
            }
            if (lane == 0) {
                const int a = sgn > 0 ? 0 : 3;
                pt(a, np) = x;
                pt(a + 1, np) = v;
                if constexpr (sizeof(real) == 4) pt(a + 2, np) = z;
            }
            ++np;
            cmin = fmin(cmin, v);
            cprev = v;
            return true;
        };
        auto finish = [&]() {  // the segment's end point and the stop test
            if (!put(t, c, zc)) return;
            if (c + real(0) - cmin > M.maxnats) {
                if (sgn > 0) {
                    *nr = np;
                    sgn = -1;
                    st = START;
                    np = nx = 0;
                    tp = cmin = cprev = delta = 0;
                } else {
                    *nl = np;
                    st = DONE;
                }
                return;
            }
            tp = t;
            st = NEXT;
        };
        auto station = [&]() {  // a storage root's point; the next one, or the segment's end again
            if (!put(xs, cs, zs)) return;
            lo = xs;
            st = ++gi < ngro ? STAT : BACK;
        };
        if (!on) st = DONE;
        while (G == 1 ? __any_sync(0xffffffffu, st != DONE) : st != DONE) {
            real te = 0;
            if (st == NEXT) {
                if (next_bp(tp, sgn, &t)) {
                    te = t;
                    st = END;
                } else {
                    hp = real(sizeof(real) == 4 ? 1e-3 : 1e-6) * fmax(real(1), fabs(tp));
                    te = tp + sgn * hp;
                    st = PROBE;
                }
            } else if (st == END || st == BACK) {
                te = t;
            } else if (st == STAT) {
                te = rt(1, gi);
            } else if (st == ROOT) {
                te = rt(0, ri);
            }
            __syncwarp();
            real v = 0;
            if (st != DONE) v = eval(te);
            const real z = nzs;
            __syncwarp();
            if (st == START) {
                save_prev();
                st = NEXT;
            } else if (st == PROBE) {
                real sl = (v + real(0) - cprev - real(0)) / hp;
                if (sl > 0)
                    delta = fmin(real(2) * M.maxnats / sl, real(1e3) * fmax(fabs(tp), real(1e-3)));
                else
                    delta = delta == 0 ? fmax(fabs(tp), real(1e-6)) : real(2) * delta;
                t = tp + sgn * delta;
                st = END;
                if (++nx > 80) {
                    rc = 0;
                    st = DONE;
                }
            } else if (st == ROOT) {
                if (put(te, v, z) && ++ri == nro) {
                    if (after == END)
                        finish();
                    else
                        station();
                }
            } else if (st != DONE) {
                // the piece lo .. te: its roots (of a segment's first pass: of both kinds)
                int ng = 0;
                if (st == END) {
                    c = v;
                    zc = z;
                    lo = tp;
                    gi = 0;
                }
                collect(lo, te, sgn, st == END, &nro, &ng);
                ri = 0;
                if (st == END) ngro = ng;
                if (st == STAT) {
                    xs = te;
                    cs = v;
                    zs = z;
                }
                after = st == STAT ? STAT : END;
                if (st == END && ngro > 0) {
                    sort_buf(1, min(ngro, ESM_PLAT_RB), sgn);
                    st = STAT;
                    if (ngro > ESM_PLAT_RB) {
                        rc = -1;
                        st = DONE;
                    }
                } else if (nro > ESM_PLAT_RB) {
                    rc = -1;
                    st = DONE;
                } else {
                    save_prev();
                    if (nro > 0) {
                        sort_buf(0, nro, sgn);
                        st = ROOT;
                    } else if (after == END) {
                        finish();
                    } else {
                        station();
                    }
                }
            }
        }
        sync();
        return rc;
    }

    __device__ static real logseg(real Ls, real x) {
        if (fabs(x) < real(1e-10)) return log(Ls) - x / 2;
        if (x > 0) return log(Ls) + log(-expm1(-x)) - log(x);
        return log(Ls) - x + log(-expm1(x)) - log(-x);
    }
    __device__ static real trexp_offset(real u, real g, real Ls, real flat) {
        real x = g * Ls;
        if (fabs(x) < flat) return u * Ls;
        if (g > 0) return -log1p(-u * (-expm1(-x))) / g;
        return Ls + log1p(-u * (-expm1(x))) / (-g);
    }
    __device__ inline real P(int i, int nl) const {
        return i < nl ? pt(3, nl - 1 - i) : (i == nl ? real(0) : pt(0, i - nl - 1));
    }
    __device__ inline real Cc(int i, int nl) const {
        return i < nl ? pt(4, nl - 1 - i) : (i == nl ? real(0) : pt(1, i - nl - 1));
    }
    __device__ inline real Zz(int i, int nl) const {
        return i < nl ? pt(5, nl - 1 - i) : (i == nl ? real(0) : pt(2, i - nl - 1));
    }

    // sample_line! (src/local.jl:1501), as Lane::sample_line: the segments' masses split over the lanes,
    // added in order
    __device__ __noinline__ real sample_line(real ucat, real uoff, bool *guard) const {
        *guard = false;
        int nr = 0, nl = 0;
        int w = walks(&nr, &nl);
        if (w < 0) *guard = true;
        if (w <= 0 || !on) return 0;
        int nseg = nl + nr;
        real mx = -INFINITY;
        for (int j = lane; j < nseg; j += G) {
            real p0 = P(j, nl), p1 = P(j + 1, nl), c0 = Cc(j, nl), c1 = Cc(j + 1, nl);
            real Ls = p1 - p0;
            real m = Ls > 0 ? -fmin(c0, c1) + logseg(Ls, fabs(c1 - c0)) : real(-INFINITY);
            lm(j) = m;
            mx = fmax(mx, m);
        }
        sync();
        mx = tmax(mx);
        for (int j = lane; j < nseg; j += G) lm(j) = exp(lm(j) - mx);
        sync();
        real tot = 0;
        for (int j = 0; j < nseg; ++j) tot += lm(j);
        real u = ucat * tot, acc = 0;
        int jj = nseg - 1;
        for (int q = 0; q < nseg; ++q) {
            acc += lm(q);
            if (u <= acc) {
                jj = q;
                break;
            }
        }
        real p0 = P(jj, nl), p1 = P(jj + 1, nl);
        real Ls = p1 - p0;
        real g = (Cc(jj + 1, nl) - Cc(jj, nl)) / Ls;
        real flat = sizeof(real) == 4 ? real(1e-4) : real(1e-10);
        if constexpr (sizeof(real) == 4) {
            auto slope = [&](int j) -> real {
                if (j < 0 || j >= nseg) return 0;
                real Lj = P(j + 1, nl) - P(j, nl);
                return Lj > 0 ? fabs((Cc(j + 1, nl) - Cc(j, nl)) / Lj) : real(0);
            };
            real gl = slope(jj - 1), gm = slope(jj), gr = slope(jj + 1);
            real z0 = Zz(jj, nl) + real(2.4e-7) * fabs(p0) * fmax(gl, gm);
            real z1 = Zz(jj + 1, nl) + real(2.4e-7) * fabs(p1) * fmax(gm, gr);
            flat = fmax(flat, z0 + z1);
        }
        return (g >= 0 || fabs(g * Ls) < flat) ? p0 + trexp_offset(uoff, g, Ls, flat)
                                               : p1 - trexp_offset(uoff, -g, Ls, flat);
    }

    // logjac (src/local.jl:1871) of the compensations, in FP64 in both builds (the log-acceptance
    // ratio is an FP64 quantity; its inputs are the build's values)
    __device__ __noinline__ double logjac(real t, bool *any) const {
        auto lg = [&](int i) -> double {
            if (S(LL.kv, i) == 0) return 0.0;
            double Q = S(LL.kq, i);
            return log(fabs((fmax(Q + (double)S(LL.kg, i) * (double)t, 0.0) + (double)S(LL.ke, i)) /
                            (double)S(LL.kp, i)));
        };
        double *lw = reinterpret_cast<double *>(sm + LL.w);
        if constexpr (G > 1) {
            sync();
            for (int i = lane; i < (lvl ? 0 : 2 * U); i += G) lw[i] = lg(i);
            sync();
        }
        double lj = 0;
        *any = false;
        for (int s = 0; s < (lvl ? 0 : 2); ++s)
            for (int u = 0; u < U; ++u) {
                const int i = 2 * u + s;
                if (S(LL.kv, i) == 0) continue;
                *any = true;
                lj += (double)S(LL.knm, i) * (G > 1 ? lw[i] : lg(i));
            }
        return lj;
    }

    // commit_block! (src/local.jl:2495): states of charge, kinked dispatch, node balances (each
    // global write by one lane; all by one, in order, where two units share a node)
    __device__ __noinline__ void commit(real t) const {
        eval(t);
        sync();
        auto end = [&](int i) {  // an end step: the compensation and the node balance
            const int u = i >> 1, n = node(u), tau = tau_end(i & 1);
            real ph = S(LL.kph, i);
            int c = 0;
            for (int p = M.up[n]; p < M.up[n + 1] && c < LL.K; ++p, ++c) {
                real ak = S(LL.ka, 5 * (i * LL.K + c));
                if (ak != 0) M.g[ix(M.ua[p], tau)] += ak * ph;
            }
            M.r[ix(n, tau)] += S(LL.dr, i);
        };
        auto inner = [&](int u, bool in, int q) {  // an interior step whose injection changes
            if (!in && quiet(u, q, t)) return;
            real dj, d1;
            sterm(u, q, t, &dj, &d1);
            M.r[ix(node(u), stp(q))] += dj;
        };
        if (dup) {
            if (lane == 0)
                for (int u = 0; u < U; ++u) {
                    for (int s = 0; s < (lvl ? 0 : 2); ++s) end(2 * u + s);
                    const bool in = inside(u, t);
                    const int nt = nterms(u, in);
                    for (int i = 0; i < nt; ++i) inner(u, in, term_q(u, in, i));
                }
        } else {
            for (int i = lane; i < (lvl ? 0 : 2 * U); i += G) end(i);
            each_term(
                [&](int u, bool *in) {
                    *in = inside(u, t);
                    return nterms(u, *in);
                },
                inner);
        }
        sync();
        for (int u = 0; u < U; ++u) {
            for (int p = lane; p < ns(); p += G) M.e[ix(uj[u], stp(q0() + p))] += t;
            if (dup) sync();
        }
        sync();
    }
};

// One class pass of the storage multiscale sweep: threads (G 1) or warps (G 32) take (block, replica)
// tasks, replica fastest, and run the class's moves in order. Blocks of one warp: the tasks of the
// middle lengths make fewer warps than the device has schedulers.
template <class real, int G>
__global__ void __launch_bounds__(32, 16) k_plateau(const __grid_constant__ DevModel<real> M,
                                                    const __grid_constant__ PlatMoves mv,
                                                    const __grid_constant__ PlatLayout LL, uint32_t sweep,
                                                    real *scratch, unsigned long long *stats) {
    extern __shared__ __align__(16) char plat_smem[];
    real local[G == 1 ? ESM_PLAT_LOCAL : 1];
    const size_t n = (size_t)gridDim.x * (32 / G);  // tasks at a time
    const size_t slot = (size_t)blockIdx.x * (32 / G) + (G == 1 ? threadIdx.x : 0);
    const bool loc = LL.total <= ESM_PLAT_LOCAL;
    real *lay = G == 32 ? reinterpret_cast<real *>(plat_smem) : loc ? local : scratch + slot;
    PLane<real, G> Ln(M, LL, lay, G == 32 || loc ? 1 : (int)n, scratch + (G == 32 ? slot * LL.gtotal : 0));
    Ln.L = mv.L;
    Ln.inorder = mv.L < ESM_PLAT_SHORT;
    unsigned long long tried = 0, moved = 0, guards = 0;
    const size_t ntask = (size_t)mv.nb * M.R;
    const size_t wbase = (size_t)blockIdx.x * (32 / G);
    for (size_t base = wbase; base < ntask; base += n) {  // (the threads of a warp stay together)
        const size_t task = base + (slot - wbase);
        Ln.on = task < ntask;
        int k = (int)((Ln.on ? task : base) / M.R);
        Ln.rep = (int)((Ln.on ? task : base) % M.R);
        Ln.b0 = mv.o + (2 * k + mv.cls) * mv.L;
        for (int m = 0; m < 8; ++m) {
            Ln.U = mv.nu[m];
            Ln.uj = mv.j[m];
            if (Ln.U <= 0) continue;
            if (Ln.on) {
                Ln.load();
                Ln.intervals();
                Ln.kinks();
            }
            uint32_t w0 = 2u * (8u * (uint32_t)mv.li + (uint32_t)m);
            double uc, uo, uj, un;
            uniform2(M.seed, ESM_TAG_SML, w0, (uint32_t)Ln.b0, (uint32_t)Ln.rep, sweep, &uc, &uo);
            bool guard;
            real t = Ln.sample_line(unit_uniform<real>(uc), unit_uniform<real>(uo), &guard);
            if (!Ln.on) continue;
            if (guard) ++guards;
            if (t != 0) {
                bool any;
                double lj = Ln.logjac(t, &any);
                if (any) {
                    uniform2(M.seed, ESM_TAG_SML, w0 + 1, (uint32_t)Ln.b0, (uint32_t)Ln.rep, sweep, &uj, &un);
                    if (uj >= exp(fmin(0.0, lj))) t = 0;
                }
            }
            if (t != 0) Ln.commit(t);
            ++tried;
            if (t != 0) ++moved;
        }
    }
    if (Ln.lane == 0) {
        if (tried) atomicAdd(&stats[0], tried);
        if (moved) atomicAdd(&stats[1], moved);
        if (guards) atomicAdd(&stats[2], guards);
    }
}

// The long-range storage sweep (storage_long_sweep!, src/storage_long.jl:245): warps or blocks of G
// threads take (unit, replica) tasks and run the unit's moves in order -- the level move (every instant of the year
// rises) and the long-range plateaus (prep_slong!, :77: one unit, the cyclic instants a+1 .. a+L,
// compensation at steps a and a+L). plan: per unit [stor index, moves, (L, a) per move]; L = T is the
// level move. The moves of different units touch different nodes (one unit per node and carrier).
// A move's points each go over up to T states and evaluate those that a bound is near: the states and
// the terms of the last two points stay in shared memory where a year of them fits (ESM_PLAT_STAGE;
// else the terms in the global slab), so that the roots between two points need no second evaluation.
// G is 256, or 32 for a year of
// at most 256 steps, where 8 warps wait for one another longer than they share (T=120, 33 units, 33
// replicas: 1.6 ms with 32, 2.1 with 256). 40 units, T=2920: 80 -> 25 ms at 16 replicas, 106 -> 47 at 64.
template <class real, int G>
__global__ void __launch_bounds__(G, 512 / G) k_storage_long(const __grid_constant__ DevModel<real> M, const int *plan,
                                                          const __grid_constant__ PlatLayout LL, int nunits,
                                                          uint32_t sweep, real *scratch, unsigned long long *stats) {
    extern __shared__ __align__(16) char plat_smem[];
    PLane<real, G> Ln(M, LL, reinterpret_cast<real *>(plat_smem), 1, scratch + (size_t)blockIdx.x * LL.gtotal);
    unsigned long long tried = 0, moved = 0, guards = 0;
    const size_t ntask = (size_t)nunits * M.R;
    for (size_t task = blockIdx.x; task < ntask; task += gridDim.x) {
        const int *pu = plan + (task / M.R) * ESM_SL_STRIDE;
        Ln.rep = (int)(task % M.R);
        Ln.U = 1;
        Ln.uj = pu;
        for (int m = 0; m < pu[1]; ++m) {
            int L = pu[2 + 2 * m], a = pu[3 + 2 * m];
            Ln.lvl = L >= M.T;
            Ln.L = Ln.lvl ? M.T : L;
            Ln.b0 = Ln.lvl ? 0 : a;
            Ln.load();
            Ln.intervals();
            if (!Ln.lvl) Ln.kinks();
            double uc, uo, uj, un;
            uniform2(M.seed, ESM_TAG_SLL, 2u * (uint32_t)m, (uint32_t)pu[0], (uint32_t)Ln.rep, sweep, &uc, &uo);
            bool guard;
            real t = Ln.sample_line(unit_uniform<real>(uc), unit_uniform<real>(uo), &guard);
            if (guard) ++guards;
            if (t != 0 && !Ln.lvl) {
                bool any;
                double lj = Ln.logjac(t, &any);
                if (any) {
                    uniform2(M.seed, ESM_TAG_SLL, 2u * (uint32_t)m + 1, (uint32_t)pu[0], (uint32_t)Ln.rep, sweep, &uj,
                             &un);
                    if (uj >= exp(fmin(0.0, lj))) t = 0;
                }
            }
            if (t != 0) Ln.commit(t);
            if (M.mlog && Ln.rep < M.mlog_nrep && Ln.lane == 0)
                M.mlog[((task / M.R) * 5 + m) * M.mlog_nrep + Ln.rep] = (double)t;
            ++tried;
            if (t != 0) ++moved;
        }
    }
    if (Ln.lane == 0) {
        if (tried) atomicAdd(&stats[0], tried);
        if (moved) atomicAdd(&stats[1], moved);
        if (guards) atomicAdd(&stats[2], guards);
    }
}

// A class pass's tasks take a warp each if the blocks are long, whose interior steps the lanes share, or
// if the tasks are no more than the warps that the device holds at 128 registers (16 an SM): by threads,
// a pass takes as long as the longest walk of 32 however few they are. 40 nodes, T=584, 16 replicas (at
// most 2336 tasks a pass): a sweep takes 61 ms by threads, 29 by warps; 12 nodes, T=24, 4 replicas: 22 and
// 6.6. Beyond, the threads of a warp share its instructions: 40 nodes, T=2920, 64 replicas, 5824 tasks of 16
// steps take 4.5 to 6.5 ms by threads, and half as many of 32 steps 4.8 to 5.4 by warps.
inline bool plat_wide(int L, size_t ntask) {
    int dev = 0, nsm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return L >= ESM_PLAT_SHORT || ntask <= (size_t)nsm * 16;
}

inline bool long_block(int T) { return T > 256; }
// the layout of a long-range task: states and terms in shared memory, the terms in the global slab, or both there
template <class real>
PlatLayout long_layout(const DevModel<real> &M, int maxd) {
    if (!long_block(M.T)) return plat_layout(M.maxpts, 1, maxd, M.T + 1, true);
    PlatLayout LL = plat_layout(M.maxpts, 1, maxd, M.T + 1, true, M.T);
    if (LL.total * sizeof(real) > ESM_PLAT_STAGE) LL = plat_layout(M.maxpts, 1, maxd, M.T + 1, true, 0, M.T);
    if (LL.total * sizeof(real) > ESM_PLAT_STAGE) LL = plat_layout(M.maxpts, 1, maxd, 0, true, 0, M.T);
    return LL;
}

// the reals of global scratch that the storage kernels use if they can have them: the slabs of 32 warps an
// SM or 2 long-range tasks an SM, or the layouts of 512 threads an SM if the largest is beyond their
// local arrays. The kernels' shared memory limit is set here.
template <class real>
size_t plateau_scratch_reals(const DevModel<real> &M, int maxd, size_t *least) {
    int dev = 0, nsm = 1, lim = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncSetAttribute(k_plateau<real, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    cudaFuncSetAttribute(k_storage_long<real, ESM_PLAT_LONG>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    const size_t thread = plat_layout(M.maxpts, ESM_PLAT_MAXU, maxd, 0, false).total;
    const size_t warp = plat_layout(M.maxpts, 1, 1, 0, true).gtotal, lng = long_layout(M, maxd).gtotal;
    const size_t t = thread <= ESM_PLAT_LOCAL ? 0 : thread;
    auto most = [](size_t a, size_t b, size_t c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); };
    *least = most(32 * t, warp, lng);  // one task each
    return most((size_t)nsm * 512 * t, (size_t)nsm * 32 * warp, (size_t)nsm * 2 * lng);
}
template <class real>
cudaError_t launch_storage_long(const DevModel<real> &M, int maxd, const int *plan, int nunits, uint32_t sweep,
                                real *scratch, size_t reals, unsigned long long *stats, cudaStream_t s) {
    const PlatLayout LL = long_layout(M, maxd);
    const size_t ntask = (size_t)nunits * M.R, slots = reals / LL.gtotal;
    const unsigned blocks = (unsigned)(ntask < slots ? ntask : slots);
    const size_t smem = LL.total * sizeof(real);
    if (long_block(M.T))
        k_storage_long<real, ESM_PLAT_LONG><<<blocks, ESM_PLAT_LONG, smem, s>>>(M, plan, LL, nunits, sweep, scratch, stats);
    else
        k_storage_long<real, 32><<<blocks, 32, smem, s>>>(M, plan, LL, nunits, sweep, scratch, stats);
    return cudaGetLastError();
}
template <class real>
cudaError_t launch_plateau(const DevModel<real> &M, int maxd, const PlatMoves &mv, uint32_t sweep, real *scratch,
                           size_t reals, unsigned long long *stats, cudaStream_t s) {
    int U = 1;
    for (int m = 0; m < 8; ++m) U = mv.nu[m] > U ? mv.nu[m] : U;
    size_t ntask = (size_t)mv.nb * M.R;
    if (plat_wide(mv.L, ntask)) {
        const PlatLayout LL = plat_layout(M.maxpts, U, maxd, mv.L + 2, true);
        const size_t slots = reals / LL.gtotal;
        k_plateau<real, 32><<<(unsigned)(ntask < slots ? ntask : slots), 32, LL.total * sizeof(real), s>>>(
            M, mv, LL, sweep, scratch, stats);
    } else {
        const PlatLayout LL = plat_layout(M.maxpts, U, maxd, 0, false);
        const size_t warps = (ntask + 31) / 32, slots = reals / LL.total / 32;
        k_plateau<real, 1><<<(unsigned)(LL.total <= ESM_PLAT_LOCAL || warps < slots ? warps : slots), 32, 0, s>>>(
            M, mv, LL, sweep, scratch, stats);
    }
    return cudaGetLastError();
}

}  // namespace esm
