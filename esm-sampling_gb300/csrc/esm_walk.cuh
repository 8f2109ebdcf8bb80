// The walk of the other line moves (angles, generators, lines, at most one storage unit; no
// compensation): one lane per (task, direction), every evaluation of the walk in one place.
//
// The one-lane walk (Lane::walk) calls the evaluation from nine places inside loops whose trip counts
// differ between the lanes, over terms that it fetches through tables in device memory: 13 to 27 of 32
// lanes active, and a task's two directions one after the other. Here a warp walks 16 tasks, both
// directions at once. A lane is a state machine: each iteration of the warp evaluates the move once for
// every lane that still walks, at whatever point the lane needs next, so the lanes stay together over
// the terms. The move's constants are in shared memory once per block, the task's values (states, flows,
// balances, breakpoints) once per task, the balances at the lane's last two points interleaved by lane
// (no bank conflicts). The points go to a local array: written once, read by their own lane.
// Evaluations that only restored the balances at a point are left out: they are saved before the roots
// of the segment are evaluated. Every value has the one-lane walk's rounding (esm_sepwalk.cuh's fma_rn).
// What bounds it: the instruction issue and latency of the evaluations, the lanes leaving the loop one
// by one. Measured per move at 40 nodes, T = 2920, 64 replicas (93440 tasks), FP32, one-lane walk and
// this one: spair 0.70 and 0.27 ms, xpair 0.54 and 0.27, potential 0.48 and 0.27, xloc 0.27 and 0.16,
// angle atoms 0.40 and 0.21, generator atoms 0.37 and 0.18.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "esm_common.cuh"

namespace esm {

#define ESM_WALK_WARPS 4     // warps of a block
#define ESM_WALK_PTS 192     // points of a lane's local arrays (a larger cap: the lane's column of a slab)
#define ESM_WALK_ROOTS 8     // node-balance roots of one segment taken at a time

// Shared memory of a move's walk: constants per block, values per task and per lane.
struct WalkLayout {
    int ng, nga, nl, nse, nns, nna;
    int nb;                                // breakpoint candidates
    int kx, ky, kak, ka, kpos;             // generators (tau, then tau - 1): dt mc, penalty, av k, coefficient, node slot
    int la, ls, lpa, lpb;                  // lines: coefficient, limit, node slots
    int consts;                            // constants, in words of 4 or 8 bytes
    int ty, tf, tr, tb, task;              // per task: generators, flows, balances (tau, then tau - 1), candidates
    int cur, prev, ro, go, lane;           // per lane: balances at the last point and before, roots, storage roots
};
template <class real>
__host__ __device__ inline WalkLayout walk_layout(int ng, int nga, int nl, int nse, int nns, int nna) {
    WalkLayout w;
    w.ng = ng;
    w.nga = nga;
    w.nl = nl;
    w.nse = nse;
    w.nns = nns;
    w.nna = nna;
    int n = ng + nga, m = nns + nna, o = 0;
    w.nb = 2 * (n + nl + nse);
    w.kx = o; o += n;
    w.ky = o; o += n;
    w.kak = o; o += n;
    w.ka = o; o += n;
    w.kpos = o; o += n;
    w.la = o; o += nl;
    w.ls = o; o += nl;
    w.lpa = o; o += nl;
    w.lpb = o; o += nl;
    w.consts = o;
    o = 0;
    w.ty = o; o += n;
    w.tf = o; o += nl;
    w.tr = o; o += m;
    w.tb = o; o += w.nb;
    w.task = o;
    o = 0;
    w.cur = o; o += m;
    w.prev = o; o += m;
    w.ro = o; o += ESM_WALK_ROOTS;
    w.go = o; o += 6 * nse;
    w.lane = o;
    return w;
}
template <class real>
__host__ __device__ inline int walk_const_bytes(const WalkLayout &w) {
    return ((int)sizeof(real) * w.consts + 15) & ~15;
}
template <class real>
__host__ __device__ inline int walk_warp_bytes(const WalkLayout &w) {
    return ((int)sizeof(real) * (16 * w.task + 32 * w.lane) + 15) & ~15;
}

template <class real>
struct WalkIndex;  // an index kept among the reals
template <>
struct WalkIndex<float> {
    __device__ static float put(int i) { return __int_as_float(i); }
    __device__ static int get(float x) { return __float_as_int(x); }
};
template <>
struct WalkIndex<double> {
    __device__ static double put(int i) { return __longlong_as_double(i); }
    __device__ static int get(double x) { return (int)__double_as_longlong(x); }
};

template <class real>
struct LineWalk {
    const DevModel<real> &M;
    const WalkLayout &W;
    const real *K;        // constants
    real *tv, *lv;        // this lane's columns of the task and the lane values
    real *pts;            // points: time, potential, round-off scale, mass
    int pstride, pcap;
    const SepUnit<real> &u;

    __device__ __forceinline__ real &T(int i) const { return tv[i * 16]; }
    __device__ __forceinline__ real &L(int i) const { return lv[i * 32]; }
    __device__ __forceinline__ real &pt(int a, int k) const { return pts[(size_t)(a * pcap + k) * pstride]; }

    __device__ __forceinline__ static void sum(real v, real &D, real &A) {
        D = add_rn(D, v);
        if constexpr (sizeof(real) == 4) A = add_rn(A, fabs(v));
    }
    // clamp_diff
    __device__ __forceinline__ static void clamp(real y0, real dy, real *dyc, real *dex) {
        real y1 = add_rn(y0, dy);
        real c0 = clampr<real>(y0, 0, 1), c1 = clampr<real>(y1, 0, 1);
        bool in = y0 > 0 && y0 < 1 && y1 > 0 && y1 < 1, above = y0 >= 1 && y1 >= 1, below = y0 <= 0 && y1 <= 0;
        *dyc = in ? dy : (above || below) ? real(0) : sub_rn(c1, c0);
        *dex = in ? real(0) : above ? dy : below ? -dy : sub_rn(fabs(sub_rn(y1, c1)), fabs(sub_rn(y0, c0)));
    }
    __device__ __forceinline__ void gens(int q0, int n, int at, real t, real &D, real &A) const {
        for (int q = q0; q < q0 + n; ++q) {
            real dyc, dex;
            clamp(T(W.ty + q), mul_rn(t, K[W.ka + q]), &dyc, &dex);
            real dp = mul_rn(K[W.kak + q], dyc);
            sum(fma_rn(K[W.ky + q], dex, mul_rn(K[W.kx + q], dp)), D, A);
            real &x = L(W.cur + at + WalkIndex<real>::get(K[W.kpos + q]));
            x = sub_rn(x, dp);
        }
    }
    __device__ __forceinline__ void nodes(int q0, int n, real &D, real &A) const {
        for (int q = q0; q < q0 + n; ++q)
            sum(mul_rn(M.dt, SepUnit<real>::phi(T(W.tr + q), L(W.cur + q), M.c_shed, M.c_dump)), D, A);
    }
    // Lane::eval: beta * (cost change) at t; the balance changes into cur, the storage term's d into dcs
    // and dca, the round-off scale into z
    __device__ __forceinline__ real eval(real t, real *z, real *dcs, real *dca) const {
        real D = 0, A = 0;
        const int m = W.nns + W.nna;
        for (int q = 0; q < m; ++q) L(W.cur + q) = 0;
        gens(0, W.ng, 0, t, D, A);
        const real cd = mul_rn(M.c_viol, M.dt);
        for (int q = 0; q < W.nl; ++q) {
            real df = mul_rn(t, K[W.la + q]), f0 = T(W.tf + q), s = K[W.ls + q];
            real f1 = add_rn(f0, df);  // hinge_diff
            real far = sub_rn(fmax(sub_rn(fabs(f1), s), real(0)), fmax(sub_rn(fabs(f0), s), real(0)));
            real h = (fabs(f0) <= s && fabs(f1) <= s) ? real(0)
                     : (f0 > s && f1 > s)             ? df
                     : (f0 < -s && f1 < -s)           ? -df
                                                      : far;
            sum(mul_rn(cd, h), D, A);
            real &a = L(W.cur + WalkIndex<real>::get(K[W.lpa + q]));
            a = add_rn(a, df);
            real &b = L(W.cur + WalkIndex<real>::get(K[W.lpb + q]));
            b = sub_rn(b, df);
        }
        real x = 0, dd = 0, dex = 0;
        if (W.nse) {  // (one unit, at the first storage slot of both steps)
            x = mul_rn(t, u.a);
            real dc;
            clamp(u.e0, x, &dc, &dex);
            dd = mul_rn(u.h, dc) / M.dt;
            real di;
            sum(u.cost(u.w, -dd, dex, &di, dcs), D, A);
            real &b = L(W.cur + u.pos);
            b = fma_rn(u.k, di, b);
        }
        nodes(0, W.nns, D, A);
        if (W.nna) {
            gens(W.ng, W.nga, W.nns, t, D, A);
            if (W.nse) {
                real di;
                sum(u.cost(u.t, dd, real(0), &di, dca), D, A);
                real &b = L(W.cur + W.nns + u.posa);
                b = fma_rn(u.k, di, b);
            }
            nodes(W.nns, W.nna, D, A);
        }
        if constexpr (sizeof(real) == 4) *z = mul_rn(mul_rn(M.beta_v, A), real(4.8e-7));
        return mul_rn(M.beta_v, D);
    }

    // One direction of walk! (src/local.jl:1294) for every lane with on; returns 1 proper, 0 improper,
    // -1 more points than the cap.
    __device__ __forceinline__ int walk(bool on, real sgn, int *npts) const {
        // the point that a lane evaluates next: 0; a breakpoint (chosen first); the slope probe of a ray
        // step; the segment's end; a storage root; the segment's end again; a node-balance root; the ends
        // of the segment again, for more roots than the buffer takes
        enum { START, NEXT, PROBE, END, STAT, BACK, ROOT, MORE0, MORE1, DONE };
        const int maxpts = M.maxpts, m = W.nns + W.nna;
        int st = on ? START : DONE, after = NEXT, rc = 0;
        real tp = 0, t = 0, lo = 0, hi = 0, last = 0;  // walked to; segment end; piece; last root taken
        real c = 0, zc = 0, cmin = 0, cprev = 0, delta = 0, hp = 0;
        real xs = 0, cs = 0, zs = 0;                   // a storage root's point
        real pdcs = 0, pdca = 0, dcs = 0, dca = 0;     // the storage term's d, before and now
        int np = 0, nx = 0, nro = 0, ri = 0, ngo = 0, gi = 0;
        int nlast = 0;  // roots of the segment taken at `last`
        bool more = false;
        auto push = [&](real x, real v, real z) {
            if (np >= maxpts) {
                rc = -1;
                st = DONE;
                return;
            }
            pt(0, np) = fabs(x);
            pt(1, np) = v;
            if constexpr (sizeof(real) == 4) pt(2, np) = z;
            ++np;
            cmin = fmin(cmin, v);
            cprev = v;
        };
        auto save = [&]() {
            for (int q = 0; q < m; ++q) L(W.prev + q) = add_rn(T(W.tr + q), L(W.cur + q));
            pdcs = dcs;
            pdca = dca;
        };
        // the sign changes of the node balances between lo and hi in walking order, as many as the buffer
        // takes; beyond: those after the roots already taken, of which nlast lie at `last`
        auto roots = [&](bool beyond) {
            int skip = beyond ? nlast : 0;
            if (!beyond) nlast = 0;
            nro = 0;
            more = false;
            for (int q = 0; q < m; ++q) {
                real x, b = add_rn(T(W.tr + q), L(W.cur + q));
                if (!sep_root<real>(L(W.prev + q), b, lo, hi, sgn, &x)) continue;
                if (beyond && !(sgn * (x - last) > 0) && (x != last || skip-- > 0)) continue;
                int j = nro;
                if (j == ESM_WALK_ROOTS) {
                    more = true;
                    --j;
                    if (!(sgn * (L(W.ro + j) - x) > 0)) continue;
                } else {
                    ++nro;
                }
                for (; j > 0 && (sgn > 0 ? x < L(W.ro + j - 1) : x > L(W.ro + j - 1)); --j) L(W.ro + j) = L(W.ro + j - 1);
                L(W.ro + j) = x;
            }
            ri = 0;
        };
        auto finish = [&]() {  // the segment's end point and the stop test
            push(t, c, zc);
            if (st == DONE) return;
            if (add_rn(c, real(0)) - cmin > M.maxnats) {
                rc = 1;
                st = DONE;
                return;
            }
            tp = t;
            st = NEXT;
        };
        auto station = [&]() {  // a storage root's point; the next one, or the segment's end again
            push(xs, cs, zs);
            if (st == DONE) return;
            lo = xs;
            ++gi;
            st = gi < ngo ? STAT : BACK;
        };
        while (__any_sync(0xffffffffu, st != DONE)) {
            if (st != DONE) {
                real te = 0;
                if (st == NEXT) {
                    bool have = false;
                    real best = 0;
                    for (int q = 0; q < W.nb; ++q) {
                        real x = T(W.tb + q);
                        if (sgn * x > 0 && sgn * (x - tp) > 0 && (!have || sgn * (x - best) < 0)) {
                            best = x;
                            have = true;
                        }
                    }
                    if (have) {
                        t = te = best;
                        st = END;
                    } else {
                        hp = real(sizeof(real) == 4 ? 1e-3 : 1e-6) * fmax(real(1), fabs(tp));
                        te = tp + sgn * hp;
                        st = PROBE;
                    }
                } else if (st == END || st == BACK) {
                    te = t;
                } else if (st == STAT) {
                    te = L(W.go + gi);
                } else if (st == ROOT) {
                    te = L(W.ro + ri);
                } else if (st == MORE0) {
                    te = lo;
                } else if (st == MORE1) {
                    te = hi;
                }
                real z = 0;
                real v = eval(te, &z, &dcs, &dca);
                bool piece = false;
                if (st == START || st == MORE0) {
                    save();
                    st = st == START ? NEXT : MORE1;
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
                } else if (st == END) {
                    c = v;
                    zc = z;
                    lo = tp;
                    ngo = 0;
                    if (W.nse) {  // the sign changes of the storage secondaries (src/local.jl:885)
#pragma unroll
                        for (int i = 0; i < 6; ++i) {
                            real d0 = i < 3 ? pdcs : pdca, d1 = i < 3 ? dcs : dca, x;
                            real a = i % 3 == 0 ? d0 : i % 3 == 1 ? (u.ein > 0 ? sub_rn(d0, u.ein) : real(1)) : sec(d0);
                            real b = i % 3 == 0 ? d1 : i % 3 == 1 ? (u.ein > 0 ? sub_rn(d1, u.ein) : real(1)) : sec(d1);
                            if (!sep_root<real>(a, b, tp, t, sgn, &x)) continue;
                            int j = ngo++;
                            for (; j > 0 && (sgn > 0 ? x < L(W.go + j - 1) : x > L(W.go + j - 1)); --j)
                                L(W.go + j) = L(W.go + j - 1);
                            L(W.go + j) = x;
                        }
                    }
                    if (ngo > 0) {
                        gi = 0;
                        st = STAT;
                    } else {
                        hi = t;
                        after = END;
                        piece = true;
                    }
                } else if (st == STAT) {
                    xs = te;
                    cs = v;
                    zs = z;
                    hi = te;
                    after = STAT;
                    piece = true;
                } else if (st == BACK) {
                    hi = t;
                    after = END;
                    piece = true;
                } else if (st == MORE1) {
                    piece = true;
                } else {  // ROOT
                    push(te, v, z);
                    nlast = nlast > 0 && te == last ? nlast + 1 : 1;
                    last = te;
                    if (st != DONE && ++ri == nro) {
                        if (more)
                            st = MORE0;
                        else if (after == END)
                            finish();
                        else
                            station();
                    }
                }
                if (piece) {
                    roots(st == MORE1);
                    save();
                    if (nro > 0)
                        st = ROOT;
                    else if (after == END)
                        finish();
                    else
                        station();
                }
            }
        }
        *npts = np;
        return rc;
    }
    __device__ __forceinline__ real sec(real d) const { return fma_rn(-d, u.eout, real(-1)); }

    // sample_line! (src/local.jl:1501) over the pair's two walks: the right walk in the even lane, the
    // left walk in the odd one; both lanes return the draw
    __device__ __forceinline__ real sample(bool on, bool left, int np, real ucat, real uoff) const {
        const unsigned all = 0xffffffffu;
        real mx = -INFINITY, q0 = 0, d0 = 0;
        int n = on ? np : 0;
        for (int k = 0; k < n; ++k) {
            real p = pt(0, k), v = pt(1, k);
            real Ls = p - q0;
            real lm = Ls > 0 ? -fmin(d0, v) + Lane<real>::logseg(Ls, fabs(v - d0)) : real(-INFINITY);
            pt(3, k) = lm;
            mx = fmax(mx, lm);
            q0 = p;
            d0 = v;
        }
        mx = fmax(mx, __shfl_xor_sync(all, mx, 1));
        for (int k = 0; k < n; ++k) pt(3, k) = exp(pt(3, k) - mx);
        // the sums in segment order: the left walk from its last point inward, then the right walk
        real s = 0;
        if (left)
            for (int k = n - 1; k >= 0; --k) s += pt(3, k);
        s = __shfl_sync(all, s, (threadIdx.x & 31) | 1);
        if (!left)
            for (int k = 0; k < n; ++k) s += pt(3, k);
        real u_ = ucat * __shfl_sync(all, s, (threadIdx.x & 31) & ~1);
        real acc = 0;
        int seg = -1;
        if (left)
            for (int k = n - 1; k >= 0; --k) {
                acc += pt(3, k);
                if (u_ <= acc) {
                    seg = k;
                    break;
                }
            }
        acc = __shfl_sync(all, acc, (threadIdx.x & 31) | 1);
        bool found = __shfl_sync(all, seg, (threadIdx.x & 31) | 1) >= 0;
        if (!left && !found) {
            seg = n - 1;
            for (int k = 0; k < n; ++k) {
                acc += pt(3, k);
                if (u_ <= acc) {
                    seg = k;
                    break;
                }
            }
        }
        bool mine = left ? seg >= 0 : !found;
        // the other walk's first point: the neighbour of this walk's first segment
        real fp = n > 0 ? pt(0, 0) : real(0), fc = n > 0 ? pt(1, 0) : real(0);
        real op = __shfl_xor_sync(all, fp, 1), oc = __shfl_xor_sync(all, fc, 1);
        real t = 0;
        if (on && mine) {
            auto P = [&](int k) -> real { return k == -2 ? -op : k < 0 ? real(0) : pt(0, k); };
            auto C = [&](int k) -> real { return k == -2 ? oc : k < 0 ? real(0) : pt(1, k); };
            // point k (outer) and k - 1 (inner) of the walk, times as distances from the start
            real po = P(seg), pi = P(seg - 1), co = C(seg), ci = C(seg - 1);
            real p0 = left ? -po : pi, p1 = left ? -pi : po, c0 = left ? co : ci, c1 = left ? ci : co;
            real Ls = p1 - p0;
            real g = (c1 - c0) / Ls;
            real flat = Lane<real>::flat_nats;
            if constexpr (sizeof(real) == 4) {
                auto slope = [&](int k) -> real {  // of segment k; -1: the other walk's first
                    if (k >= n) return 0;
                    real Lk = P(k) - P(k - 1);
                    return Lk > 0 ? fabs((C(k) - C(k - 1)) / Lk) : real(0);
                };
                auto Z = [&](int k) -> real { return k < 0 ? real(0) : pt(2, k); };
                real gm = slope(seg), gi = slope(seg - 1), go = slope(seg + 1);
                real zi = Z(seg - 1) + real(2.4e-7) * fabs(pi) * fmax(gi, gm);
                real zo = Z(seg) + real(2.4e-7) * fabs(po) * fmax(gm, go);
                flat = fmax(flat, left ? zo + zi : zi + zo);
            }
            t = sep_pick<real>(p0, p1, g, Ls, uoff, flat);
        }
        real to = __shfl_xor_sync(all, t, 1);
        return mine ? t : to;
    }
};

// The shared memory of a move's walk in a block with one warp, by its header; more than any block has where
// the walk is not this file's: kinks, several storage units, or a separable move (one that the block walk does
// not take keeps the one-lane walk, which advances its potential along the units' slopes: other roundings).
template <class real>
__device__ inline int walk_bytes(const int *h) {
    if (h[3] > 0 || h[4] > 0 || h[1] > 1 || sep_units(h) > 0) return 0x7fffffff;
    const WalkLayout w = walk_layout<real>(h[0], h[6], h[2], h[1], h[5], h[7]);
    return walk_const_bytes<real>(w) + walk_warp_bytes<real>(w);
}
// whether the move of a descriptor's header is walked so in a block with `region` bytes
__device__ inline bool walk_move(const int *hdr, int region) { return hdr[13] <= region; }
template <class real>
__device__ inline WalkLayout desc_walk(const Desc<real> &d) {
    const int *h = d.hdr;
    return walk_layout<real>(h[0], h[6], h[2], h[1], h[5], h[7]);
}

// The walks of move mi of one model by the warps of a block, as many as its shared memory (region bytes
// at smem) holds; next(n), called by lane 0 of each of the n warps, gives the first of its next 16 tasks (none from `end`
// on). scratch: the warp's slab for the points where the cap exceeds the local arrays.
template <class real, class Next>
__device__ __forceinline__ void walk_run(const DevModel<real> &M, const Desc<real> &d, const WalkLayout &W, char *smem,
                                         int region, real *scratch, const int *steps, int nsteps, uint32_t sweep, int mi,
                                         int end, unsigned int &tried, unsigned int &moved, unsigned int &guards,
                                         Next next) {
    real *K = (real *)smem;
    const int n = W.ng + W.nga;
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        bool a = q >= W.ng;
        int j = a ? d.gia[q - W.ng] : d.gi[q];
        real k = M.kc_d[j];
        K[W.kx + q] = mul_rn(M.dt, M.d_mc[j]);
        K[W.ky + q] = mul_rn(mul_rn(M.c_viol, M.dt), add_rn(k, M.kappa0));
        K[W.kak + q] = mul_rn(M.d_avail[j], k);
        K[W.ka + q] = a ? d.gaa[q - W.ng] : d.ga[q];
        K[W.kpos + q] = WalkIndex<real>::put(a ? d.gposa[q - W.ng] : d.gpos[q]);
    }
    for (int q = threadIdx.x; q < W.nl; q += blockDim.x) {
        K[W.la + q] = d.ldf[q];
        K[W.ls + q] = M.ls[d.li[q]];
        K[W.lpa + q] = WalkIndex<real>::put(d.lpa[q]);
        K[W.lpb + q] = WalkIndex<real>::put(d.lpb[q]);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int cb = walk_const_bytes<real>(W), wb = walk_warp_bytes<real>(W);
    const int nw = (region - cb) / wb;
    if (wib >= nw) return;
    real *tv = (real *)(smem + cb + (size_t)wib * wb), *lv = tv + 16 * W.task;
    tv += lane >> 1;
    lv += lane;
    real local[4 * ESM_WALK_PTS];
    const bool loc = M.maxpts <= ESM_WALK_PTS;
    real *pts = loc ? local : scratch + lane;
    SepUnit<real> u{};
    LineWalk<real> S{M, W, K, tv, lv, pts, loc ? 1 : 32, loc ? ESM_WALK_PTS : M.maxpts, u};
    const bool left = lane & 1;
    const int T = M.T;
    while (true) {
        int task0 = 0;
        if (lane == 0) task0 = next(nw);
        task0 = __shfl_sync(0xffffffffu, task0, 0);
        if (task0 >= end) break;
        const int task = task0 + (lane >> 1);
        const bool on = task < end;
        int rep = 0, tau = 0, qs = 0;
        if (on) {
            rep = task % M.R;
            qs = task / M.R;
            tau = steps[qs];
        }
        const int taum = (tau - 1 + T) % T, tau1 = (tau + 1) % T;
        auto ix = [&](int x, int t) -> size_t { return sidx(x, t, rep, T, M.R); };
        // the task's values, by its two lanes in turn; the breakpoints (finalize!, src/local.jl:656),
        // 0 where there is none
        __syncwarp();
        if (on) {
            auto bp = [&](int q, real a, real b) {
                S.T(W.tb + q) = isfinite(a) ? a : real(0);
                S.T(W.tb + q + 1) = isfinite(b) ? b : real(0);
            };
            for (int q = left; q < n; q += 2) {
                real y0 = q < W.ng ? M.g[ix(d.gi[q], tau)] : M.g[ix(d.gia[q - W.ng], taum)], a = K[W.ka + q];
                S.T(W.ty + q) = y0;
                bp(2 * q, (real(0) - y0) / a, (real(1) - y0) / a);
            }
            for (int q = left; q < W.nl; q += 2) {
                real f0 = M.F[ix(d.li[q], tau)], df = K[W.la + q], se = K[W.ls + q];
                S.T(W.tf + q) = f0;
                bp(2 * (n + q), (se - f0) / df, (-se - f0) / df);
            }
            for (int q = left; q < W.nns; q += 2) S.T(W.tr + q) = M.r[ix(d.nds[q], tau)];
            for (int q = left; q < W.nna; q += 2) S.T(W.tr + W.nns + q) = M.r[ix(d.nda[q], taum)];
            if (W.nse) {
                int j = d.si[0];
                real e0 = M.e[ix(j, tau)];
                u.load(M, M.kc_s[j], M.s_hours[j], M.s_qt[j], M.s_etain[j], M.s_etaout[j], M.s_mc[j], d.sa[0], e0,
                       clampr<real>(M.e[ix(j, tau1)], 0, 1), clampr<real>(M.e[ix(j, taum)], 0, 1));
                u.pos = d.spos[0];
                u.posa = d.sposa[0];
                if (!left) bp(2 * (n + W.nl), (real(0) - e0) / u.a, (real(1) - e0) / u.a);
            }
        }
        __syncwarp();
        int np = 0;
        int w = S.walk(on, left ? real(-1) : real(1), &np);
        int wr = __shfl_sync(0xffffffffu, w, lane & ~1), wl = __shfl_sync(0xffffffffu, w, lane | 1);
        // the right walk's outcome counts first
        w = wr != 1 ? wr : wl;
        bool both = on && w == 1;
        double uc = 0, uo = 0;
        if (both) uniform2(M.seed, ESM_TAG_LANE, 2 * (uint32_t)mi, (uint32_t)tau, (uint32_t)rep, sweep, &uc, &uo);
        real t = S.sample(both, left, np, unit_uniform<real>(uc), unit_uniform<real>(uo));
        if (!both) t = 0;
        if (on && !left) {
            if (t != 0) {  // commit (apply_step!, src/local.jl:2507)
                real z, dcs, dca;
                S.eval(t, &z, &dcs, &dca);
                for (int q = 0; q < W.nga; ++q) {
                    real *p = &M.g[ix(d.gia[q], taum)];
                    *p = fma_rn(t, K[W.ka + W.ng + q], *p);
                }
                for (int q = 0; q < W.nna; ++q) M.r[ix(d.nda[q], taum)] = add_rn(S.T(W.tr + W.nns + q), S.L(W.cur + W.nns + q));
                for (int q = 0; q < W.ng; ++q) {
                    real *p = &M.g[ix(d.gi[q], tau)];
                    *p = fma_rn(t, K[W.ka + q], *p);
                }
                if (W.nse) M.e[ix(d.si[0], tau)] = fma_rn(t, u.a, u.e0);
                for (int q = 0; q < d.hdr[8]; ++q) {
                    real *p = &M.theta[ix(d.thn[q], tau)];
                    *p = fma_rn(t, d.tha[q], *p);
                }
                for (int q = 0; q < W.nl; ++q) M.F[ix(d.li[q], tau)] = fma_rn(t, K[W.la + q], S.T(W.tf + q));
                for (int q = 0; q < W.nns; ++q) M.r[ix(d.nds[q], tau)] = add_rn(S.T(W.tr + q), S.L(W.cur + q));
            }
            if (M.mlog && rep < M.mlog_nrep) M.mlog[((size_t)mi * nsteps + qs) * M.mlog_nrep + rep] = (double)t;
            ++tried;
            if (w < 0) ++guards;
            if (t != 0) ++moved;
        }
    }
}

}  // namespace esm
