// lbfgs_group.cuh — the restart reduction and bounded L-BFGS polish of
// pso_fit_single_model (src/parametric.rs:1864-1972; lbfgs_refine,
// :1453-1535: argmin 0.11 LBFGS with memory 7, gradient tolerance 1e-6, cost
// tolerance machine epsilon, 50 iterations, and the MINPACK Moré–Thuente
// line search with ftol 1e-4, gtol 0.9, xtol 1e-10, initial step 1), with
// four polishes per warp.
//
// The bands of the metric's workload hold ~45 observations.  Spread over a
// whole warp, one cost evaluation left most lanes one observation, and the
// work per evaluation that does not scale with the band (the parameters'
// exponentials and gathers, the reductions, the line search's scalar FP64
// arithmetic, which every lane repeated) dominated the polish.  Here each
// group of eight lanes runs its own polish: lane j of a group holds
// component j of every parameter-space vector, and the group's lanes split
// its band's observations (j, j + 8, ...).  One warp instruction of the
// vector algebra or of the line search now serves four polishes.
//
// The polish is written as a state machine whose one suspension point is the
// cost evaluation.  Each round every group evaluates its pending point (the
// warp's lanes together: the same model, each group its own band), then
// advances its own state: the accurate re-check of near-tied restarts, one
// Moré–Thuente step, the L-BFGS update and two-loop direction, or the final
// clamped evaluation.  A group whose polish has ended takes the next band
// from the model's queue; bands are queued longest first, so the groups of a
// warp hold bands of similar length and their observation loops end
// together.
//
// The polish's double-float terms and FP64 line search are long code, and it
// would wait for instructions (measured on GB300, more resident warps at
// different points of it made it slower).  The warps of a block run a round
// in step: a block barrier before and after the evaluation, so that they
// fetch the same code: 0.6 to 0.8 stall cycles an issue instead of 18.7.  1,000
// uneven sources polish in 79 ms in step and in 96 ms without the barriers.
// What bounds it then is the FP64 pipe, 62 % busy at 1,000 sources and 47 % at
// 5,000, and the barrier's wait for the block's slowest warp (4.7 and 6.1
// cycles an issue).  The group's scalar state and the
// per-lane vectors wait in shared memory, leaving the registers to the evaluation.
//
// Where the batch leaves warps free, a band gets a whole warp: four
// observations then go through the term for one fetch of it, and
// add_round_v8 adds them in the eight lanes' order, so the result does not
// depend on the batch.
//
// Arithmetic: the reference's algorithm in FP64 (lbfgs.cuh restates it for
// one thread).  The dot products are sums over the eight lanes by xor 4, 2, 1
// exchanges; the curvature pairs sit in a ring of seven (newest first in the
// two-loop recursion); the observation terms are double-float (ff.cuh,
// models_ff.cuh) with the FP64 term wherever an exponent or the prediction
// could leave FP32's range, summed per lane and then by a reduce-scatter
// over the group's eight lanes.
#pragma once

#include <math.h>

#include "lane_cost.cuh"
#include "lbfgs.cuh"

#ifndef FULL
#define FULL 0xffffffffu
#endif

namespace lcf {

// A group's scalar state, in shared memory during the cost evaluation, which is
// bound by latency and so by the warps resident per SM: kept out of the
// registers there.  Each lane of the group works on a copy of its own and all
// write the same values back, with a barrier between the last read and the
// first write: no lane may read what another has moved on, converged or not.
// LbScalars, the polish and its line search, is read and written every round,
// the band and the choice of the restart only where they change.  (One source's
// polish 6.5 ms, 1,000 sources' 86; with the scalars updated in place by all
// lanes the same.)
struct alignas(16) LbScalars {
    double f, prev_f, best_f;
    double dginit, dgtest, finit, width, width1, stx, fx, dgx, sty, fy, dgy, stp, stmin, stmax;
    int cm, head, it, evals, fp64_evals, infoc, ls_iter;
    bool brackt, stage1;
};
struct LbBand {
    double t_first, t_last, inv_nd;
    int64_t off;
    int n, b;
};
struct LbRestarts {
    double best_c, acc[3];
    int acc_mask, nc, best_r;
};
struct LbCounts {
    unsigned long long pol, it, ev, obs, fp64;
};

// Per warp, in shared memory: the curvature pairs, 1 / (y.s) and the
// two-loop coefficients, [ring slot][lane], and the four groups' states.
struct LbWarpShared {
    double S[7][32], Y[7][32], rho[7][32], alpha[7][32];
    double V[7][32];  // per lane: x, g, search direction, trial point and gradient, best point, swarm point
    LbScalars st[4];
    LbBand band[4];
    LbRestarts rs[4];
    LbCounts counts[4];  // written by the group's first lane
};

// a.b over the eight lanes of this lane's group (mask gm)
__device__ __forceinline__ double gdot(double a, double b, unsigned gm) {
    double v = a * b;
    v += __shfl_xor_sync(gm, v, 4);
    v += __shfl_xor_sync(gm, v, 2);
    v += __shfl_xor_sync(gm, v, 1);
    return v;
}

__device__ __forceinline__ ff shfl_xor_ff_m(ff v, int m, unsigned gm) {
    return ffm(__shfl_xor_sync(gm, v.hi, m), __shfl_xor_sync(gm, v.lo, m));
}

// Reduce-scatter of eight per-lane values over a group of eight lanes
// (4 + 2 + 1 exchanges): lane j returns the group's total of v[j].
__device__ __forceinline__ ff group_rs8_ff(const ff* v, unsigned gm) {
    const int lane = threadIdx.x & 31;
    const bool b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
    ff a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = ff_add(b2 ? v[4 + i] : v[i], shfl_xor_ff_m(b2 ? v[i] : v[4 + i], 4, gm));
#pragma unroll
    for (int i = 0; i < 2; i++) b[i] = ff_add(b1 ? a[2 + i] : a[i], shfl_xor_ff_m(b1 ? a[i] : a[2 + i], 2, gm));
    return ff_add(b0 ? b[1] : b[0], shfl_xor_ff_m(b0 ? b[0] : b[1], 1, gm));
}
__device__ __forceinline__ double group_rs8(const double* v, unsigned gm) {
    const int lane = threadIdx.x & 31;
    const bool b2 = lane & 4, b1 = lane & 2, b0 = lane & 1;
    double a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = (b2 ? v[4 + i] : v[i]) + __shfl_xor_sync(gm, b2 ? v[i] : v[4 + i], 4);
#pragma unroll
    for (int i = 0; i < 2; i++) b[i] = (b1 ? a[2 + i] : a[i]) + __shfl_xor_sync(gm, b1 ? a[i] : a[2 + i], 2);
    return (b0 ? b[1] : b[0]) + __shfl_xor_sync(gm, b0 ? b[0] : b[1], 1);
}

// A group's band: where its observations start, their count (0 for a group
// without a polish), the time span, 1 / n and this lane's box bounds.
struct GroupBand {
    int64_t off;
    int n;
    double t_first, t_last, inv_nd, lo_j, hi_j;
};

// The observation terms in FP64 (lb_obs_term) for the FP32-range fallback:
// this lane's share of the group's band, v = {nll, gradient partials}.
template <int MODEL, int G>
__device__ __noinline__ int group_fp64_terms(const double* t, const double* flux, const double* var, const double* uf,
                                             const uint8_t* up, int n, const double* q, const double* ep,
                                             const double* rp, double se2, bool want_grad, double* v) {
    int nonfinite = 0;
    Model64 mod;
    mod.init_pre(MODEL, q, ep, rp);
    double nll = 0.0, gl[MAXP];
#pragma unroll
    for (int k = 0; k < MAXP; k++) gl[k] = 0.0;
    for (int i = (int)(threadIdx.x & (G - 1)); i < n; i += G)
        lb_obs_term<MODEL>(mod, t[i], var[i], flux[i], up[i], uf[i], se2, want_grad, nll, gl, nonfinite);
    v[0] = nll;
#pragma unroll
    for (int k = 0; k < MAXP; k++) v[1 + k] = gl[k];
    return nonfinite;
}

// The eight sums of a band that a whole warp evaluates in the eight-lane
// order: lane v + 8 u holds the term vector v8 of the (4 r + u)-th observation
// of sum lane v in round r.  The four lanes of a sum lane trade components
// (xor 16, then xor 8), so that lane v + 8 u ends with components 2 u and
// 2 u + 1 of all four observations, and adds them in the observations' order:
// the bits of eight lanes that take four observations each, one after another.
__device__ __forceinline__ void add_round_v8(const ff* v8, ff& s0, ff& s1) {
    const int lane = threadIdx.x & 31;
    const bool b4 = lane & 16, b3 = lane & 8;
    ff own[4], oth[4];  // this lane's and its xor-16 partner's components 4 b4 .. 4 b4 + 3
#pragma unroll
    for (int i = 0; i < 4; i++) {
        own[i] = b4 ? v8[4 + i] : v8[i];
        oth[i] = shfl_xor_ff_m(b4 ? v8[i] : v8[4 + i], 16, FULL);
    }
    ff p[2][4];  // [component][observation u]
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const ff a = b3 ? own[2 + c] : own[c], b = b3 ? oth[2 + c] : oth[c];
        const ff ra = shfl_xor_ff_m(b3 ? own[c] : own[2 + c], 8, FULL);
        const ff rb = shfl_xor_ff_m(b3 ? oth[c] : oth[2 + c], 8, FULL);
        // observation u of lane bits (b4, b3): own a = (b4, b3), b = (!b4, b3), ra = (b4, !b3), rb = (!b4, !b3)
        const ff x0 = b4 ? b : a, x2 = b4 ? a : b;      // u with bit 0 = b3
        const ff y0 = b4 ? rb : ra, y2 = b4 ? ra : rb;  // u with bit 0 = !b3
        p[c][0] = b3 ? y0 : x0;
        p[c][1] = b3 ? x0 : y0;
        p[c][2] = b3 ? y2 : x2;
        p[c][3] = b3 ? x2 : y2;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        s0 = ff_add(s0, p[0][u]);
        s1 = ff_add(s1, p[1][u]);
    }
}

// Cost and projected gradient of the bounded problem (BoundedPsoCost,
// src/parametric.rs:1500-1535) at the point whose component j is xj in lane
// j of each group: PsoCost::cost_from_slice with the population prior and
// the Villar constraint, and PsoCost::gradient.  G lanes a group (8, or 32:
// the whole warp, whose four sets of eight lanes hold the same vectors); the
// observations are summed in the order of V lanes (8 or 32).
// Warp-collective (every lane calls it; a group with B.n == 0 evaluates
// nothing of use).  Returns 1 when the group's terms ran in FP64.
template <int MODEL, int G, int V>
__device__ __forceinline__ int group_cost_grad(const DeviceBatch& d, const GroupBand& B, double xj, bool want_grad,
                                               double& fo, double& gj) {
    constexpr int np = n_params_of(MODEL), se = se_idx_of(MODEL);
    const int lane = threadIdx.x & 31, j = lane & 7, g0 = lane & (32 - G);
    const unsigned gm = G == 32 ? FULL : 0xffu << g0;
    // lane j forms e^(+-p_j) of its own component in double-float; the group's
    // vectors are gathered by shuffles
    const double qj = fmin(fmax(xj, B.lo_j), B.hi_j);
    const ff qjf = ff_from(qj);
    const ff ejf = ff_exp(qjf), rjf = ff_exp(ff_neg(qjf));
    double q[MAXP];
    ff ef[MAXP], rf[MAXP];
#pragma unroll
    for (int k = 0; k < MAXP; k++) {
        q[k] = k < np ? __shfl_sync(FULL, qj, g0 + k) : 0.0;
        ef[k] = k < np ? shfl_ff(ejf, g0 + k) : ffm(1.0f, 0.0f);
        rf[k] = k < np ? shfl_ff(rjf, g0 + k) : ffm(1.0f, 0.0f);
    }
    const ff se2f = ff_sqr(ef[se]);  // sigma_extra = exp(p[se]), squared
    bool constrained = false;
    double f = 0.0;
    if (MODEL == VILLAR) {
        // Villar constraint of PsoCost (src/parametric.rs:1305-1318):
        // beta = p1, gamma = e^p2, tr = e^p4, tf = e^p5
        const ff beta = ff_from(q[1]), gamma = ef[2], itr = rf[4], tf = ef[5];
        const ff one = ffm(1.0f, 0.0f), zero = ffm(0.0f, 0.0f);
        const ff c1 = ff_sub(ff_mul(gamma, beta), one);
        const ff c2 = ff_sub(ff_mul(ff_exp(ff_neg(ff_mul(gamma, itr))), ff_sub(ff_mul(tf, itr), one)), one);
        const ff c3 = ff_add(ff_sub(ff_mul(beta, tf), one), ff_mul(beta, gamma));
        const ff cc = ff_add(ff_add(c1.hi > 0.0f ? c1 : zero, c2.hi > 0.0f ? c2 : zero), c3.hi > 0.0f ? c3 : zero);
        if (cc.hi > 0.0f) {
            f = 1e12 + 10000.0 * ff_to(cc);
            constrained = true;
        }
    }
    // population prior, one component per lane
    const double zj = j < np ? (qj - c_pop_c[MODEL][j]) * c_pop_iw[MODEL][j] : 0.0;
    const double prior = gdot(0.5 * zj, zj, FULL);
    int nonfinite = 0, fp64 = 0;
    double nsum = 0.0, gs = 0.0;
    // double-float terms unless an exponent or the prediction could leave
    // FP32's range over the band's span, or an upper limit's gradient ratio
    // does (a group-uniform decision)
    const double t0 = q[t0_idx_of(MODEL)];
    bool in_ff = B.n == 0 || ff_range_ok<MODEL>(q, rf, B.t_first - t0, B.t_last - t0);
    if (in_ff) {
        FfModel<MODEL> fm;
        fm.init(q, ef, rf);
        ff nf = ffm(0.0f, 0.0f), gf[MAXP];
#pragma unroll
        for (int k = 0; k < MAXP; k++) gf[k] = ffm(0.0f, 0.0f);
        int redo = 0;
        const float4* fa = d.ffa + B.off;
        const float2* fb = d.ffb + B.off;
        ff s0 = ffm(0.0f, 0.0f), s1 = ffm(0.0f, 0.0f);
        if constexpr (G == V) {
            for (int i = lane & (G - 1); i < B.n; i += G)
                ff_obs_term<MODEL>(fm, fa[i], fb[i], se2f, want_grad, nf, gf, nonfinite, redo);
        } else {
            for (int i0 = 0; i0 < B.n; i0 += 32) {
                ff t[8];
#pragma unroll
                for (int k = 0; k < 8; k++) t[k] = ffm(0.0f, 0.0f);
                if (i0 + lane < B.n)
                    ff_obs_term<MODEL>(fm, fa[i0 + lane], fb[i0 + lane], se2f, want_grad, t[0], t + 1, nonfinite, redo);
                add_round_v8(t, s0, s1);
            }
        }
        in_ff = __ballot_sync(gm, redo) == 0u;
        if (in_ff) {
            nonfinite = __ballot_sync(gm, nonfinite) != 0u;
            const ff v[8] = {nf, gf[0], gf[1], gf[2], gf[3], gf[4], gf[5], gf[6]};
            if (G != V) {
                // lane v + 8 u: the totals of components 2 u, 2 u + 1, summed as
                // group_rs8_ff does (ff_add commutes)
#pragma unroll
                for (int k = 4; k; k >>= 1) {
                    s0 = ff_add(s0, shfl_xor_ff_m(s0, k, FULL));
                    s1 = ff_add(s1, shfl_xor_ff_m(s1, k, FULL));
                }
                const double t0s = ff_to(s0), t1s = ff_to(s1);
                nsum = __shfl_sync(FULL, t0s, 0);
                const int src = 8 * (((j + 1) & 7) >> 1);
                const double ge = __shfl_sync(FULL, t0s, src), go = __shfl_sync(FULL, t1s, src);
                gs = ((j + 1) & 1) ? go : ge;
            } else if (G == 32) {  // lane l: the warp's total of v[(l >> 2) & 7]
                const double tot = ff_to(reduce_scatter8_ff(v));
                nsum = __shfl_sync(FULL, tot, 0);
                gs = __shfl_sync(FULL, tot, (4 * (1 + j)) & 31);
            } else {  // lane j: the group's total of v[j]
                const double tot = ff_to(group_rs8_ff(v, gm));
                nsum = __shfl_sync(gm, tot, g0);
                gs = __shfl_sync(gm, tot, g0 + ((j + 1) & 7));
            }
        }
    }
    if (!in_ff) {
        fp64 = 1;
        double ep[MAXP], rp[MAXP], v[8];
#pragma unroll
        for (int k = 0; k < MAXP; k++) {
            ep[k] = ff_to(ef[k]);
            rp[k] = ff_to(rf[k]);
        }
        const double se2 = ep[se] * ep[se];
        const int64_t o = B.off;
        // (a warp summing in the eight-lane order: each set of eight lanes does it all)
        const int nf64 = group_fp64_terms<MODEL, V>(d.t64 + o, d.f64 + o, d.var64 + o, d.uf64 + o, d.up + o, B.n, q,
                                                    ep, rp, se2, want_grad, v);
        nonfinite = __ballot_sync(gm, nf64) != 0u;
        if (V == 32) {
            const double tot = reduce_scatter8(v);
            nsum = __shfl_sync(FULL, tot, 0);
            gs = __shfl_sync(FULL, tot, (4 * (1 + j)) & 31);
        } else {
            const double tot = group_rs8(v, gm);
            nsum = __shfl_sync(gm, tot, g0);
            gs = __shfl_sync(gm, tot, g0 + ((j + 1) & 7));
        }
    }
    if (!constrained) f = nonfinite ? BIG_COST : (nsum + prior * B.inv_nd) * B.inv_nd;
    fo = f;
    gj = (nonfinite || j >= np) ? 0.0 : gs * B.inv_nd;
    if ((xj <= B.lo_j && gj > 0.0) || (xj >= B.hi_j && gj < 0.0)) gj = 0.0;
    return fp64;
}

// Two swarm result costs closer than the FP32 estimate's error (3e-5 of the
// reference value; the special values 1e99, +inf and the Villar constraint's
// 1e12 + 1e4 c compare as they are).
__device__ __forceinline__ bool swarm_cost_tie(double a, double ref) {
    if (!(fabs(ref) < 1e11) || !(fabs(a) < 1e11)) return a == ref;
    return fabs(a - ref) <= 3e-5 * fabs(ref);
}

// A polish's phases: the point a group evaluates next, and what it does with
// the result.
enum LbPhase : int {
    LB_FETCH = 0,  // take a band from the queue
    LB_ACC,        // accurate cost of a restart's swarm result (no gradient)
    LB_START,      // cost and gradient at the chosen restart's parameters
    LB_LS,         // a line-search trial point (with gradient)
    LB_TAIL,       // the line search's 100 steps ran out: cost at its last point
    LB_FINAL,      // cost at the clamped best point
    LB_DONE        // the queue is empty
};

// Polishes the queued bands of MODEL with G lanes a band (8: four bands a
// warp; 32: one), summing in the order of V lanes: d.polish_order[i] for the indices i in [lo, hi) that this
// warp's groups take from the queue counter `next`, the block's warps running
// each round in step.
// Out of line: the instantiations of a model then take their registers separately.
#ifndef LCF_LB_QUEUE_ATTR
#define LCF_LB_QUEUE_ATTR __noinline__
#endif
template <int MODEL, int G, int V>
__device__ LCF_LB_QUEUE_ATTR void polish_queue(const DeviceBatch& d, LbWarpShared& sh, int lo, int hi, int* next) {
    constexpr int np = n_params_of(MODEL), t0i = t0_idx_of(MODEL), M = 7, MAXIT = 50;
    const double ftol = 1e-4, gtol = 0.9, xtol = 1e-10, xtrapf = 4.0, stpmin = 0.0, stpmax = INFINITY;
    const double tol_grad = 1e-6, tol_cost = 2.220446049250313e-16;
    const int lane = threadIdx.x & 31, j = lane & 7, gl = lane & (G - 1), g0 = lane & (32 - G);
    const unsigned gm = G == 32 ? FULL : 0xffu << g0;

    int phase = LB_FETCH;
    // this lane's components: box bounds, the swarm's parameter, the point
    // evaluated next, the iterate, its gradient, the search direction, the
    // trial point and its gradient, the best point
    double lo_j = 0.0, hi_j = 0.0, xe = 0.0;
    double &x = sh.V[0][lane], &g = sh.V[1][lane], &dv = sh.V[2][lane], &xo = sh.V[3][lane], &go = sh.V[4][lane],
           &bx = sh.V[5][lane], &pj = sh.V[6][lane];
    x = g = dv = xo = go = bx = pj = 0.0;
    // the group's scalars: this lane's copy
    LbScalars st;
    // the polish
    double &f = st.f, &prev_f = st.prev_f, &best_f = st.best_f;
    int &cm = st.cm, &head = st.head, &it = st.it, &evals = st.evals, &fp64_evals = st.fp64_evals;
    // the line search
    double &dginit = st.dginit, &dgtest = st.dgtest, &finit = st.finit, &width = st.width, &width1 = st.width1;
    double &stx = st.stx, &fx = st.fx, &dgx = st.dgx, &sty = st.sty, &fy = st.fy, &dgy = st.dgy;
    double &stp = st.stp, &stmin = st.stmin, &stmax = st.stmax;
    int &infoc = st.infoc, &ls_iter = st.ls_iter;
    bool &brackt = st.brackt, &stage1 = st.stage1;
    f = 0.0;
    prev_f = best_f = INFINITY;
    cm = it = evals = fp64_evals = 0;
    head = M - 1;
    dginit = dgtest = finit = width = width1 = stx = fx = dgx = sty = fy = dgy = stp = stmin = stmax = 0.0;
    infoc = 1;
    ls_iter = 0;
    brackt = false;
    stage1 = true;
    LbBand& band = sh.band[lane / G];
    LbRestarts& rs = sh.rs[lane / G];
    LbCounts& counts = sh.counts[lane / G];
    band = {0.0, 0.0, 1.0, 0, 0, 0};
    counts = {0, 0, 0, 0, 0};

    auto restarts = [&](int b) { return d.pso_res + (size_t)(b * 8 + MODEL) * 3; };
    auto finish = [&](int b, double cost) {
        ModelFit& F = d.fits[b * 8 + MODEL];
        if (gl == 0) F.cost = cost;
        if (gl < MAXP) F.params[gl] = gl < np ? pj : NAN;
        phase = LB_FETCH;
    };
    auto converged = [&]() { return lb_sqrt(gdot(g, g, gm)) < tol_grad || fabs(prev_f - f) < tol_cost; };

    while (true) {
        // groups without a polish take bands until one needs polishing
        while (phase == LB_FETCH) {
            int i = 0;
            if (gl == 0) i = lo + atomicAdd(next, 1);
            i = __shfl_sync(gm, i, g0);
            if (i >= hi) {
                phase = LB_DONE;
                break;
            }
            const int b = d.polish_order[i];
            const BandStats bs = d.stats[b];
            if (!bs.valid) continue;
            const PsoResult* R = restarts(b);
            if (R[0].iters < 0) continue;  // this model was not fitted for this band
            double best_c = INFINITY;
            int best_r = -1;
            for (int r = 0; r < 3; r++)
                if (R[r].iters >= 0 && R[r].cost < best_c) { best_c = R[r].cost; best_r = r; }
            pj = (best_r >= 0 && j < np) ? pso_param(R[best_r], j) : 0.0;
            if (MODEL == METZGER || best_r < 0) {  // MetzgerKN keeps its swarm result
                finish(b, best_c);
                continue;
            }
            lo_j = j < np ? c_lo[MODEL][j] : 0.0;
            hi_j = j < np ? c_hi[MODEL][j] : 0.0;
            const double t0_lo = fmax(bs.t_first - 30.0, c_lo[MODEL][t0i]);
            const double t0_hi = fmin(bs.t_peak + 10.0, c_hi[MODEL][t0i]);
            if (j == t0i && t0_lo < t0_hi) { lo_j = t0_lo; hi_j = t0_hi; }
            // the restarts' swarms report FP32 estimates of their best costs:
            // the chosen restart's cost, and the choice among restarts within
            // the estimates' error of it, are settled on accurate costs (the
            // first strict minimum, as the reference's restart loop)
            int acc_mask = 0;
            for (int r = 0; r < 3; r++)
                if (R[r].iters >= 0 && (r == best_r || swarm_cost_tie(R[r].cost, best_c))) acc_mask |= 1 << r;
            __syncwarp(gm);  // the last band's state is read
            band = {bs.t_first, bs.t_last, 1.0 / (double)max(bs.n, 1), bs.off, bs.n, b};
            rs = {best_c, {INFINITY, INFINITY, INFINITY}, acc_mask, __popc(acc_mask), best_r};
            __syncwarp(gm);
            evals = 0;
            fp64_evals = 0;
            it = 0;
            xe = j < np ? pso_param(R[__ffs(acc_mask) - 1], j) : 0.0;
            phase = LB_ACC;
        }
        // in step, the block's warps evaluate together (see the header): a
        // barrier before and after the evaluation
        const bool active = phase != LB_DONE;
        if (!__syncthreads_or(active)) break;
        if constexpr (MODEL == METZGER) continue;  // never polished (every group is done)
        const bool want_grad = phase == LB_START || phase == LB_LS;
        GroupBand B;
        B.off = band.off;
        B.n = active ? band.n : 0;
        B.t_first = band.t_first;
        B.t_last = band.t_last;
        B.inv_nd = band.inv_nd;
        B.lo_j = lo_j;
        B.hi_j = hi_j;
        double fe = 0.0, ge = 0.0;
        int used64 = 0;
        sh.st[lane / G] = st;
        if (__any_sync(FULL, active)) used64 = group_cost_grad<MODEL, G, V>(d, B, xe, want_grad, fe, ge);
        __syncthreads();
        st = sh.st[lane / G];
        __syncwarp(gm);  // read by the whole group before the next round's write
        if (!active) continue;
        fp64_evals += used64;
        // the transition of this group's phase; the steps shared by several
        // phases (accepting a line-search point, a new direction, the next
        // trial point, the end of the polish) run once each, below the switch
        bool do_accept = false, do_begin = false, do_trial = false, do_end = false;
        double fnew = 0.0, end_cost = 0.0;
        switch (phase) {
            case LB_ACC: {
                LbRestarts q = rs;
                __syncwarp(gm);
                const int r = __ffs(q.acc_mask) - 1;
                if (r == 0) q.acc[0] = fe;
                else if (r == 1) q.acc[1] = fe;
                else q.acc[2] = fe;
                q.acc_mask &= q.acc_mask - 1;
                const PsoResult* R = restarts(band.b);
                if (q.acc_mask) {
                    rs = q;
                    xe = j < np ? pso_param(R[__ffs(q.acc_mask) - 1], j) : 0.0;
                    break;
                }
                if (q.nc > 1) {
                    q.best_r = -1;
                    q.best_c = INFINITY;
                    if (q.acc[0] < q.best_c) { q.best_c = q.acc[0]; q.best_r = 0; }
                    if (q.acc[1] < q.best_c) { q.best_c = q.acc[1]; q.best_r = 1; }
                    if (q.acc[2] < q.best_c) { q.best_c = q.acc[2]; q.best_r = 2; }
                    if (q.best_r < 0) q.best_r = 0;
                    pj = j < np ? pso_param(R[q.best_r], j) : 0.0;
                } else {
                    q.best_c = q.best_r == 0 ? q.acc[0] : q.best_r == 1 ? q.acc[1] : q.acc[2];
                }
                rs = q;
                x = pj;
                xe = x;
                phase = LB_START;
                break;
            }
            case LB_START:
                evals++;
                f = fe;
                g = ge;
                best_f = INFINITY;
                prev_f = INFINITY;
                bx = x;
                if (f < best_f) { best_f = f; bx = x; }
                cm = 0;
                head = M - 1;
                if (converged() || it >= MAXIT) {
                    xe = fmin(fmax(bx, lo_j), hi_j);
                    phase = LB_FINAL;
                } else {
                    do_begin = true;
                }
                break;
            case LB_LS: {
                evals++;
                const double fl = fe;
                go = ge;
                const double dg = gdot(go, dv, gm);
                const double ftest1 = finit + stp * dgtest;
                int info = 0;
                if ((brackt && (stp <= stmin || stp >= stmax)) || infoc == 0) info = 6;
                if (stp == stpmax && fl <= ftest1 && dg <= dgtest) info = 5;
                if (stp == stpmin && (fl > ftest1 || dg >= dgtest)) info = 4;
                if (brackt && stmax - stmin <= xtol * stmax) info = 2;
                if (fl <= ftest1 && fabs(dg) <= gtol * (-dginit)) info = 1;
                if (info != 0) {
                    fnew = fl;
                    do_accept = true;
                    break;
                }
                if (stage1 && fl <= ftest1 && dg >= fmin(ftol, gtol) * dginit) stage1 = false;
                const bool modified = stage1 && fl <= fx && fl > ftest1;
                // cstep on the modified function psi (MINPACK) or on f itself
                double fxa = fx, fya = fy, dgxa = dgx, dgya = dgy, fpa = fl, dpa = dg;
                if (modified) {
                    fpa = fl - stp * dgtest;
                    fxa = fx - stx * dgtest;
                    fya = fy - sty * dgtest;
                    dpa = dg - dgtest;
                    dgxa = dgx - dgtest;
                    dgya = dgy - dgtest;
                }
                // (copies: a reference into st would keep it out of the registers)
                double stxa = stx, stya = sty, stpa = stp;
                bool bracketed = brackt;
                infoc = lb_cstep(stxa, fxa, dgxa, stya, fya, dgya, stpa, fpa, dpa, bracketed, stmin, stmax);
                stx = stxa;
                sty = stya;
                stp = stpa;
                brackt = bracketed;
                if (modified) {
                    fx = fxa + stx * dgtest;
                    fy = fya + sty * dgtest;
                    dgx = dgxa + dgtest;
                    dgy = dgya + dgtest;
                } else {
                    fx = fxa;
                    fy = fya;
                    dgx = dgxa;
                    dgy = dgya;
                }
                if (brackt) {
                    if (fabs(sty - stx) >= 0.66 * width1) stp = stx + 0.5 * (sty - stx);
                    width1 = width;
                    width = fabs(sty - stx);
                }
                if (++ls_iter == 100) {
                    xe = xo;  // argmin evaluates the last trial point once more
                    phase = LB_TAIL;
                } else {
                    do_trial = true;
                }
                break;
            }
            case LB_TAIL:
                evals++;
                fnew = fe;  // with the last trial's gradient
                do_accept = true;
                break;
            case LB_FINAL:
                evals++;
                end_cost = rs.best_c;
                if (fe < end_cost && isfinite(fe)) {
                    pj = xe;
                    end_cost = fe;
                }
                do_end = true;
                break;
            default: break;
        }
        if (do_accept) {  // the line search accepted (xo, fnew, go)
            const double sj = xo - x, yj = go - g;
            head = head == M - 1 ? 0 : head + 1;
            sh.S[head][lane] = sj;
            sh.Y[head][lane] = yj;
            sh.rho[head][lane] = lb_div(1.0, gdot(yj, sj, gm));
            cm = cm < M ? cm + 1 : M;
            x = xo;
            g = go;
            prev_f = f;
            f = fnew;
            if (f < best_f) { best_f = f; bx = x; }
            it++;
            if (converged() || it >= MAXIT) {
                xe = fmin(fmax(bx, lo_j), hi_j);
                phase = LB_FINAL;
            } else {
                do_begin = true;
            }
        }
        if (do_begin) {  // an L-BFGS iteration: two-loop direction, line search start
            double gamma = 1.0;
            if (cm > 0) {
                const double sn = sh.S[head][lane], yn = sh.Y[head][lane];
                gamma = lb_div(gdot(sn, yn, gm), gdot(yn, yn, gm));
            }
            double q = g;
            int s = head;
#pragma unroll 1
            for (int k = 0; k < cm; k++) {
                const double a = sh.rho[s][lane] * gdot(sh.S[s][lane], q, gm);
                sh.alpha[s][lane] = a;
                q -= sh.Y[s][lane] * a;
                s = s == 0 ? M - 1 : s - 1;
            }
            double r = q * gamma;
#pragma unroll 1
            for (int k = cm - 1; k >= 0; k--) {
                s = s == M - 1 ? 0 : s + 1;
                const double beta = gdot(sh.Y[s][lane], r, gm) * sh.rho[s][lane];
                r += sh.S[s][lane] * (sh.alpha[s][lane] - beta);
            }
            dv = -r;
            dginit = gdot(g, dv, gm);
            if (dginit >= 0.0) {  // not a descent direction: argmin stops with an error
                end_cost = rs.best_c;
                do_end = true;
            } else {
                brackt = false;
                stage1 = true;
                infoc = 1;
                finit = f;
                dgtest = ftol * dginit;
                width = stpmax - stpmin;
                width1 = 2.0 * width;
                stx = 0.0; fx = finit; dgx = dginit;
                sty = 0.0; fy = finit; dgy = dginit;
                stp = 1.0;
                ls_iter = 0;
                phase = LB_LS;
                do_trial = true;
            }
        }
        if (do_trial) {  // the top of a line-search step: its trial point
            if (brackt) {
                stmin = fmin(stx, sty);
                stmax = fmax(stx, sty);
            } else {
                stmin = stx;
                stmax = stp + xtrapf * (stp - stx);
            }
            stp = fmax(stp, stpmin);
            stp = fmin(stp, stpmax);
            if ((brackt && (stp <= stmin || stp >= stmax)) || infoc == 0 || (brackt && stmax - stmin <= xtol * stmax))
                stp = stx;
            xo = x + stp * dv;
            xe = xo;
        }
        if (do_end) {
            if (gl == 0) {
                counts.pol++;
                counts.it += (unsigned long long)it;
                counts.ev += (unsigned long long)evals;
                counts.obs += (unsigned long long)evals * (unsigned long long)band.n;
                counts.fp64 += (unsigned long long)fp64_evals * (unsigned long long)band.n;
            }
            finish(band.b, end_cost);
        }
    }
    // the work counters, summed over the warp's groups
    __syncwarp();
    unsigned long long c_pol = counts.pol, c_it = counts.it, c_ev = counts.ev, c_obs = counts.obs, c_fp64 = counts.fp64;
    __syncwarp();
#pragma unroll
    for (int m = G; m < 32; m <<= 1) {
        c_pol += __shfl_xor_sync(FULL, c_pol, m);
        c_it += __shfl_xor_sync(FULL, c_it, m);
        c_ev += __shfl_xor_sync(FULL, c_ev, m);
        c_obs += __shfl_xor_sync(FULL, c_obs, m);
        c_fp64 += __shfl_xor_sync(FULL, c_fp64, m);
    }
    if (lane == 0 && c_pol) {
        atomicAdd(&d.ctr->lb_polishes, c_pol);
        atomicAdd(&d.ctr->lb_iters, c_it);
        atomicAdd(&d.ctr->lb_evals, c_ev);
        atomicAdd(&d.ctr->lb_obs_evals, c_obs);
        atomicAdd(&d.ctr->lb_obs_evals_by_model[MODEL], c_obs);
        if (c_fp64) atomicAdd(&d.ctr->lb_fp64_obs_evals_by_model[MODEL], c_fp64);
    }
}

}  // namespace lcf
