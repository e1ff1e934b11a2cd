// joint.cu — the joint multi-band Villar fit (fit_parametric_multiband,
// src/parametric.rs:3815-4131) that fit_parametric uses for sources with two
// or more bands when fit_all_models is false (:3742-3761).
//
// A persistent grid of teams (one block, or a cluster of four) takes
// (source, restart) tasks: 200 particles search the 7 * n_bands joint space
// (the most populated band's Villar parameters, then per-band offsets) with
// the reference's PSO (200 particles, 1500 iterations, stall 60; seeds 42 /
// 137 / 271, restart 1 seeded).  The source's bands are staged in shared
// memory; positions, velocities and personal bests are double-float pairs in
// the team's global slice, column-major (parameter j of particle p at
// [j * 200 + p]).
// The reference's asynchronous global best (each particle moves with the
// best after the particles before it) is reproduced by speculative rounds,
// as in the per-band swarm: the particles from `start` on move with the
// current best and are evaluated; the first one that improves the best is
// accepted with those before it, and the rest are recomputed (1.2 to 1.4
// rounds an iteration).  Costs are FP32 evaluations of the reference's
// band-balanced cost (Villar constraint on every band, 1e99 for a non-finite
// prediction, population prior on the reference band and the relative priors
// of de Soto et al. on the offsets) with double-float band sums.
//
// joint_pick_kernel then writes each band's Villar parameters (reference +
// offset) into the per-band outputs, after which the per-band SVI / Laplace,
// refinements, magnitude chi2 and MultiBazin stages run unchanged.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "ff.cuh"
#include "lcf_internal.cuh"
#include "models_f32.cuh"

namespace lcf {

namespace cg = cooperative_groups;

#define FULL 0xffffffffu

constexpr int JP = 200;          // particles (src/parametric.rs:3951-3956)
constexpr int J_MAXIT = 1500;
constexpr int J_STALL = 60;
constexpr int J_THREADS = 448;   // of a block
constexpr int J_WARPS = J_THREADS / 32;

// de Soto et al. relative priors of the offsets, src/parametric.rs:3771-3786
static __device__ __constant__ float c_rel_mean[7] = {-0.015f * 2.302585093f, -0.001f, -0.095f * 2.302585093f,
                                                      -1.181f, -0.195f * 2.302585093f, -0.323f * 2.302585093f,
                                                      -0.025f * 2.302585093f};
static __device__ __constant__ float c_rel_sigma[7] = {0.08f * 2.302585093f, 0.008f, 0.25f * 2.302585093f, 1.5f,
                                                       0.35f * 2.302585093f, 0.25f * 2.302585093f,
                                                       0.30f * 2.302585093f};

// the same in FP64 for the box and the seed particle (as the reference
// computes them)
static __device__ __constant__ double c_rel_mean64[7] = {-0.015 * 2.302585092994045684, -0.001,
                                                         -0.095 * 2.302585092994045684, -1.181,
                                                         -0.195 * 2.302585092994045684, -0.323 * 2.302585092994045684,
                                                         -0.025 * 2.302585092994045684};
static __device__ __constant__ double c_rel_sigma64[7] = {0.08 * 2.302585092994045684, 0.008,
                                                          0.25 * 2.302585092994045684, 1.5,
                                                          0.35 * 2.302585092994045684, 0.25 * 2.302585092994045684,
                                                          0.30 * 2.302585092994045684};

struct JointBands {
    int nb;                 // bands in rank order
    int n[J_MAX_BANDS];     // observations per band
    int off[J_MAX_BANDS];   // first observation in the staged records
    int n_total;
    // the band balancing (n_total / nb) / n[b] and 1 / max(n_total, 1),
    // formed once per task: the FP64 divisions of the reference's cost
    // (src/parametric.rs:3815-4131) become multiplications by double-float
    // pairs, which move the cost by ~1e-14, far below its FP32 evaluation's
    // ~1e-7
    ff wf[J_MAX_BANDS];
    ff inv_total_f;
};

// The joint cost of one particle (column p of the position pairs xs),
// evaluated by T consecutive lanes (r = 0 .. T - 1) of a warp; every lane of
// the warp calls it, `live` marks the lanes that have a particle.  Lane r
// evaluates observations r, r + T, ...; the terms are then added in two Kahan
// chains, even and odd observations, whatever T is: each lane adds the terms
// of its parity in the order of the observations, taking them from the lanes
// that evaluated them.  The cost's bits therefore do not depend on T.
__device__ double joint_cost(const JointBands& jb, const float4* obs, const float2* xs, int p, int T, int r, bool live) {
    const int lane = threadIdx.x & 31, h = r & 1, from = (lane & ~(T - 1)) + h;
    double cost = 0.0;
    bool open = live;  // the cost is not decided yet
    float ref[7];
    if (live)
#pragma unroll
        for (int j = 0; j < 7; j++) ref[j] = xs[j * JP + p].x;
    else
#pragma unroll
        for (int j = 0; j < 7; j++) ref[j] = 0.0f;
    {
        float c = VillarF::constraint_swarm(ref);
        if (open && c > 0.0f) { cost = 1e12 + 10000.0 * (double)c; open = false; }
    }
    // the band sums as double-float pairs: ~1e-14 relative, far below the FP32
    // terms' own error, on the FP32 pipe instead of FP64's 1/64 rate; ff_add
    // is commutative, so both parities' lanes form the same cost
    ff balanced = ffm(0.0f, 0.0f);
    for (int b = 0; b < jb.nb; b++) {
        float bp[7];
#pragma unroll
        for (int j = 0; j < 7; j++) bp[j] = b == 0 || !live ? ref[j] : ref[j] + xs[(7 * b + j) * JP + p].x;
        if (b > 0) {
            float c = VillarF::constraint_swarm(bp);
            if (open && c > 0.0f) { cost = 1e12 + 10000.0 * (double)c; open = false; }
        }
        if (!__any_sync(FULL, open)) break;
        const float se = expf(bp[6]);
        const float se2 = se * se;
        VillarF e;
        e.init(bp);
        Nll acc;
        acc.reset();
        const float4* o = obs + jb.off[b];
        const int n = jb.n[b];
        if (T == 2) {
            if (open)
                for (int i = h; i < n; i += 2) {
                    float4 q = o[i];
                    int st = ST_OK;
                    float pr = e.eval(q.x, q.y, st);
                    acc.obs(q, pr, st, se2);
                }
        } else {
            for (int i0 = 0; i0 < n; i0 += T) {
                const float4 q = o[min(i0 + r, n - 1)];
                int st = ST_OK;
                const float pr = e.eval(q.x, q.y, st);
                float term = 0.0f;
                const bool plain = st == ST_OK && Nll::ordinary(q, pr, se2, term);
                if (!__any_sync(FULL, open && !plain)) {
                    for (int k = 0; k < T; k += 2) {
                        const float tk = __shfl_sync(FULL, term, from + k);
                        if (i0 + h + k < n) acc.add(tk);
                    }
                } else {
                    for (int k = 0; k < T; k += 2) {
                        const float pk = __shfl_sync(FULL, pr, from + k);
                        const int sk = __shfl_sync(FULL, st, from + k);
                        if (i0 + h + k < n) acc.obs(o[i0 + h + k], pk, sk, se2);
                    }
                }
            }
        }
        const ff part = ff_add(ffm(acc.s, 0.0f), -acc.c);
        ff band_nll = ff_add(part, ffm(__shfl_xor_sync(FULL, part.hi, 1), __shfl_xor_sync(FULL, part.lo, 1)));
        const float ob = __shfl_xor_sync(FULL, acc.big, 1);
        float big = acc.big;
        if (ob > -INFINITY) big = big > -INFINITY ? fmaxf(big, ob) + log1pf(expf(-fabsf(big - ob))) : ob;
        const int fl = acc.nonfinite | (acc.inf << 1);
        const int flags = fl | __shfl_xor_sync(FULL, fl, 1);
        if (open) {
            if (flags & 1) { cost = BIG_COST; open = false; }
            else if (flags & 2) { cost = INFINITY; open = false; }
            else if (big > -INFINITY) {
                if (big > LN_DBL_MAX) { cost = INFINITY; open = false; }
                else band_nll = ff_add(band_nll, ff_from(exp((double)big)));
            }
        }
        if (n > 0) balanced = ff_add(balanced, ff_mul(band_nll, jb.wf[b]));
    }
    if (!open) return cost;
    // population prior of the reference band, relative priors of the offsets
    float lp = 0.0f;
#pragma unroll
    for (int j = 0; j < 7; j++) {
        float w = (float)c_pop_w[VILLAR][j];
        if (w > 0.0f) {
            float z = (ref[j] - (float)c_pop_c[VILLAR][j]) / w;
            lp += 0.5f * z * z;
        }
    }
    for (int b = 1; b < jb.nb; b++)
#pragma unroll
        for (int j = 0; j < 7; j++) {
            float z = (xs[(7 * b + j) * JP + p].x - c_rel_mean[j]) / c_rel_sigma[j];
            lp += 0.5f * z * z;
        }
    return ff_to(ff_mul(ff_add(balanced, lp), jb.inv_total_f));
}

// A task's team of C blocks, a cluster: particle p belongs to block p mod C.
template <int C>
struct JointTeam {
    static __device__ __forceinline__ int rank() { return C == 1 ? 0 : (int)cg::this_cluster().block_rank(); }
    static __device__ __forceinline__ void sync() {
        if (C == 1) __syncthreads();
        else {
            __syncwarp();
            cg::this_cluster().sync();
        }
    }
    // writes v to *p of every block
    template <class V>
    static __device__ __forceinline__ void put(V* p, V v) {
        if (C == 1) *p = v;
        else
#pragma unroll
            for (int k = 0; k < C; k++) *cg::this_cluster().map_shared_rank(p, k) = v;
    }
    // The first particle of the team whose flag is set (or JP).  One sync; the
    // caller's next one protects s_first.
    static __device__ int first(bool flag, int p, int* s_first) {
        const int lane = threadIdx.x & 31;
        const unsigned m = __ballot_sync(FULL, flag);
        const int q = __shfl_sync(FULL, p, m ? __ffs(m) - 1 : 0);
        if (lane == 0) put(&s_first[rank() * J_WARPS + (threadIdx.x >> 5)], m ? q : JP);
        sync();
        int v = JP;
        for (int k = lane; k < C * J_WARPS; k += 32) v = min(v, s_first[k]);
        return __reduce_min_sync(FULL, v);
    }
    // Lanes of a particle when the particles from `start` on move: as many as
    // the team's threads allow, so that the later rounds of an iteration,
    // whose few particles would leave most warps idle, are shorter.
    static __device__ __forceinline__ int lanes_of(int start) {
        constexpr int MOST = C == 1 ? 4 : 2 * C;
        int T = 2 * C;
        while (T < MOST && (JP - start + C - 1) / C * 2 * T <= J_THREADS) T *= 2;
        return T;
    }
    // This thread's particle of those from `start` on.
    static __device__ __forceinline__ int particle(int start, int T) {
        return start + ((rank() - start) & (C - 1)) + threadIdx.x / T * C;
    }
};

// Floats of a team's slice of joint_state: per parameter and particle two
// positions, two velocities and a personal best as double-float pairs, and
// per particle the personal best's FP64 cost; the table of inertia weights.
static __host__ __device__ size_t joint_state_floats(int max_d) { return (size_t)(10 * max_d + 2) * JP + 2 * J_MAXIT; }

// The persistent joint swarm: each team takes (source, restart) tasks from a
// device counter.  The state is kept in the team's slice of joint_state
// (L1/L2-resident, coalesced), so that shared memory holds only the staged
// observations.  Positions move as double-float pairs with the reference's
// FP64 draws and box: rounding only the joint swarm's positions to FP32 in
// the FP64 restatement moves the joint cost of 29 of the reference's 30 real
// ZTF sources by more than 1e-4, 13 of them by more than 1 % (up to 72 %).
// The cost is evaluated in FP32 at the leading floats.
//
// A round of a task alone on an SM was 33,000 cycles at 90 observations and
// 21 parameters: 15,000 in the cost (issue and MUFU of 13 warps), 9,500 in
// the moves (a dimension's loads waited out one after another), 3,400 in the
// FP64 of the inertia weight and the stall test, the rest in barriers.  So
//   - a particle's trial goes to the other of two states and is accepted by
//     the iteration's parity, not recomputed and copied;
//   - the weights are a table, and the stall test runs only in iterations
//     that improved the best (in the others it falls as before);
//   - where the batch leaves the register file free (PER_SM = 1), a move's
//     loads are issued two dimensions at a time; three and four measured the
//     same, and with 72 registers (PER_SM = 2) more than one spills;
//   - the next iteration's draws are asked into L2 early (2 %);
//   - a lone task is spread over a cluster of four blocks, each with every
//     fourth particle, whose rounds meet in two cluster barriers.
// This stage of 100 basic sources (3 x 30): 44 -> 31 ms; of 500 uneven ones:
// 145 -> 103; the whole fit of 20 long ones (3 x 1000): 442 -> 189.
template <int C, int PER_SM>
__global__ void __launch_bounds__(J_THREADS, PER_SM) joint_pso_kernel(DeviceBatch d) {
    using Team = JointTeam<C>;
    constexpr int U = PER_SM == 1 ? 2 : 1;  // dimensions whose loads a move issues at once
    const int rank = Team::rank();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x;
    __shared__ JointBands jb;
    __shared__ int s_first[C * J_WARPS], s_q[C];
    __shared__ double s_gc, s_min[C];
    __shared__ int s_task;
    __shared__ ff s_lo[J_MAX_D], s_hi[J_MAX_D], s_vm[J_MAX_D], s_g[J_MAX_D];
    __shared__ double s_tpeak;
    const int DM = d.joint_max_d;
    float4* obs = reinterpret_cast<float4*>(smem_raw);
    // the team's slice of the swarm state: two positions and velocities of
    // each particle (iteration `it` moves from the state `it & 1` to the
    // other: every particle is accepted once in an iteration), its personal
    // best and that one's cost
    const size_t S = (size_t)DM * JP;
    float2* xs = reinterpret_cast<float2*>(d.joint_state + blockIdx.x / C * joint_state_floats(DM));
    float2* vs = xs + 2 * S;
    float2* pb = vs + 2 * S;
    double* pbc = reinterpret_cast<double*>(pb + S);
    ff* ws = reinterpret_cast<ff*>(pbc + JP);  // the iterations' inertia weights
    for (int i = tid; i < J_MAXIT; i += J_THREADS)  // the team's blocks write the same
        ws[i] = ff_from(__dsub_rn(0.9, __dmul_rn(__dmul_rn(__dsub_rn(0.9, 0.4), (double)i), 1.0 / (double)J_MAXIT)));
    const int n_tasks = 3 * d.n_joint;
    while (true) {
        Team::sync();
        if (rank == 0 && tid == 0) Team::put(&s_task, atomicAdd(&d.ctr->joint_head, 1));
        Team::sync();
        const int task = s_task;
        if (task >= n_tasks) break;
        const int js = task / 3, restart = task % 3;
        const int src = d.joint_src[js];
        // ---- the source's valid bands in rank order
        if (tid == 0) {
            int nb = 0, tot = 0;
            for (int r = 0; r < J_MAX_BANDS; r++) {
                for (int b = d.src_off[src]; b < d.src_off[src + 1]; b++) {
                    const BandStats& bs = d.stats[b];
                    if (bs.valid && bs.rank == r) {
                        jb.n[nb] = bs.n;
                        jb.off[nb] = tot;
                        tot += bs.n;
                        nb++;
                    }
                }
            }
            jb.nb = nb;
            jb.n_total = tot;
            const double scale = (double)tot / (double)max(nb, 1);
            for (int b = 0; b < nb; b++) {
                jb.wf[b] = ff_from(jb.n[b] > 0 ? scale / (double)jb.n[b] : 0.0);
            }
            jb.inv_total_f = ff_from(1.0 / (double)max(tot, 1));
        }
        __syncthreads();
        const int nb = jb.nb, D = 7 * nb;
        if (nb == 0) continue;
        // stage the bands' records
        for (int r = 0; r < nb; r++) {
            int b_idx = -1;
            for (int b = d.src_off[src]; b < d.src_off[src + 1]; b++)
                if (d.stats[b].valid && d.stats[b].rank == r) b_idx = b;
            const BandStats bs = d.stats[b_idx];
            for (int i = tid; i < bs.n; i += J_THREADS) obs[jb.off[r] + i] = d.obs[bs.off + i];
        }
        // ---- bounds in FP64 (src/parametric.rs:3860-3882): Villar box with the
        // reference band's data-informed t0 (no lo < hi check), offsets at
        // +-3 sigma of the relative priors; vmax = (hi - lo) / 2
        if (tid == 0) {
            int b_ref = -1;
            for (int b = d.src_off[src]; b < d.src_off[src + 1]; b++)
                if (d.stats[b].valid && d.stats[b].rank == 0) b_ref = b;
            const BandStats bs = d.stats[b_ref];
            s_tpeak = bs.t_peak;
            for (int j = 0; j < D; j++) {
                double lo, hi;
                if (j < 7) {
                    lo = c_lo[VILLAR][j];
                    hi = c_hi[VILLAR][j];
                    if (j == 3) {
                        lo = fmax(bs.t_first - 30.0, lo);
                        hi = fmin(bs.t_peak + 10.0, hi);
                    }
                } else {
                    lo = -3.0 * c_rel_sigma64[j % 7];
                    hi = 3.0 * c_rel_sigma64[j % 7];
                }
                s_lo[j] = ff_from(lo);
                s_hi[j] = ff_from(hi);
                s_vm[j] = ff_from(__dmul_rn(0.5, __dsub_rn(hi, lo)));
            }
        }
        __syncthreads();
        const double t_peak = s_tpeak;
        const double* dr = d.joint_draws64 + (size_t)restart * d.joint_init_per_seed;
        const float2* d15 = d.joint_draws15 + (size_t)restart * d.joint_draws_per_seed;
        const bool seeded = restart == 1;
        // ---- initialisation (pso_minimize :1677-1692; seeded :1189-1210) in
        // FP64 without contractions; the seed particle (:3884-3895) is the
        // population prior centre with t0 = t_peak - 5 and the relative
        // priors' means, clamped to the box
        int T = Team::lanes_of(0);
        int r = tid & (T - 1), p = Team::particle(0, T);
        bool active = p < JP;
        if (active) {
            for (int j = r; j < D; j += T) {
                const double lo = ff_to(s_lo[j]), hi = ff_to(s_hi[j]), vmax = ff_to(s_vm[j]);
                double x, v;
                if (seeded) {
                    if (p == 0) {
                        double c = j < 7 ? c_pop_c[VILLAR][j] : c_rel_mean64[j % 7];
                        if (j == 3) c = t_peak - 5.0;
                        x = fmin(fmax(c, lo), hi);
                        v = __dmul_rn(__dmul_rn(vmax, 0.2), __dsub_rn(2.0 * dr[j], 1.0));
                    } else {
                        const int o = D + 2 * D * (p - 1);
                        x = __dadd_rn(lo, __dmul_rn(dr[o + j], __dsub_rn(hi, lo)));
                        v = __dmul_rn(__dmul_rn(vmax, 0.2), __dsub_rn(2.0 * dr[o + D + j], 1.0));
                    }
                } else {
                    const int o = 2 * D * p;
                    x = __dadd_rn(lo, __dmul_rn(dr[o + 2 * j], __dsub_rn(hi, lo)));
                    v = __dmul_rn(__dmul_rn(vmax, 0.2), __dsub_rn(2.0 * dr[o + 2 * j + 1], 1.0));
                }
                const ff xf = ff_from(x), vf = ff_from(v);
                const size_t k = (size_t)j * JP + p;
                xs[k] = make_float2(xf.hi, xf.lo);
                vs[k] = make_float2(vf.hi, vf.lo);
                pb[k] = xs[k];
            }
        }
        __syncthreads();
        double c = joint_cost(jb, obs, xs, p, T, r, active);
        if (!active) c = INFINITY;
        if (active && r == 0) pbc[p] = c;
        int evals = active && r == 0 ? 1 : 0;
        // global best after the sequential initial loop: the first strict
        // minimum, in particle order
        {
            double* s_warp = reinterpret_cast<double*>(s_g);  // not yet in use
            static_assert(sizeof(s_g) >= J_WARPS * sizeof(double), "a minimum per warp");
            double mn = c;
            for (int k = 16; k; k >>= 1) mn = fmin(mn, __shfl_xor_sync(FULL, mn, k));
            if ((tid & 31) == 0) s_warp[tid >> 5] = mn;
            __syncthreads();
            double g = INFINITY;
            for (int w = 0; w < J_WARPS; w++) g = fmin(g, s_warp[w]);
            int q = JointTeam<1>::first(active && c == g && g < INFINITY, p, s_first);
            if (C > 1) {
                if (tid == 0) {
                    Team::put(&s_min[rank], g);
                    Team::put(&s_q[rank], q);
                }
                Team::sync();
                for (int k = 0; k < C; k++)
                    if (s_min[k] < g || (s_min[k] == g && s_q[k] < q)) {
                        g = s_min[k];
                        q = s_q[k];
                    }
            }
            if (q < JP) {
                if (active && p == q) {
                    for (int j = r; j < D; j += T) {
                        const float2 x = xs[(size_t)j * JP + p];
                        Team::put(&s_g[j], ffm(x.x, x.y));
                    }
                    if (r == 0) Team::put(&s_gc, g);
                }
            } else {
                if (tid == 0) s_gc = INFINITY;
                if (tid < D) s_g[tid] = ffm(0.0f, 0.0f);
            }
        }
        Team::sync();
        const int base = seeded ? 2 * D * JP - D : 2 * D * JP;
        int stall = 0, it = 0;
        double prev = s_gc;
        for (; it < J_MAXIT; it++) {
            const ff w = ws[it];
            const float2* rnd = d15 + base + (size_t)it * 2 * D * JP;
            // the next iteration's draws towards L2 while this one computes
            if (it + 1 < J_MAXIT)
                for (int k = (tid * C + rank) * 16; k < 2 * D * JP; k += J_THREADS * C * 16)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(rnd + 2 * D * JP + k));
            int start = 0;
            bool improved = false;
            while (start < JP) {
                T = Team::lanes_of(start);
                r = tid & (T - 1);
                p = Team::particle(start, T);
                active = p < JP;
                const int cur = it & 1;
                float2* xn_p = xs + (cur ^ 1) * S;
                double best = INFINITY;  // the particle's personal best
                if (active) {
                    // the particle's move into its other state, its lanes
                    // taking alternate dimensions
                    best = pbc[p];
                    const float2 *x0 = xs + cur * S + p, *v0 = vs + cur * S + p;
                    float2* vn_p = vs + (cur ^ 1) * S + p;
                    const float2* rp = rnd + (size_t)2 * D * p;
                    // U dimensions' loads at once: a load that misses L1
                    // takes longer than a dimension's arithmetic
                    for (int j0 = r; j0 < D; j0 += U * T) {
                        float2 x[U], v[U], b[U], a1[U], a2[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int j = j0 + u * T;
                            if (j < D) {
                                const size_t k = (size_t)j * JP;
                                x[u] = x0[k], v[u] = v0[k], b[u] = pb[k + p], a1[u] = rp[2 * j], a2[u] = rp[2 * j + 1];
                            }
                        }
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int j = j0 + u * T;
                            if (j < D) {
                                const size_t k = (size_t)j * JP;
                                ff xn, vn;
                                ff_move(ffm(x[u].x, x[u].y), ffm(v[u].x, v[u].y), ffm(b[u].x, b[u].y), s_g[j], w, a1[u],
                                        a2[u], s_vm[j], s_lo[j], s_hi[j], xn, vn);
                                xn_p[k + p] = make_float2(xn.hi, xn.lo);
                                vn_p[k] = make_float2(vn.hi, vn.lo);
                            }
                        }
                    }
                }
                __syncwarp();  // the particle's dimensions, before its cost
                if (__any_sync(FULL, active)) {
                    c = joint_cost(jb, obs, xn_p, p, T, r, active);
                    evals += active && r == 0;
                }
                const double gc = s_gc;
                const int q = Team::first(active && c < gc, p, s_first);
                const int qe = min(q, JP - 1);
                // the particles up to the first that improves the global best
                // keep their moves; that one is the best of the next round
                if (active && p <= qe) {
                    if (c < best) {
                        for (int j = r; j < D; j += T) pb[(size_t)j * JP + p] = xn_p[(size_t)j * JP + p];
                        if (r == 0) pbc[p] = c;
                    }
                    if (p == q) {
                        for (int j = r; j < D; j += T) {
                            const float2 x = xn_p[(size_t)j * JP + p];
                            Team::put(&s_g[j], ffm(x.x, x.y));
                        }
                        if (r == 0) Team::put(&s_gc, c);
                    }
                }
                Team::sync();
                improved |= q < JP;
                start = qe + 1;
            }
            // without an improvement the test falls as it did before: not met
            const double gc = s_gc;
            if (improved && prev - gc > 0.01 * fmax(fabs(prev), 1e-10)) {
                stall = 0;
                prev = gc;
            } else if (++stall >= J_STALL) {
                it++;
                break;
            }
        }
        // ---- result
        const int mine = __reduce_add_sync(FULL, evals);
        if ((tid & 31) == 0) s_first[tid >> 5] = mine;
        __syncthreads();
        if (tid == 0) {
            int all = 0;
            for (int w = 0; w < J_WARPS; w++) all += s_first[w];
            Team::put(&s_q[rank], all);
        }
        Team::sync();
        if (rank == 0) {
            JointResult& R = d.joint_res[(size_t)js * 3 + restart];
            if (tid == 0) {
                int all = 0;
                for (int k = 0; k < C; k++) all += s_q[k];
                R.cost = s_gc;
                R.iters = it;
                R.evals = all;
                atomicAdd(&d.ctr->particle_obs_evals, (unsigned long long)all * (unsigned long long)jb.n_total);
            }
            if (tid < J_MAX_D) {
                R.params[tid] = tid < D ? s_g[tid].hi : 0.0f;
                R.params_lo[tid] = tid < D ? s_g[tid].lo : 0.0f;
            }
        }
    }
}

// Best of the three restarts; each band (rank k) gets reference + offset k.
__global__ void joint_pick_kernel(DeviceBatch d) {
    const int js = blockIdx.x * blockDim.x + threadIdx.x;
    if (js >= d.n_joint) return;
    const int src = d.joint_src[js];
    const JointResult* R = d.joint_res + (size_t)js * 3;
    double best = INFINITY;
    int br = -1;
    for (int r = 0; r < 3; r++)
        if (R[r].cost < best) { best = R[r].cost; br = r; }
    for (int b = d.src_off[src]; b < d.src_off[src + 1]; b++) {
        const BandStats bs = d.stats[b];
        BandOut& o = d.out[b];
        o.model = -1;
        for (int m = 0; m < 8; m++) o.per_chi2[m] = NAN;
        if (!bs.valid || br < 0) continue;  // no finite joint cost: not fitted
        const int k = bs.rank;
        o.model = VILLAR;
        o.pso_cost = best;
        o.per_chi2[VILLAR] = isfinite(best) ? best : NAN;
        for (int j = 0; j < MAXP; j++) {
            if (j >= 7) { o.pso_params[j] = NAN; continue; }
            const double ref = (double)R[br].params[j] + (double)R[br].params_lo[j];
            const double off = (double)R[br].params[7 * k + j] + (double)R[br].params_lo[7 * k + j];
            o.pso_params[j] = k == 0 ? ref : ref + off;
        }
    }
}

size_t joint_state_bytes(int grid, int max_d) { return grid * joint_state_floats(max_d) * sizeof(float); }

size_t joint_smem_bytes(int max_obs, int max_d) {
    (void)max_d;
    return (size_t)max_obs * sizeof(float4);
}

// How the joint swarm runs: blocks of a task's team, and blocks an SM holds.
// All forms give the same bits (5,400 uneven sources fitted in each).
//   - Four blocks a task as long as the teams' blocks fill the device at most
//     one and a half times, or, for sources whose observations carry the
//     round, up to a task an SM.  Total ms of a fit, one block -> four:
//     1 basic source 11.9 -> 9.9, 20: 32.1 -> 30.1, 30: 24.6 -> 26.0;
//     6 uneven ones (up to 1,500 observations) 61 -> 38, 35: 54.7 -> 47.4,
//     50: 58.5 -> 58.8, 100: 74.6 -> 100; 40 of 3 x 1000 574 -> 334.  Two
//     blocks are between the two or worse than both, eight within 10 % of
//     four at a source and behind from 12 on.
//   - One block an SM (126 registers) up to three tasks an SM, two (72
//     registers) from there: 150 basic sources 44.0 against 47.5, 200: 53.5
//     against 52.2; 100 uneven ones 74.6 against 84.1, 500: 176 against 152.
struct JointForm {
    int blocks, per_sm;
    void (*kernel)(DeviceBatch);
};
static JointForm joint_form(int n_joint, int max_obs, size_t smem, int num_sms) {
    const int n_tasks = 3 * n_joint;
    const bool room = smem <= 200 * 1024;  // the team's exchange takes static shared memory
    if (room && (8 * n_tasks <= 3 * num_sms || (max_obs >= 256 && n_tasks <= num_sms)))
        return {4, 1, joint_pso_kernel<4, 1>};
    if (n_tasks <= 3 * num_sms) return {1, 1, joint_pso_kernel<1, 1>};
    return {1, 2, joint_pso_kernel<1, 2>};
}

// Teams of the persistent joint swarm: as many as are resident at once.
int joint_grid(int n_joint, int max_obs, int max_d, int num_sms) {
    const size_t smem = joint_smem_bytes(max_obs, max_d);
    const JointForm f = joint_form(n_joint, max_obs, smem, num_sms);
    int per_sm = 0;
    if (cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f.kernel, J_THREADS, smem) != cudaSuccess)
        per_sm = 1;
    return std::max(1, std::max(1, per_sm) * num_sms / f.blocks);
}

int launch_joint(const DeviceBatch& d, cudaStream_t s) {
    if (d.n_joint == 0) return 0;
    const size_t smem = joint_smem_bytes(d.joint_max_obs, d.joint_max_d);
    const JointForm f = joint_form(d.n_joint, d.joint_max_obs, smem, d.num_sms);
    if (cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -1;
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim = {(unsigned)f.blocks, 1, 1};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f.blocks * std::min(d.joint_grid, 3 * d.n_joint));
    cfg.blockDim = dim3(J_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &cluster;
    cfg.numAttrs = f.blocks > 1 ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, f.kernel, d) != cudaSuccess) return -1;
    joint_pick_kernel<<<(d.n_joint + 127) / 128, 128, 0, s>>>(d);
    return 0;
}

}  // namespace lcf
