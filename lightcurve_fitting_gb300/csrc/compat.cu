// compat.cu — the reference's CUDA FFI, with the names and signatures its Rust
// host binds (src/gpu_cuda.rs:17-164) and the semantics of the kernels behind
// them (cuda/models.cu, cuda/svi.cu), so that an unmodified `GpuContext`
// links against liblcf_gb300.so.  FP64 throughout, device pointers, the
// legacy default stream, void return (errors surface through
// cudaGetLastError, as in the reference).  `grid` and `block` are accepted
// and ignored: the launch shapes are this library's.
//
//   launch_{bazin,...,metzger_kn}      model evaluation at draws x times
//   launch_batch_pso_cost             swarm cost of (source, particle) rows
//   launch_batch_pso_cost_multi_bazin the same for MultiBazin, K per source
//   launch_batch_svi_fit              the reference GPU's SVI, one source each
//
// The reference runs one thread per (source, particle) row, or one warp per
// source with lane 0 doing the bookkeeping; here a block takes a source and a
// chunk of its rows, or a warp a source, the lanes split the observations, and
// the FP64 partial sums are then combined (the same terms, summed in a
// different order).
#include <cuda_runtime.h>

#include "lcf_internal.cuh"
#include "lane_cost.cuh"
#include "models_f64.cuh"

namespace {

// ---------------------------------------------------------------------------
// Model evaluation (cuda/models.cu:590-617)
// ---------------------------------------------------------------------------
__global__ void eval_draws_kernel(int m, const double* p, const double* t, double* o, int nd, int nt, int np) {
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)nd * nt) return;
    int dd = (int)(idx / nt), ti = (int)(idx % nt);
    o[idx] = lcf::eval_model_f64(m, p + (int64_t)dd * np, t[ti]);
}

// MetzgerKN over the whole (unsorted) times array of one draw, as the
// reference's metzger_kn_eval (cuda/models.cu:146-260): one ODE over the
// draw's largest phase, normalised by its peak.
__global__ void metzger_draws_kernel(const double* p, const double* t, double* o, int nd, int nt, int np,
                                     double* tmp) {
    int dd = blockIdx.x * blockDim.x + threadIdx.x;
    if (dd >= nd) return;
    // sort the times by insertion into tmp (stable), evaluate, scatter back
    double* ts = tmp + (int64_t)dd * 2 * nt;
    double* ys = ts + nt;
    for (int i = 0; i < nt; i++) {
        double v = t[i];
        int j = i;
        while (j > 0 && ts[j - 1] > v) { ts[j] = ts[j - 1]; j--; }
        ts[j] = v;
    }
    lcf::metzger_f64(p + (int64_t)dd * np, ts, nt, ys);
    for (int i = 0; i < nt; i++) {
        // position of t[i] in the sorted array (first match of equal times)
        int lo = 0, hi = nt;
        while (lo < hi) {
            int mid = (lo + hi) / 2;
            if (ts[mid] < t[i]) lo = mid + 1; else hi = mid;
        }
        o[(int64_t)dd * nt + i] = ys[lo];
    }
}

void eval_draws(int m, const double* p, const double* t, double* o, int nd, int nt, int np) {
    int64_t total = (int64_t)nd * nt;
    if (total <= 0) return;
    eval_draws_kernel<<<(int)((total + 255) / 256), 256>>>(m, p, t, o, nd, nt, np);
}

// One observation's term of the reference GPU cost (cuda/models.cu:546-581):
// (pred - y)^2 / v + ln v for a detection, -ln Phi((u - pred) / sqrt v) for
// an upper limit, with v = obs_var + sigma_extra^2.  No 1/2, no prior, no
// Villar constraint, no MetzgerKN peak rescale: those belong to the CPU
// path's PsoCost, not to this kernel.
__device__ __forceinline__ double gpu_obs_term(double pred, double y, double var, int up, double uf, double se2) {
    const double tv = var + se2;
    if (up) return -lcf::log_normal_cdf_f64((uf - pred) / sqrt(tv));
    const double d = pred - y;
    return d * d / tv + log(tv);
}

// ---------------------------------------------------------------------------
// batch_pso_cost (cuda/models.cu:516-584): costs[s * n_part + k] = sum of the
// terms / n for positions[s][k][n_params], sigma_extra the last parameter;
// 1e99 for an empty source or a non-finite prediction.
//
// Bound by the FP64 pipe (one warp instruction per 16 cycles and SM), so by
// the FP64 instructions per evaluation and by the lanes that have none.  A
// block takes one source and a chunk of its particles: thread = (particle,
// slot), the COST_BLOCK / chunk slots split the observations, and the slots'
// sums meet in shared memory.  30 particles fill 120 of 128 threads whatever
// the band's length; a warp a row, its lanes over the observations, left 24 %
// of the lanes idle on the ~51-observation bands of the uneven workload.  The
// exponentials of a particle's log-parameters are formed once, spread over the
// block, instead of at every observation.  10,000 uneven bands x 30 particles,
// Villar, GB300: 5.3 ms, against 9.2 ms for a warp a row.
// ---------------------------------------------------------------------------
constexpr int COST_BLOCK = 128;
template <int M>
__global__ void __launch_bounds__(COST_BLOCK) pso_cost_kernel(const double* all_t, const double* all_f,
                                                              const double* all_var, const int* all_up,
                                                              const double* all_uf, const int* offs, const double* pos,
                                                              double* costs, int n_part, int np, int chunk) {
    __shared__ double s_c[2 * lcf::MAXP][COST_BLOCK];  // parameters, then their exponentials
    __shared__ double s_se2[COST_BLOCK], s_sum[COST_BLOCK];
    __shared__ int s_bad[COST_BLOCK];
    const int chunks = (n_part + chunk - 1) / chunk;
    const int s = blockIdx.x / chunks, k0 = (blockIdx.x % chunks) * chunk, tid = threadIdx.x;
    const int nk = min(n_part - k0, chunk);  // particles of this block
    const int o0 = offs[s], o1 = offs[s + 1];
    double* out = costs + (int64_t)s * n_part + k0;
    if (o1 - o0 <= 0) {
        for (int k = tid; k < nk; k += COST_BLOCK) out[k] = 1e99;
        return;
    }
    const double* rows = pos + ((int64_t)s * n_part + k0) * np;
    // a parameter of a particle per thread and turn; rows past np read as 0
    for (int q = tid; q < nk * lcf::MAXP; q += COST_BLOCK) {
        const int k = q / lcf::MAXP, j = q - k * lcf::MAXP;
        const double v = j < np ? rows[k * np + j] : 0.0;
        s_c[j][k] = v;
        if (lcf::log_param(M, j)) s_c[lcf::MAXP + j][k] = exp(v);
        if (M == 3 && j == 3) s_c[lcf::MAXP + 3][k] = lcf::nickel_fraction(v);
        if (j == np - 1) {
            const double sx = exp(v);
            s_se2[k] = sx * sx;
        }
    }
    __syncthreads();
    const int slots = COST_BLOCK / nk, slot = tid / nk, k = tid - slot * nk;
    double nll = 0.0;
    int bad = 0;
    if (slot < slots) {
        double p[lcf::MAXP], e[lcf::MAXP];
#pragma unroll
        for (int j = 0; j < lcf::MAXP; j++) {
            p[j] = s_c[j][k];
            e[j] = s_c[lcf::MAXP + j][k];
        }
        const double se2 = s_se2[k];
        for (int i = o0 + slot; i < o1; i += slots) {
            const double pred = lcf::eval_model_e<double>(M, p, lcf::ExpTable{e}, all_t[i]);
            if (!isfinite(pred)) {
                bad = 1;
                break;
            }
            nll += gpu_obs_term(pred, all_f[i], all_var[i], all_up[i], all_uf[i], se2);
        }
    }
    s_sum[tid] = nll;
    s_bad[tid] = bad;
    __syncthreads();
    if (tid < nk) {
        for (int q = 1; q < slots; q++) {
            nll += s_sum[q * nk + tid];
            bad |= s_bad[q * nk + tid];
        }
        out[tid] = bad ? 1e99 : nll / (double)(o1 - o0);
    }
}

// MetzgerKN: one warp per row, its lanes over the observations (each
// observation integrates its own ODE, cuda/models_device.h:458-470, which
// dwarfs the rest).
__global__ void __launch_bounds__(256) pso_cost_metzger_kernel(const double* all_t, const double* all_f,
                                                               const double* all_var, const int* all_up,
                                                               const double* all_uf, const int* offs,
                                                               const double* pos, double* costs, int n_src,
                                                               int n_part, int np) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= (int64_t)n_src * n_part) return;
    const int s = (int)(row / n_part);
    const int o0 = offs[s], o1 = offs[s + 1];
    if (o1 - o0 <= 0) {
        if (lane == 0) costs[row] = 1e99;
        return;
    }
    double p[lcf::MAXP];
#pragma unroll
    for (int j = 0; j < lcf::MAXP; j++) p[j] = j < np ? pos[row * np + j] : 0.0;
    const double sx = exp(pos[row * np + np - 1]);
    const double se2 = sx * sx;
    double nll = 0.0;
    int bad = 0;
    for (int i = o0 + lane; i < o1; i += 32) {
        const double pred = lcf::metzger_at_obs_f64(p, all_t[i]);
        if (!isfinite(pred)) {
            bad = 1;
            break;
        }
        nll += gpu_obs_term(pred, all_f[i], all_var[i], all_up[i], all_uf[i], se2);
    }
    bad = lcf::warp_or(bad);
    nll = lcf::warp_sum_d(nll);
    if (lane == 0) costs[row] = bad ? 1e99 : nll / (double)(o1 - o0);
}

// ---------------------------------------------------------------------------
// batch_pso_cost_multi_bazin (cuda/models.cu:295-362): sum of K Bazin
// components (log A, t0, log tau_rise, log tau_fall each) plus the shared
// baseline B and log sigma_extra; K = source_k[s], rows padded to n_params.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) pso_cost_mb_kernel(const double* all_t, const double* all_f,
                                                          const double* all_var, const int* all_up,
                                                          const double* all_uf, const int* offs, const double* pos,
                                                          double* costs, const int* source_k, int n_src, int n_part,
                                                          int np) {
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (row >= (int64_t)n_src * n_part) return;
    const int s = (int)(row / n_part);
    const int o0 = offs[s], o1 = offs[s + 1];
    if (o1 - o0 <= 0) {
        if (lane == 0) costs[row] = 1e99;
        return;
    }
    const int k = source_k[s];
    const double* p = pos + row * np;
    const double sx = exp(p[4 * k + 1]);
    const double se2 = sx * sx;
    const double b = p[4 * k];
    double nll = 0.0;
    int bad = 0;
    for (int i = o0 + lane; i < o1; i += 32) {
        const double t = all_t[i];
        double sum = 0.0;
        for (int c = 0; c < k; c++) {
            const double* q = p + 4 * c;
            const double dt = t - q[1];
            sum += exp(q[0]) * exp(-dt / exp(q[3])) * (1.0 / (1.0 + exp(-(dt / exp(q[2])))));
        }
        const double pred = sum + b;
        if (!isfinite(pred)) {
            bad = 1;
            break;
        }
        nll += gpu_obs_term(pred, all_f[i], all_var[i], all_up[i], all_uf[i], se2);
    }
    bad = lcf::warp_or(bad);
    nll = lcf::warp_sum_d(nll);
    if (lane == 0) costs[row] = bad ? 1e99 : nll / (double)(o1 - o0);
}

// ---------------------------------------------------------------------------
// batch_svi_fit (cuda/svi.cu:48-330): the reference GPU's SVI of one source
// per warp.  Its semantics, which differ from the CPU path's svi_fit:
//   * noise from xorshift64 seeded 42 + source * 123456789, uniforms
//     (x & (2^53 - 1)) / (2^53 - 1), Box-Muller per parameter (u1 then u2);
//   * prior centres and widths from the caller's arrays;
//   * MetzgerKN by its per-observation ODE, with forward differences
//     h = max(1e-5, 1e-5 |theta_j|) for its gradient;
//   * early stop after >= 50 steps once the ELBO's EMA(0.1) has not improved
//     by 1 % for 20 steps;
//   * log sigma clamped to [-6, 2] and reported without the CPU path's
//     ln 4 inflation; rows padded with 0 up to max_params; an empty source
//     gets elbo -1e99 and nothing else.
// A step's work beside the observations is per parameter (a draw's Box-Muller
// pair, the prior, Adam), and the FP64 pipe charges a warp instruction alike
// for one lane and for 32.  So each parameter has lanes of its own: lanes
// 4 (j + 1) .. 4 (j + 1) + 3 hold parameter j (the even ones its mean's Adam
// state, the odd ones its log sigma's), and lanes 0..3 the log-likelihood,
// which is where the reduce-scatter of the eight FP64 sums leaves them.  Every
// lane steps the same generator state (integer work) and keeps its own
// parameter's two draws.  The terms, sums and their order are those of one
// lane doing it all.  One warp a block, so that a finished source frees its
// slot at once.  Bound by the FP64 pipe.  3,000 uneven bands, 300 steps x 4
// samples, GB300: 449 ms, against 680 ms with every lane doing all of it.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long xs_next(unsigned long long& x) {
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    return x;
}
__device__ __forceinline__ double xs_uniform(unsigned long long x) {
    return (double)(x & 0x1FFFFFFFFFFFFFULL) / (double)0x1FFFFFFFFFFFFFULL;
}

struct SviArgs {
    const double *all_t, *all_f, *all_var;
    const int* all_up;
    const double* all_uf;
    const double *pso_params, *prior_c, *prior_w;
    double *out_mu, *out_ls, *out_elbo;
    int max_params, n_steps, n_samples;
    double lr;
};

template <int M>
__device__ __noinline__ void svi_source(const SviArgs& A, int s, int o0, int o1, int np, int se) {
    constexpr int MP = lcf::MAXP;
    const int lane = threadIdx.x & 31;
    const int j = (lane >> 2) - 1;  // this lane's parameter (-1: none)
    const bool own = j >= 0 && j < np, odd = lane & 1;
    const int64_t base = (int64_t)s * A.max_params;
    double mu = own ? A.pso_params[base + j] : 0.0, ls = -1.0;
    const double pc = own ? A.prior_c[base + j] : 0.0;
    const double w = own ? A.prior_w[base + j] : 1.0;
    const double pw2 = w * w;
    double am = 0.0, av = 0.0;
    auto of = [](double v, int k) { return __shfl_sync(FULL, v, 4 * (k + 1)); };
    unsigned long long rng = 42ULL + (unsigned long long)s * 123456789ULL;
    const double PI = 3.14159265358979323846;
    double final_elbo = -1e300, ema = -1e300, best = -1e300;
    int stall = 0, t_adam = 0;
    for (int step = 0; step < A.n_steps; step++) {
        const double sg = exp(ls);
        double gmu = 0.0, gls = 0.0, elbo_sum = 0.0;
        for (int smp = 0; smp < A.n_samples; smp++) {
            unsigned long long x1 = 1, x2 = 1;
            for (int q = 0; q < np; q++) {
                const unsigned long long a = xs_next(rng), b = xs_next(rng);
                if (q == j) {
                    x1 = a;
                    x2 = b;
                }
            }
            const double u1 = fmax(xs_uniform(x1), 1e-10), u2 = xs_uniform(x2);
            const double eps = sqrt(-2.0 * log(u1)) * cos(2.0 * PI * u2);
            const double thj = own ? mu + sg * eps : 0.0;
            const double ej = exp(thj);
            double th[MP], e[MP];
#pragma unroll
            for (int k = 0; k < MP; k++) {
                th[k] = of(thj, k);
                e[k] = (lcf::log_param(M, k)) ? of(ej, k) : 0.0;
            }
            if (M == 3) e[3] = lcf::nickel_fraction(th[3]);
            const double sx = of(ej, se);
            const double se2 = sx * sx;
            double v[8], dse = 0.0;  // log-likelihood and its gradient
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = 0.0;
            for (int i = o0 + lane; i < o1; i += 32) {
                const double t = A.all_t[i];
                double pred, g[MP];
                if constexpr (M != 7) pred = lcf::eval_model_e<double>(M, th, lcf::ExpTable{e}, t);
                else pred = lcf::metzger_at_obs_f64(th, t);
                if (!isfinite(pred)) continue;
                if constexpr (M != 7) {
                    lcf::model_grad_e<double>(M, th, lcf::ExpTable{e}, t, g);
                } else {
                    double tp[MP];
                    for (int k = 0; k < MP; k++) tp[k] = th[k];
                    for (int q = 0; q < np; q++) {
                        if (q == se) {
                            g[q] = 0.0;
                            continue;
                        }
                        const double h = fmax(1e-5, 1e-5 * fabs(th[q]));
                        tp[q] = th[q] + h;
                        const double pp = lcf::metzger_at_obs_f64(tp, t);
                        tp[q] = th[q];
                        g[q] = isfinite(pp) ? (pp - pred) / h : 0.0;
                    }
                    g[se] = 0.0;
                }
                const double tv = A.all_var[i] + se2;
                double dpred;
                if (A.all_up[i]) {
                    // ln Phi(z) and the density over the CDF in its 1 + erf
                    // form (the reference's gradient), sharing the A&S pieces
                    const double ist = rsqrt(tv), dz = A.all_uf[i] - pred, z = dz * ist;
                    const double a = fabs(z * 0.70710678118654752440);
                    const double q = 1.0 / (1.0 + 0.3275911 * a);
                    const double e2 =
                        q * (0.254829592 + q * (-0.284496736 + q * (1.421413741 + q * (-1.453152027 + q * 1.061405429)))) *
                        exp(-a * a);
                    const double lc = z < -30.0 ? -0.5 * z * z - 0.5 * log(2.0 * PI) - log(-z)
                                                : log(fmax(z > 0.0 ? 1.0 - 0.5 * e2 : 0.5 * e2, 1e-300));
                    if (!(z > 8.0)) v[0] += lc;  // NaN: ln 1e-300, as log_normal_cdf_f64 has it
                    const double erf = z >= 0.0 ? 1.0 - e2 : -(1.0 - e2);
                    const double phi = exp(-0.5 * z * z) * 0.39894228040143267794;
                    const double ratio = phi / fmax(0.5 * (1.0 + erf), 1e-300);
                    dpred = -ratio * ist;
                    dse += ratio * (-z * se2 * (ist * ist));
                } else {
                    const double it = 1.0 / tv;
                    const double r = A.all_f[i] - pred;
                    const double r2 = r * r;
                    v[0] += -0.5 * (r2 * it + log(2.0 * PI * tv));
                    dpred = r * it;
                    dse += (r2 * it * it - it) * se2;
                }
#pragma unroll
                for (int k = 0; k < MP; k++)
                    if (k < np && k != se && k < lcf::n_params_of(M) && isfinite(g[k])) v[1 + k] += dpred * g[k];
            }
#pragma unroll
            for (int k = 0; k < MP; k++)
                if (k == se) v[1 + k] = dse;
            // lane l: the warp's sum of v[l >> 2]
            const double tot = lcf::reduce_scatter8(v);
            const double d = thj - pc;
            const double lpj = -0.5 * d * d / pw2;
            double lp = 0.0;
            for (int q = 0; q < np; q++) lp += of(lpj, q);
            const double df = tot + (-d / pw2);
            gmu += df;
            gls += df * sg * eps;
            elbo_sum += __shfl_sync(FULL, tot, 0) + lp;
        }
        const double ns = (double)A.n_samples;
        double ent = 0.0;
        for (int q = 0; q < np; q++) ent += of(ls, q);
        gmu /= ns;
        gls /= ns;
        ent += 0.5 * (double)np * log(2.0 * PI * 2.71828182845904523536);
        final_elbo = elbo_sum / ns + ent;
        t_adam++;
        const double bc = 1.0 - pow(odd ? 0.999 : 0.9, (double)t_adam);
        const double bco = __shfl_xor_sync(FULL, bc, 1);
        const double bc1 = odd ? bco : bc, bc2 = odd ? bc : bco;
        const double gr = odd ? -(gls + 1.0) : -gmu;
        double val = odd ? ls : mu;
        if (isfinite(gr)) {
            am = 0.9 * am + 0.1 * gr;
            av = 0.999 * av + 0.001 * gr * gr;
            val -= A.lr * (am / bc1) / (sqrt(av / bc2) + 1e-8);
        }
        const double oth = __shfl_xor_sync(FULL, val, 1);
        mu = odd ? oth : val;
        ls = fmax(-6.0, fmin(2.0, odd ? val : oth));
        if (step >= 50) {
            ema = ema < -1e290 ? final_elbo : 0.1 * final_elbo + 0.9 * ema;
            if (ema - best > 0.01 * fmax(fabs(best), 1e-10)) {
                best = ema;
                stall = 0;
            } else if (++stall >= 20) {
                break;
            }
        }
    }
    if ((lane & 3) == 0 && own && j < A.max_params) {
        A.out_mu[base + j] = mu;
        A.out_ls[base + j] = fmax(-6.0, fmin(2.0, ls));
    }
    for (int q = max(np, 0) + lane; q < A.max_params; q += 32) A.out_mu[base + q] = A.out_ls[base + q] = 0.0;
    if (lane == 0) A.out_elbo[s] = final_elbo;
}

__global__ void __launch_bounds__(32, 16) svi_fit_kernel(SviArgs A, const int* offs, const int* model_ids,
                                                      const int* n_params_arr, const int* se_idx_arr) {
    const int s = blockIdx.x;
    const int o0 = offs[s], o1 = offs[s + 1];
    if (o1 - o0 <= 0) {
        if (threadIdx.x == 0) A.out_elbo[s] = -1e99;
        return;
    }
    const int np = min(n_params_arr[s], lcf::MAXP), se = se_idx_arr[s];
    switch (model_ids[s]) {
        case 0: svi_source<0>(A, s, o0, o1, np, se); break;
        case 1: svi_source<1>(A, s, o0, o1, np, se); break;
        case 2: svi_source<2>(A, s, o0, o1, np, se); break;
        case 3: svi_source<3>(A, s, o0, o1, np, se); break;
        case 4: svi_source<4>(A, s, o0, o1, np, se); break;
        case 5: svi_source<5>(A, s, o0, o1, np, se); break;
        case 7: svi_source<7>(A, s, o0, o1, np, se); break;
        default: svi_source<6>(A, s, o0, o1, np, se); break;
    }
}

}  // namespace

extern "C" {
void launch_bazin(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(0, p, t, o, nd, nt, np); }
void launch_villar(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(1, p, t, o, nd, nt, np); }
void launch_tde(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(2, p, t, o, nd, nt, np); }
void launch_arnett(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(3, p, t, o, nd, nt, np); }
void launch_magnetar(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(4, p, t, o, nd, nt, np); }
void launch_shock_cooling(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(5, p, t, o, nd, nt, np); }
void launch_afterglow(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) { eval_draws(6, p, t, o, nd, nt, np); }
void launch_metzger_kn(const double* p, const double* t, double* o, int nd, int nt, int np, int, int) {
    if (nd <= 0 || nt <= 0) return;
    double* tmp = nullptr;
    if (cudaMalloc(&tmp, (size_t)nd * 2 * nt * sizeof(double)) != cudaSuccess) return;
    metzger_draws_kernel<<<(nd + 63) / 64, 64>>>(p, t, o, nd, nt, np, tmp);
    cudaFree(tmp);
}

void launch_batch_pso_cost(const double* all_times, const double* all_flux, const double* all_obs_var,
                           const int* all_is_upper, const double* all_upper_flux, const int* source_offsets,
                           const double* positions, double* costs, int n_sources, int n_particles, int n_params,
                           int model_id, int, int) {
    if (n_sources <= 0 || n_particles <= 0 || n_params < 1 || n_params > lcf::MAXP || model_id < 0 || model_id > 7) return;
    const int64_t rows = (int64_t)n_sources * n_particles;
    if (model_id == 7) {
        pso_cost_metzger_kernel<<<(int)((rows * 32 + 255) / 256), 256>>>(all_times, all_flux, all_obs_var, all_is_upper,
                                                                         all_upper_flux, source_offsets, positions,
                                                                         costs, n_sources, n_particles, n_params);
        return;
    }
    using Kernel = void (*)(const double*, const double*, const double*, const int*, const double*, const int*,
                            const double*, double*, int, int, int);
    static const Kernel kernels[7] = {pso_cost_kernel<0>, pso_cost_kernel<1>, pso_cost_kernel<2>, pso_cost_kernel<3>,
                                      pso_cost_kernel<4>, pso_cost_kernel<5>, pso_cost_kernel<6>};
    // particles a block: up to 42 (three slots or more, in equal chunks), fewer
    // (down to 2) where that leaves the chip short of four rounds of blocks
    // (eight resident on an SM at 64 registers a thread): a smaller chunk gives
    // its particles more slots, so shorter chains of observations and a shorter
    // tail (1,000 uneven bands x 40, Villar: 1.08 ms with one chunk, 0.78 with
    // this rule, 1.31 for a warp a row)
    int device = 0, sms = 1;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int64_t enough = 4 * (int64_t)sms * 8;
    int chunk = (n_particles + 41) / 42;
    chunk = (n_particles + chunk - 1) / chunk;
    while (chunk > 2 && (int64_t)n_sources * ((n_particles + chunk - 1) / chunk) < enough) chunk = (chunk + 1) / 2;
    const unsigned blocks = (unsigned)n_sources * (unsigned)((n_particles + chunk - 1) / chunk);
    kernels[model_id]<<<blocks, COST_BLOCK>>>(all_times, all_flux, all_obs_var, all_is_upper, all_upper_flux,
                                              source_offsets, positions, costs, n_particles, n_params, chunk);
}

void launch_batch_pso_cost_multi_bazin(const double* all_times, const double* all_flux, const double* all_obs_var,
                                       const int* all_is_upper, const double* all_upper_flux,
                                       const int* source_offsets, const double* positions, double* costs,
                                       const int* source_k, int n_sources, int n_particles, int n_params, int, int) {
    const int64_t rows = (int64_t)n_sources * n_particles;
    if (rows <= 0 || n_params < 6) return;
    pso_cost_mb_kernel<<<(int)((rows * 32 + 255) / 256), 256>>>(all_times, all_flux, all_obs_var, all_is_upper,
                                                                all_upper_flux, source_offsets, positions, costs,
                                                                source_k, n_sources, n_particles, n_params);
}

void launch_batch_svi_fit(const double* all_times, const double* all_flux, const double* all_obs_var,
                          const int* all_is_upper, const double* all_upper_flux, const int* source_offsets,
                          const double* pso_params, const int* model_ids, const int* n_params_arr,
                          const int* se_idx_arr, const double* prior_centers, const double* prior_widths,
                          double* out_mu, double* out_log_sigma, double* out_elbo, int n_sources, int max_params,
                          int n_steps, int n_samples, double lr, int, int) {
    if (n_sources <= 0 || max_params < 1) return;
    const SviArgs args = {all_times, all_flux, all_obs_var, all_is_upper, all_upper_flux, pso_params, prior_centers,
                          prior_widths, out_mu, out_log_sigma, out_elbo, max_params, n_steps, n_samples, lr};
    svi_fit_kernel<<<n_sources, 32>>>(args, source_offsets, model_ids, n_params_arr, se_idx_arr);
}
}
