// finalize.cu — the FP64 stages after model selection and the dependent
// PSO stages' task builders:
//   * Laplace (laplace_fit, src/parametric.rs:2623-2693): central finite
//     difference Hessian of the unnormalised negative log-posterior over the
//     shape parameters, Jacobi eigen-decomposition, eigenvalue clamp 1e-6;
//   * profile_t0_refine (:2788-3008), profile_refine_all (:2705-2786) and the
//     magnitude-space chi2 (:3680-3711);
//   * the profile t0 search (:1767-1849) and the greedy MultiBazin K = 1..4
//     fit (:1008-1157), whose PSO runs execute in pso.cu and whose task lists
//     are appended here on the device, so the whole sequence needs no host
//     round trip.
// One warp per band, the lanes splitting the observations and the FP64 sums
// reduced across the warp; MetzgerKN, whose light curve is a sequential
// integration, takes a block per band with an integration a lane.
#include <cuda_runtime.h>

#include <algorithm>

#include "lcf_internal.cuh"
#include "metzger_block.cuh"
#include "models_f32.cuh"
#include "models_f64.cuh"

namespace lcf {

#define FULL 0xffffffffu

__device__ __forceinline__ double wsum(double v) {
    for (int k = 16; k; k >>= 1) v += __shfl_xor_sync(FULL, v, k);
    return v;
}

struct BandView {
    const double *t, *f, *fe, *var, *uf, *mag;
    const uint8_t* up;
    int n;
    double peak;
};
__device__ __forceinline__ BandView band_view(const DeviceBatch& d, const BandStats& bs) {
    BandView v;
    v.t = d.t64 + bs.off; v.f = d.f64 + bs.off; v.fe = d.fe64 + bs.off; v.var = d.var64 + bs.off;
    v.uf = d.uf64 + bs.off; v.mag = d.mag64 + bs.off; v.up = d.up + bs.off;
    v.n = bs.n; v.peak = bs.peak;
    return v;
}

// neg_log_posterior, src/parametric.rs:2464-2511 (models other than
// MetzgerKN).  Out of line: called for one value and, rarely, for a stencil,
// and inlined it would change how the Hessian's own products are contracted.
__device__ __noinline__ double neg_log_posterior_w(int m, const BandView& b, const double* p) {
    int lane = threadIdx.x & 31;
    Model64 mod;
    mod.init(m, p);
    double se2 = exp(2.0 * p[se_idx_of(m)]);
    double nll = 0.0;
    int nonfinite = 0;
    for (int i = lane; i < b.n; i += 32) {
        double pr = mod.eval(b.t[i], nullptr);
        if (!isfinite(pr)) { nonfinite = 1; continue; }
        double tv = b.var[i] + se2;
        if (b.up[i]) nll -= log_normal_cdf_f64((b.uf[i] - pr) / sqrt(tv));
        else {
            double dd = pr - b.f[i];
            nll += 0.5 * (dd * dd / tv + log(2.0 * 3.14159265358979323846 * tv));
        }
    }
    if (__any_sync(FULL, nonfinite)) return 1e99;
    nll = wsum(nll);
    double nlp = 0.0;
    for (int j = 0; j < n_params_of(m); j++) {
        double w = c_pri_w[m][j], dd = p[j] - c_pri_c[m][j];
        nlp += 0.5 * dd * dd / (w * w);
    }
    __syncwarp();
    return nll + nlp;
}

// ---------------------------------------------------------------------------
// The refinement scans of models other than MetzgerKN evaluate the model in
// FP32 (the evaluators of models_f32.cuh, on the band's FP32 time records)
// and form each observation's term in FP64 from per-band constants that do
// not change across the scans (sigma_extra is fixed there): 1/tv, 1/sqrt(tv)
// and ln(2 pi tv).  The scans compare log-likelihoods against thresholds
// 0.5 apart and pick grid points, so FP32 prediction rounding (1e-7
// relative) moves no decision except a value within ~1e-5 of a threshold.
// ---------------------------------------------------------------------------
__device__ void scan_constants(const BandView& b, double se2, double* cst, int i0, int stride) {
    for (int i = i0; i < b.n; i += stride) {
        double tv = b.var[i] + se2;
        cst[3 * i] = 1.0 / tv;
        cst[3 * i + 1] = 1.0 / sqrt(tv);
        cst[3 * i + 2] = log(2.0 * 3.14159265358979323846 * tv);
    }
}

// FP32 prediction -> FP64 value; false for a prediction the reference finds
// non-finite (skipped by the scans).  Huge predictions come back through
// their logarithm (ST_BIG) and are finite in FP64.
__device__ __forceinline__ bool pred_f64(float pf, int st, double& pr) {
    if (st == ST_NONFINITE) return false;
    pr = st == ST_BIG ? exp((double)pf) : (double)pf;
    return true;
}

__device__ __forceinline__ double ll_term(const BandView& b, int i, double pr, const double* cst) {
    const double* c = cst + 3 * i;
    if (b.up[i]) {
        double z = (b.uf[i] - pr) * c[1];
        if (z > -1e15) return (double)log_normal_cdf_f((float)z);
        return -0.5 * z * z - 0.9189385332046727 - log(-z);
    }
    double r = b.f[i] - pr;
    return -0.5 * (r * r * c[0] + c[2]);
}

template <class F>
__device__ double ll_scan_t(const double* p, const float4* obs, const BandView& b, const double* cst) {
    F e;
    e.init64(p);
    double ll = 0.0;
    for (int i = threadIdx.x & 31; i < b.n; i += 32) {
        float4 o = obs[i];
        int st = ST_OK;
        float pf = e.eval(o.x, o.y, st);
        double pr;
        if (!pred_f64(pf, st, pr)) continue;
        ll += ll_term(b, i, pr, cst);
    }
    return wsum(ll);
}

// Band log-likelihood skipping non-finite predictions (the profile scans,
// src/parametric.rs:2716-2726, :2916-2932), models other than MetzgerKN
__device__ double band_ll_fast(int m, const double* p, const float4* obs, const BandView& b, const double* cst) {
    switch (m) {
        case BAZIN: return ll_scan_t<BazinF>(p, obs, b, cst);
        case VILLAR: return ll_scan_t<VillarF>(p, obs, b, cst);
        case TDE: return ll_scan_t<TdeF>(p, obs, b, cst);
        case ARNETT: return ll_scan_t<ArnettF>(p, obs, b, cst);
        case MAGNETAR: return ll_scan_t<MagnetarF>(p, obs, b, cst);
        case SHOCK: return ll_scan_t<ShockF>(p, obs, b, cst);
        default: return ll_scan_t<AfterglowF>(p, obs, b, cst);
    }
}

// Weighted sums of the unit-amplitude shape for the amplitude (and baseline)
// solve of profile_t0_refine: sw, sy, sf, syf, sff over detections.
template <class F>
__device__ void shape_sums_t(const double* p, const float4* obs, const BandView& b, const double* cst, double* s5) {
    F e;
    e.init64(p);
    double sw = 0, sy = 0, sf = 0, syf = 0, sff = 0;
    for (int i = threadIdx.x & 31; i < b.n; i += 32) {
        if (b.up[i]) continue;
        float4 o = obs[i];
        int st = ST_OK;
        float pf = e.eval(o.x, o.y, st);
        double sh;
        if (!pred_f64(pf, st, sh) || !isfinite(sh)) continue;
        double w = cst[3 * i];
        sw += w; sy += w * b.f[i]; sf += w * sh; syf += w * b.f[i] * sh; sff += w * sh * sh;
    }
    s5[0] = wsum(sw); s5[1] = wsum(sy); s5[2] = wsum(sf); s5[3] = wsum(syf); s5[4] = wsum(sff);
}

__device__ void shape_sums_fast(int m, const double* p, const float4* obs, const BandView& b, const double* cst,
                                double* s5) {
    switch (m) {
        case BAZIN: shape_sums_t<BazinF>(p, obs, b, cst, s5); break;
        case VILLAR: shape_sums_t<VillarF>(p, obs, b, cst, s5); break;
        case TDE: shape_sums_t<TdeF>(p, obs, b, cst, s5); break;
        case ARNETT: shape_sums_t<ArnettF>(p, obs, b, cst, s5); break;
        case MAGNETAR: shape_sums_t<MagnetarF>(p, obs, b, cst, s5); break;
        case SHOCK: shape_sums_t<ShockF>(p, obs, b, cst, s5); break;
        default: shape_sums_t<AfterglowF>(p, obs, b, cst, s5); break;
    }
}

// ---------------------------------------------------------------------------
// MetzgerKN refinement scans: a block per band, one scan point per lane
// (metzger_block.cuh).
// ---------------------------------------------------------------------------
struct MzPeak {
    const uint8_t* up;
    double mx;  // largest unnormalised detection interpolant
    __device__ void operator()(int j, double l) {
        if (!up[j]) mx = fmax(mx, l);
    }
};

struct MzLl {
    const BandView* b;
    const double* cst;
    double scale, ll;
    __device__ void term(int j, double pr) {
        if (!isfinite(pr)) return;
        const double* c = cst + 3 * j;
        if (b->up[j]) {
            ll += log_normal_cdf_f64((b->uf[j] - pr) * c[1]);
        } else {
            double r = b->f[j] - pr;
            ll += -0.5 * (r * r * c[0] + c[2]);
        }
    }
};

// The same for MetzgerKN by one lane (rescale: the PSO cost's peak rescale)
__device__ double metzger_ll_lane(MzTables& T, int slot, int col, const double* p, const BandView& b,
                                  const double* cst, bool rescale) {
    int j_start = b.n;
    double l_peak;
    bool ok = mz_sweep(T, p, slot, col, l_peak);
    bool valid = ok && l_peak > 0.0 && isfinite(l_peak);
    double scale = 1.0;
    if (rescale) {
        // largest normalised detection prediction; invalid sweeps and the
        // observations before t0 predict 0
        MzPeak pk{b.up, -INFINITY};
        if (valid) mz_visit(T, slot, col, p[3], b.t, b.n, j_start, pk);
        double mx = -INFINITY;
        int z_end = valid ? j_start : b.n;
        for (int j = 0; j < z_end; j++)
            if (!b.up[j]) mx = fmax(mx, 0.0);
        if (valid) mx = fmax(mx, pk.mx / l_peak);
        if (mx > 1e-10 && isfinite(mx)) scale = fmin(fmax(1.0 / mx, 0.1), 10.0);
    }
    MzLl acc{&b, cst, scale, 0.0};
    if (valid) {
        j_start = 0;
        while (j_start < b.n && b.t[j_start] - p[3] <= 0.0) j_start++;
    }
    int z_end = valid ? j_start : b.n;
    for (int j = 0; j < z_end; j++) acc.term(j, 0.0 * scale);
    if (valid) {
        // the interpolants, normalised
        struct Norm {
            MzLl* a;
            double lpk;
            __device__ void operator()(int j, double l) { a->term(j, l / lpk * a->scale); }
        } nv{&acc, l_peak};
        mz_visit(T, slot, col, p[3], b.t, b.n, j_start, nv);
    }
    return acc.ll;
}

// shape sums of profile_t0_refine for MetzgerKN by one lane: sw, sy, sf,
// syf, sff over detections of the normalised prediction
__device__ void metzger_shape_lane(MzTables& T, int slot, int col, const double* p, const BandView& b,
                                   const double* cst, double* s5) {
    int j_start;
    double l_peak;
    bool ok = mz_sweep(T, p, slot, col, l_peak);
    bool valid = ok && l_peak > 0.0 && isfinite(l_peak);
    double sw = 0, sy = 0, sf = 0, syf = 0, sff = 0;
    for (int j = 0; j < b.n; j++) {
        if (valid && !(b.t[j] - p[3] <= 0.0)) break;
        if (b.up[j]) continue;
        double w = cst[3 * j];
        sw += w; sy += w * b.f[j];
    }
    if (valid) {
        struct Sums {
            const BandView* b;
            const double* cst;
            double lpk, sw, sy, sf, syf, sff;
            __device__ void operator()(int j, double l) {
                if (b->up[j]) return;
                double sh = l / lpk;
                if (!isfinite(sh)) return;
                double w = cst[3 * j], fj = b->f[j];
                sw += w; sy += w * fj; sf += w * sh; syf += w * fj * sh; sff += w * sh * sh;
            }
        } su{&b, cst, l_peak, sw, sy, sf, syf, sff};
        mz_visit(T, slot, col, p[3], b.t, b.n, j_start, su);
        sw = su.sw; sy = su.sy; sf = su.sf; syf = su.syf; sff = su.sff;
    }
    s5[0] = sw; s5[1] = sy; s5[2] = sf; s5[3] = syf; s5[4] = sff;
}

// Magnitude-space chi2 of a MetzgerKN band by one warp: the prediction at mu
// (table 0), or at the PSO parameters where fewer than half are positive.
__device__ double metzger_mag_chi2(MzTables& T, const BandStats& bs, const BandView& b, const BandOut& o,
                                   const double* mu) {
    const int lane = threadIdx.x & 31;
    constexpr int np = 5, PSO_SLOT = 24;
    double l_peak;
    int valid = 0, slot = 0, col = 62;
    const double* use = mu;
    auto sweep = [&]() {
        int v = 0;
        if (lane == 0) v = mz_sweep(T, use, slot, col, l_peak) && !(l_peak <= 0.0 || !isfinite(l_peak));
        __syncwarp();
        l_peak = __shfl_sync(FULL, l_peak, 0);
        valid = __shfl_sync(FULL, v, 0);
    };
    auto pred = [&](int i) {
        const double ph = b.t[i] - use[3];
        if (!valid || ph <= 0.0) return 0.0;
        int g = 0;
        for (int step = 128; step; step >>= 1)
            if (g + step <= MZ_NG && ph > T.row[g + step - 1][0][slot]) g += step;
        return mz_interp(T, slot, col, ph, g) / l_peak;
    };
    sweep();
    int npos = 0;
    for (int i = lane; i < b.n; i += 32) npos += (pred(i) * b.peak > 0.0) ? 1 : 0;
    for (int k = 16; k; k >>= 1) npos += __shfl_xor_sync(FULL, npos, k);
    double pso[MAXP];
    // the joint fit always takes mu (src/parametric.rs:4057-4073)
    if (npos < b.n / 2 && !bs.joint) {
        for (int j = 0; j < np; j++) pso[j] = o.pso_params[j];
        use = pso;
        slot = PSO_SLOT;
        col = 63;
        __syncwarp();
        mz_tabulate(T, 1, bs.t_last, [&](int) { return pso[3]; }, lane, 32, PSO_SLOT);
        __syncwarp();
        sweep();
    }
    double msum = 0.0;
    int mcount = 0;
    for (int i = lane; i < b.n; i += 32) {
        double pf = pred(i) * b.peak;
        if (pf > 0.0 && b.f[i] > 0.0) {
            double mpred = -2.5 * log10(pf) + 23.9;
            double merr = 1.0857 * b.fe[i] / b.f[i];
            if (merr > 0.0) {
                double r = b.mag[i] - mpred;
                msum += r * r / (merr * merr);
                mcount++;
            }
        }
    }
    msum = wsum(msum);
    for (int k = 16; k; k >>= 1) mcount += __shfl_xor_sync(FULL, mcount, k);
    return mcount > 0 ? msum / (double)mcount : NAN;
}

// profile_t0_refine, profile_refine_all and the magnitude chi2 of the
// MetzgerKN bands (np = 5, t0 = p[3], sigma_extra = p[4]; no baseline
// parameter).  The sequential decisions run uniformly on the gathered values.
// On the t0 grid warp 0 takes the profiled amplitude and its likelihood while
// warp 1 takes the likelihoods at mu; then warps 0 and 1 take the 61
// all-parameter points while warp 2 takes the magnitude chi2.  Bound by the
// FP64 pipe.  The refinements of 600 bands x 8 models, GB300: 70 ms with a warp
// a MetzgerKN band, each lane integrating its own ODE twice; 21 ms now.
__global__ void __launch_bounds__(MZ_BLOCK) refine_metzger_kernel(DeviceBatch d) {
    extern __shared__ __align__(16) unsigned char mz_raw[];
    MzTables& T = *reinterpret_cast<MzTables*>(mz_raw);
    __shared__ double s_ll[MZ_LANES], s_ell[32], s_mag;
    constexpr int m = METZGER, np = 5, se = 4, t0i = 3, NG = 25, NE = 1 + 4 * 15;
    static_assert(NG <= MZ_SLOTS && NE < 62 && 1 + 15 <= 24, "MetzgerKN scan tables");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_metzger = d.ctr->band_hist[0];  // band_order's first (band_order_kernel)
    if (tid == 0) T.lum = reinterpret_cast<double(*)[MZ_LANES]>(d.mz_lum + blockIdx.x * MZ_LUM);
    for (int ib = blockIdx.x; ib < n_metzger; ib += gridDim.x) {
        const int band = d.band_order[ib];
        const BandStats bs = d.stats[band];
        BandOut& o = d.out[band];
        const BandView b = band_view(d, bs);
        double* cst = d.scratch64 + 5 * bs.off;
        double mu[MAXP], ls[MAXP];
        for (int j = 0; j < np; j++) { mu[j] = o.mu[j]; ls[j] = o.log_sigma[j]; }
        scan_constants(b, exp(2.0 * mu[se]), cst, tid, MZ_BLOCK);
        const double t0_lo = bs.t_first - 30.0, t0_hi = bs.t_peak_all + 5.0;
        if (t0_lo < t0_hi) {
            auto grid = [&](int gi) { return t0_lo + (t0_hi - t0_lo) * (double)gi / (double)(NG - 1); };
            mz_tabulate(T, NG, bs.t_last, grid, tid, MZ_BLOCK);
            __syncthreads();
            if (warp < 2 && lane < NG) {
                double p[MAXP];
                for (int j = 0; j < np; j++) p[j] = mu[j];
                p[t0i] = grid(lane);
                if (warp == 0) {
                    // profiled amplitude at each grid t0, then its log-likelihood (rescaled)
                    double saved_la = p[0];
                    p[0] = 0.0;
                    double s5[5];
                    metzger_shape_lane(T, lane, lane, p, b, cst, s5);
                    double syf = s5[3], sff = s5[4];
                    if (sff > 1e-20 && syf / sff > 1e-10) p[0] = log(syf / sff);
                    else p[0] = saved_la;
                    s_ll[lane] = metzger_ll_lane(T, lane, lane, p, b, cst, true);
                } else {
                    // log-likelihood at mu with t0 on each grid point (no rescale)
                    s_ell[lane] = metzger_ll_lane(T, lane, 32 + lane, p, b, cst, false);
                }
            }
            __syncthreads();
            double best_t0 = mu[t0i], best_ll = -INFINITY;
            for (int gi = 0; gi < NG; gi++) {
                double l = s_ll[gi];
                if (l > best_ll) { best_ll = l; best_t0 = grid(gi); }
            }
            double lo1 = best_t0, hi1 = best_t0, thr = best_ll - 0.5;
            for (int gi = NG - 1; gi >= 0; gi--) {
                double t0 = grid(gi);
                if (t0 >= best_t0) continue;
                if (s_ell[gi] >= thr) lo1 = t0;
                else break;
            }
            for (int gi = 0; gi < NG; gi++) {
                double t0 = grid(gi);
                if (t0 <= best_t0) continue;
                if (s_ell[gi] >= thr) hi1 = t0;
                else break;
            }
            mu[t0i] = best_t0;
            ls[t0i] = log(fmax((hi1 - lo1) / 2.0, 0.1));
        }
        __syncthreads();
        // profile_refine_all: evaluation 0 = mu, 1 + 15 j + gi = parameter j
        // on grid point gi; table 0 = mu's t0, 1 + gi = t0's grid
        auto scan = [&](int j, int gi) {
            double slo = c_lo[m][j], shi = c_hi[m][j];
            return slo + (shi - slo) * (double)gi / 14.0;
        };
        mz_tabulate(T, 16, bs.t_last, [&](int k) { return k == 0 ? mu[t0i] : scan(t0i, k - 1); }, tid, MZ_BLOCK);
        __syncthreads();
        if (tid < NE) {
            double p[MAXP];
            for (int k = 0; k < np; k++) p[k] = mu[k];
            int slot = 0;
            if (tid > 0) {
                int j = (tid - 1) / 15, gi = (tid - 1) % 15;
                p[j] = scan(j, gi);
                if (j == t0i) slot = 1 + gi;
            }
            s_ll[tid] = metzger_ll_lane(T, slot, tid, p, b, cst, false);
        }
        if (warp == 2) {
            const double mc = metzger_mag_chi2(T, bs, b, o, mu);
            if (lane == 0) s_mag = mc;
        }
        __syncthreads();
        if (tid == 0) {
            double thr = s_ll[0] - 0.5;
            for (int j = 0; j < np; j++) {
                if (j == se) continue;
                double mu_j = mu[j], svi_sigma = exp(ls[j]);
                double slo = c_lo[m][j], shi = c_hi[m][j];
                if (shi - slo < 1e-10) continue;
                double l1 = mu_j, h1 = mu_j;
                for (int gi = 0; gi < 15; gi++) {
                    double val = scan(j, gi);
                    if (s_ll[1 + j * 15 + gi] >= thr) { l1 = fmin(l1, val); h1 = fmax(h1, val); }
                }
                double prof = fmax((h1 - l1) / 2.0, 1e-6);
                ls[j] = log(fmax(fmax(svi_sigma, prof), c_pop_w[m][j]));
            }
            for (int j = 0; j < np; j++) { o.mu[j] = mu[j]; o.log_sigma[j] = ls[j]; }
            o.mag_chi2 = s_mag;
        }
        __syncthreads();
    }
}

// symmetric_eigen (Jacobi), src/parametric.rs:2517-2587
__device__ void jacobi_eigen(double* a, int n, double* ev, double* V) {
    for (int i = 0; i < n * n; i++) V[i] = 0.0;
    for (int i = 0; i < n; i++) V[i * n + i] = 1.0;
    int max_iter = 100 * n * n;
    for (int itr = 0; itr < max_iter; itr++) {
        double mv = 0.0;
        int p = 0, q = 1;
        for (int i = 0; i < n; i++)
            for (int j = i + 1; j < n; j++) {
                double v = fabs(a[i * n + j]);
                if (v > mv) { mv = v; p = i; q = j; }
            }
        double app = a[p * n + p], aqq = a[q * n + q], apq = a[p * n + q];
        // the reference stops below 1e-15 absolute, which a Hessian with
        // entries ~1e6 never reaches (its rotations leave ~1e-10): it then
        // runs all 100 n^2 rotations, each of them below rounding level once
        // the largest off-diagonal element is below 1e-15 of its diagonal
        // pair.  Stopping there too changes the eigenvalues at rounding level
        // and spares the FP64 trigonometry of those rotations.
        if (mv < 1e-15 || mv <= 1e-15 * sqrt(fabs(app * aqq))) break;
        double th = fabs(app - aqq) < 1e-30 ? 0.78539816339744830962 : 0.5 * atan(2.0 * apq / (app - aqq));
        double c = cos(th), s = sin(th);
        for (int i = 0; i < n; i++) {
            double aip = a[i * n + p], aiq = a[i * n + q];
            a[i * n + p] = c * aip + s * aiq;
            a[i * n + q] = -s * aip + c * aiq;
        }
        for (int j = 0; j < n; j++) {
            double apj = a[p * n + j], aqj = a[q * n + j];
            a[p * n + j] = c * apj + s * aqj;
            a[q * n + j] = -s * apj + c * aqj;
        }
        a[p * n + p] = c * c * app + 2.0 * c * s * apq + s * s * aqq;
        a[q * n + q] = s * s * app - 2.0 * c * s * apq + c * c * aqq;
        a[p * n + q] = 0.0;
        a[q * n + p] = 0.0;
        for (int i = 0; i < n; i++) {
            double vip = V[i * n + p], viq = V[i * n + q];
            V[i * n + p] = c * vip + s * viq;
            V[i * n + q] = -s * vip + c * viq;
        }
    }
    for (int i = 0; i < n; i++) ev[i] = a[i * n + i];
}

// ---------------------------------------------------------------------------
// The order in which the per-band kernels take the bands (band_order[warp]):
// a counting sort by selected model and length.  MetzgerKN, whose uncertainty
// and refinements cost the most, is first, the unfitted bands last; no result
// depends on the order.
//   - A batch that keeps the warp slots full goes model by model, so that the
//     warps resident on an SM run one model's code, and inside a model longest
//     first, in classes of 8 observations: a block's four bands then end
//     together (10,000 uneven sources, SVI 178 -> 162 ms, refinements 41 -> 28
//     against bands of a model in any order; longest first over all models
//     221 and 59).
//   - One of up to 4,096 bands waits for its longest bands: they come first, in
//     classes of 64 observations over all models (1,000 sources, SVI 38 ms
//     against 43 model by model, 2,400 given pairs 33 against 37 in all).  At
//     9,000 bands SVI is 60 against 68 ms, but the refinements 20 against 12.
// ---------------------------------------------------------------------------
constexpr int BO_LEN = 64, BO_KEYS = 9 * BO_LEN;
__device__ __forceinline__ int band_order_key(const DeviceBatch& d, int b, bool by_length) {
    const int m = d.out[b].model;
    const BandStats& st = d.stats[b];
    const int g = !st.valid || m < 0 ? 8 : m == METZGER ? 0 : 1 + m;
    const int len = BO_LEN - 1 - min(st.n >> (by_length ? 6 : 3), BO_LEN - 1);
    return by_length && g > 0 && g < 8 ? BO_LEN + 7 * len + g - 1 : g * BO_LEN + len;
}
// One block: the list is a few reads a band, less than two more launches.  On
// return band_hist[0] is the number of MetzgerKN bands (band_order's first).
constexpr int BO_BLOCK = 1024;
__global__ void __launch_bounds__(BO_BLOCK) band_order_kernel(DeviceBatch d, bool by_length) {
    __shared__ int pos[BO_KEYS];
    const int tid = threadIdx.x;
    for (int k = tid; k < BO_KEYS; k += BO_BLOCK) pos[k] = 0;
    __syncthreads();
    for (int b = tid; b < d.n_bands; b += BO_BLOCK) atomicAdd(&pos[band_order_key(d, b, by_length)], 1);
    __syncthreads();
    if (tid < 32) {  // a lane's neighbouring keys, then the lanes' sums
        constexpr int PER = BO_KEYS / 32;
        int sum = 0;
        for (int k = 0; k < PER; k++) sum += pos[tid * PER + k];
        int run = sum;
        for (int o = 1; o < 32; o *= 2) {
            const int v = __shfl_up_sync(FULL, run, o);
            if (tid >= o) run += v;
        }
        run -= sum;
        for (int k = 0; k < PER; k++) {
            const int v = pos[tid * PER + k];
            pos[tid * PER + k] = run;
            run += v;
        }
        __syncwarp();
        if (tid == 0) d.ctr->band_hist[0] = pos[BO_LEN];
    }
    __syncthreads();
    for (int b = tid; b < d.n_bands; b += BO_BLOCK) d.band_order[atomicAdd(&pos[band_order_key(d, b, by_length)], 1)] = b;
}
void launch_band_order(const DeviceBatch& d, cudaStream_t s) {
    if (d.n_bands == 0) return;
    band_order_kernel<<<1, BO_BLOCK, 0, s>>>(d, d.n_bands <= 4096);
}

// neg_log_posterior (src/parametric.rs:2464-2511) of MetzgerKN at one
// parameter vector, by one lane: the terms in observation order, as the
// reference sums them.
__device__ double metzger_nlp_lane(MzTables& T, int slot, int col, const BandView& b, const double* p) {
    MzPeak pk{b.up, -INFINITY};
    int j_start = b.n;
    double l_peak;
    bool ok = mz_sweep(T, p, slot, col, l_peak) && l_peak > 0.0 && isfinite(l_peak);
    if (ok) mz_visit(T, slot, col, p[3], b.t, b.n, j_start, pk);
    // the predictions before the first visited observation are 0
    double mx = pk.mx / l_peak;
    for (int j = 0; j < (ok ? j_start : b.n); j++)
        if (!b.up[j]) mx = ok ? fmax(mx, 0.0) : 0.0;
    if (!ok) mx = b.n > 0 ? 0.0 : -INFINITY;
    const double scale = (mx > 1e-10 && isfinite(mx)) ? fmin(fmax(1.0 / mx, 0.1), 10.0) : 1.0;
    const double se2 = exp(2.0 * p[se_idx_of(METZGER)]);
    struct Terms {
        const BandView* b;
        double peak, scale, se2, nll;
        int nonfinite;
        __device__ void term(int i, double pr) {
            if (!isfinite(pr)) { nonfinite = 1; return; }
            const double tv = b->var[i] + se2;
            if (b->up[i]) nll -= log_normal_cdf_f64((b->uf[i] - pr) / sqrt(tv));
            else {
                const double dd = pr - b->f[i];
                nll += 0.5 * (dd * dd / tv + log(2.0 * 3.14159265358979323846 * tv));
            }
        }
        __device__ void operator()(int j, double l) { term(j, (l / peak) * scale); }
    } tm{&b, l_peak, scale, se2, 0.0, 0};
    if (ok) {
        for (int j = 0; j < j_start; j++) tm.term(j, 0.0 * scale);
        mz_visit(T, slot, col, p[3], b.t, b.n, j_start, tm);
    } else {
        for (int j = 0; j < b.n; j++) tm.term(j, 0.0 * scale);
    }
    if (tm.nonfinite) return 1e99;
    double nlp = 0.0;
    for (int j = 0; j < n_params_of(METZGER); j++) {
        const double w = c_pri_w[METZGER][j], dd = p[j] - c_pri_c[METZGER][j];
        nlp += 0.5 * dd * dd / (w * w);
    }
    return tm.nll + nlp;
}

// Analytic Hessian of neg_log_posterior (src/parametric.rs:2464-2507) over the
// shape parameters idx[0..ns), sigma_extra held fixed as laplace_fit holds
// it (:2623-2693).  Forward mode over the analytic gradient: column k is the
// derivative along parameter idx[k] of
//   sum_i dl_i/dpred * grad pred_i + the prior's gradient,
// i.e. sum_i (d2l_i/dpred2 g_j g_k + dl_i/dpred h_jk) + the prior's 1 / w^2
// on the diagonal, with g = grad pred and its column h from the model
// gradient evaluated on Dual numbers, and the upper-limit term's log-CDF
// derivatives from a second-order Taylor number.  The reference takes the
// same matrix by central differences of its cost (4 evaluations per pair,
// step 1e-4 max(|theta|, 1)).  Models 0..6; warp-collective, lanes over
// observations.  Returns false when a prediction or an entry is not finite
// (the caller then takes the reference's finite differences).
__device__ bool laplace_hessian_analytic(int m, const BandView& b, const double* mp, const int* idx, int ns,
                                         double* H) {
    const int lane = threadIdx.x & 31;
    const int nf = n_params_of(m), se = se_idx_of(m);
    const double se2 = exp(2.0 * mp[se]);
    int bad = 0;
    for (int sk = 0; sk < ns; sk++) {
        Dual q[MAXP];
        for (int j = 0; j < nf; j++) q[j] = Dual(mp[j], j == idx[sk] ? 1.0 : 0.0);
        double col[MAXP];
        for (int sj = 0; sj < ns; sj++) col[sj] = 0.0;
        for (int i = lane; i < b.n; i += 32) {
            Dual g[MAXP];
            model_grad_t<Dual>(m, q, Dual(b.t[i]), g);
            const double pr = eval_model_f64(m, mp, b.t[i]);
            if (!isfinite(pr)) {
                bad = 1;
                continue;
            }
            const double tv = b.var[i] + se2;
            double a1, a2;  // dl / dpred and d2l / dpred2
            if (b.up[i]) {
                // l = -log Phi(z), z = (u - pred) / s
                const double s = sqrt(tv);
                const Jet2 L = log_normal_cdf_jet(Jet2((b.uf[i] - pr) / s, 1.0, 0.0));
                a1 = L.c1 / s;
                a2 = -2.0 * L.c2 / tv;
            } else {
                // l = ((pred - y)^2 / tv + ln(2 pi tv)) / 2
                a1 = (pr - b.f[i]) / tv;
                a2 = 1.0 / tv;
            }
            const double gk = g[idx[sk]].v;
            for (int sj = 0; sj < ns; sj++) col[sj] += a2 * g[idx[sj]].v * gk + a1 * g[idx[sj]].d;
        }
        for (int sj = 0; sj < ns; sj++) {
            double v = wsum(col[sj]);
            if (sj == sk) {
                const double w = c_pri_w[m][idx[sj]];
                v += 1.0 / (w * w);
            }
            H[sj * ns + sk] = v;
        }
    }
    for (int a = 0; a < ns; a++)
        for (int c = a; c < ns; c++) {
            const double v = 0.5 * (H[a * ns + c] + H[c * ns + a]);
            H[a * ns + c] = v;
            H[c * ns + a] = v;
            if (!isfinite(v)) bad = 1;
        }
    return !__any_sync(FULL, bad);
}

// sigma from the Hessian's inverse (Jacobi eigen-decomposition, eigenvalue
// clamp 1e-6), and the band's outputs (:2664-2693); one thread.
__device__ void laplace_write(BandOut& o, int m, const double* mp, double* H, int ns, double f0) {
    const int nf = n_params_of(m), se = se_idx_of(m);
    double ev[MAXP], V[36];
    jacobi_eigen(H, ns, ev, V);
    double sls[MAXP];
    for (int i = 0; i < ns; i++) {
        double sum = 0.0;
        for (int k = 0; k < ns; k++) sum += V[i * ns + k] * V[i * ns + k] * (1.0 / fmax(ev[k], 1e-6));
        sls[i] = 0.5 * log(fmax(sum, 1e-30));
    }
    int s2 = 0;
    for (int i = 0; i < MAXP; i++) {
        o.mu[i] = i < nf ? mp[i] : NAN;
        if (i >= nf) o.log_sigma[i] = NAN;
        else if (i == se) o.log_sigma[i] = log(c_pri_w[m][i]);
        else o.log_sigma[i] = sls[s2++];
    }
    o.elbo = -f0;
    o.svi_steps = 0;
}

__global__ void laplace_kernel(DeviceBatch d) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= d.n_bands) return;
    warp = d.band_order[warp];
    BandStats bs = d.stats[warp];
    BandOut& o = d.out[warp];
    if (!bs.valid || o.model < 0 || o.model == METZGER) return;
    BandView b = band_view(d, bs);
    int m = o.model, nf = n_params_of(m), se = se_idx_of(m);
    double mp[MAXP];
    for (int j = 0; j < nf; j++) mp[j] = o.pso_params[j];
    int idx[MAXP], ns = 0;
    for (int i = 0; i < nf; i++)
        if (i != se) idx[ns++] = i;
    double H[36];
    // the analytic Hessian (forward over the adjoint); points with non-finite
    // predictions keep the reference's central differences
    const double f0 = neg_log_posterior_w(m, b, mp);
    const bool analytic = f0 < 1e99 && laplace_hessian_analytic(m, b, mp, idx, ns, H);
    for (int si = 0; si < ns && !analytic; si++) {
        int i = idx[si];
        double hi = 1e-4 * fmax(fabs(mp[i]), 1.0);
        for (int sj = si; sj < ns; sj++) {
            int j = idx[sj];
            double hj = 1e-4 * fmax(fabs(mp[j]), 1.0);
            double q[MAXP];
            double fv[4];
            const double si_[4] = {1, 1, -1, -1}, sj_[4] = {1, -1, 1, -1};
            for (int k = 0; k < 4; k++) {
                for (int t = 0; t < nf; t++) q[t] = mp[t];
                q[i] += si_[k] * hi;
                q[j] += sj_[k] * hj;
                fv[k] = neg_log_posterior_w(m, b, q);
            }
            double h = (fv[0] - fv[1] - fv[2] + fv[3]) / (4.0 * hi * hj);
            H[si * ns + sj] = h;
            H[sj * ns + si] = h;
        }
    }
    if ((threadIdx.x & 31) == 0) laplace_write(o, m, mp, H, ns, f0);
}

// MetzgerKN, whose gradient is itself a finite difference in the reference,
// keeps the reference's central differences of the cost (:2623-2693), a block
// per band with the stencil's points spread over its lanes: point 0 is the MAP
// (its cost f0), points 1 + 4k .. 4 + 4k the four evaluations of the k-th pair
// (si <= sj).  The 41 points take 7 values of t0 (metzger_block.cuh).  A basic
// batch with one MetzgerKN band, GB300: Laplace 6.6 -> 1.9 ms.
__global__ void __launch_bounds__(MZ_BLOCK) laplace_metzger_kernel(DeviceBatch d) {
    extern __shared__ __align__(16) unsigned char mz_raw[];
    MzTables& T = *reinterpret_cast<MzTables*>(mz_raw);
    __shared__ double s_c[MZ_LANES];
    constexpr int m = METZGER, np = 5, ns = 4, t0i = 3;  // shape parameters 0 .. 3
    constexpr int npts = 1 + 2 * ns * (ns + 1);
    static_assert(npts <= MZ_LANES && n_params_of(m) == np && se_idx_of(m) == ns, "MetzgerKN stencil");
    const int tid = threadIdx.x;
    const int n_metzger = d.ctr->band_hist[0];
    if (tid == 0) T.lum = reinterpret_cast<double(*)[MZ_LANES]>(d.mz_lum + blockIdx.x * MZ_LUM);
    for (int ib = blockIdx.x; ib < n_metzger; ib += gridDim.x) {
        const int band = d.band_order[ib];
        const BandStats bs = d.stats[band];
        BandOut& o = d.out[band];
        const BandView b = band_view(d, bs);
        double mp[MAXP];
        for (int j = 0; j < np; j++) mp[j] = o.pso_params[j];
        auto step = [&](int i) { return 1e-4 * fmax(fabs(mp[i]), 1.0); };
        // t0 of table k: 0 the MAP's, 1 and 2 one step up and down, 3 + s4 both
        // perturbations of the (t0, t0) pair
        mz_tabulate(T, 7, bs.t_last, [&](int k) {
            double t0 = mp[t0i];
            const double h = step(t0i);
            if (k == 1 || k == 2) t0 += (k == 1 ? 1.0 : -1.0) * h;
            if (k >= 3) {
                const int s4 = k - 3;
                t0 += (s4 < 2 ? 1.0 : -1.0) * h;
                t0 += ((s4 & 1) == 0 ? 1.0 : -1.0) * h;
            }
            return t0;
        }, tid, MZ_BLOCK);
        __syncthreads();
        if (tid < npts) {
            double q[MAXP];
            for (int t = 0; t < np; t++) q[t] = mp[t];
            int slot = 0;
            if (tid > 0) {
                int k = (tid - 1) >> 2, si = 0;
                while (k >= ns - si) { k -= ns - si; si++; }
                const int sj = si + k, s4 = (tid - 1) & 3;
                const double hi = step(si), hj = step(sj);
                q[si] += (s4 < 2 ? 1.0 : -1.0) * hi;
                q[sj] += ((s4 & 1) == 0 ? 1.0 : -1.0) * hj;
                if (si == t0i) slot = 3 + s4;
                else if (sj == t0i) slot = (s4 & 1) == 0 ? 1 : 2;
            }
            s_c[tid] = metzger_nlp_lane(T, slot, tid, b, q);
        }
        __syncthreads();
        if (tid == 0) {
            double H[36];
            int k = 0;
            for (int si = 0; si < ns; si++) {
                const double hi = step(si);
                for (int sj = si; sj < ns; sj++, k++) {
                    const double hj = step(sj);
                    const double h = (s_c[1 + 4 * k] - s_c[2 + 4 * k] - s_c[3 + 4 * k] + s_c[4 + 4 * k]) / (4.0 * hi * hj);
                    H[si * ns + sj] = h;
                    H[sj * ns + si] = h;
                }
            }
            laplace_write(o, m, mp, H, ns, s_c[0]);
        }
        __syncthreads();
    }
}

void launch_laplace(const DeviceBatch& d, cudaStream_t s) {
    if (d.n_bands == 0) return;
    int64_t threads = (int64_t)d.n_bands * 32;
    laplace_kernel<<<(int)((threads + 127) / 128), 128, 0, s>>>(d);
}
void launch_laplace_metzger(const DeviceBatch& d, cudaStream_t s) {
    if (d.n_bands == 0) return;
    laplace_metzger_kernel<<<std::min(d.n_bands, d.num_sms), MZ_BLOCK, sizeof(MzTables), s>>>(d);
}

// profile_t0_refine + profile_refine_all + mag chi2 of the models other than
// MetzgerKN, a warp per band: FP32 model evaluation, FP64 terms
#ifndef LCF_REFINE_BLOCK
#define LCF_REFINE_BLOCK 128
#endif
__global__ void refine_kernel(DeviceBatch d) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (warp >= d.n_bands) return;
    warp = d.band_order[warp];
    BandStats bs = d.stats[warp];
    BandOut& o = d.out[warp];
    if (!bs.valid || o.model < 0 || o.model == METZGER) return;
    BandView b = band_view(d, bs);
    int m = o.model, np = n_params_of(m), se = se_idx_of(m), t0i = t0_idx_of(m);
    double* scr = d.scratch64 + 5 * bs.off;
    double mu[MAXP], ls[MAXP];
    for (int j = 0; j < np; j++) { mu[j] = o.mu[j]; ls[j] = o.log_sigma[j]; }
    const float4* obs = d.obs + bs.off;
    scan_constants(b, exp(2.0 * mu[se]), scr, lane, 32);
    __syncwarp();
    auto scan_ll = [&](const double* p) { return band_ll_fast(m, p, obs, b, scr); };
    // ---- profile_t0_refine
    {
        double t0_lo = bs.t_first - 30.0, t0_hi = bs.t_peak_all + 5.0;
        if (t0_lo < t0_hi) {
            const int NG = 25;
            bool has_b = (m == BAZIN || m == TDE);
            double best_t0 = mu[t0i], best_ll = -INFINITY;
            for (int gi = 0; gi < NG; gi++) {
                double t0 = t0_lo + (t0_hi - t0_lo) * (double)gi / (double)(NG - 1);
                double p[MAXP];
                for (int j = 0; j < np; j++) p[j] = mu[j];
                p[t0i] = t0;
                double saved_la = p[0];
                p[0] = 0.0;
                double saved_b = 0.0;
                if (has_b) { saved_b = p[1]; p[1] = 0.0; }
                double s5[5];
                shape_sums_fast(m, p, obs, b, scr, s5);
                const double sw = s5[0], sy = s5[1], sf = s5[2], syf = s5[3], sff = s5[4];
                if (has_b) {
                    double det = sw * sff - sf * sf;
                    if (fabs(det) > 1e-20) {
                        double a_opt = (sw * syf - sf * sy) / det, b_opt = (sff * sy - sf * syf) / det;
                        if (a_opt > 1e-10) { p[0] = log(a_opt); p[1] = b_opt; }
                        else { p[0] = saved_la; p[1] = saved_b; }
                    } else { p[0] = saved_la; p[1] = saved_b; }
                } else {
                    if (sff > 1e-20 && syf / sff > 1e-10) p[0] = log(syf / sff);
                    else p[0] = saved_la;
                }
                double ll = scan_ll(p);
                if (ll > best_ll) { best_ll = ll; best_t0 = t0; }
            }
            double lo1 = best_t0, hi1 = best_t0, thr = best_ll - 0.5;
            for (int gi = NG - 1; gi >= 0; gi--) {
                double t0 = t0_lo + (t0_hi - t0_lo) * (double)gi / (double)(NG - 1);
                if (t0 >= best_t0) continue;
                double p[MAXP];
                for (int j = 0; j < np; j++) p[j] = mu[j];
                p[t0i] = t0;
                if (scan_ll(p) >= thr) lo1 = t0;
                else break;
            }
            for (int gi = 0; gi < NG; gi++) {
                double t0 = t0_lo + (t0_hi - t0_lo) * (double)gi / (double)(NG - 1);
                if (t0 <= best_t0) continue;
                double p[MAXP];
                for (int j = 0; j < np; j++) p[j] = mu[j];
                p[t0i] = t0;
                if (scan_ll(p) >= thr) hi1 = t0;
                else break;
            }
            mu[t0i] = best_t0;
            ls[t0i] = log(fmax((hi1 - lo1) / 2.0, 0.1));
        }
    }
    // ---- profile_refine_all
    {
        double map_ll = scan_ll(mu);
        double thr = map_ll - 0.5;
        for (int j = 0; j < np; j++) {
            if (j == se) continue;
            double mu_j = mu[j];
            double svi_sigma = exp(ls[j]);
            double slo = c_lo[m][j], shi = c_hi[m][j];
            if (shi - slo < 1e-10) continue;
            double l1 = mu_j, h1 = mu_j;
            for (int gi = 0; gi < 15; gi++) {
                double val = slo + (shi - slo) * (double)gi / 14.0;
                double p[MAXP];
                for (int k = 0; k < np; k++) p[k] = mu[k];
                p[j] = val;
                double ll = scan_ll(p);
                if (ll >= thr) { l1 = fmin(l1, val); h1 = fmax(h1, val); }
            }
            double prof = fmax((h1 - l1) / 2.0, 1e-6);
            double prior_sigma = c_pop_w[m][j];
            ls[j] = log(fmax(fmax(svi_sigma, prof), prior_sigma));
        }
    }
    // ---- magnitude-space chi2 with the refined mu (PSO params if fewer
    // than half of the predictions are positive)
    double msum = 0.0;
    int mcount = 0;
    {
        Model64 P;
        P.init(m, mu);
        int npos = 0;
        for (int i = lane; i < b.n; i += 32) npos += (P.eval(b.t[i], nullptr) * b.peak > 0.0) ? 1 : 0;
        for (int k = 16; k; k >>= 1) npos += __shfl_xor_sync(FULL, npos, k);
        __syncwarp();
        const double* use = mu;
        double pso[MAXP];
        // the joint fit always takes mu (src/parametric.rs:4057-4073)
        if (npos < b.n / 2 && !bs.joint) {
            for (int j = 0; j < np; j++) pso[j] = o.pso_params[j];
            use = pso;
        }
        Model64 Q;
        Q.init(m, use);
        for (int i = lane; i < b.n; i += 32) {
            double pf = Q.eval(b.t[i], nullptr) * b.peak;
            if (pf > 0.0 && b.f[i] > 0.0) {
                double mpred = -2.5 * log10(pf) + 23.9;
                double merr = 1.0857 * b.fe[i] / b.f[i];
                if (merr > 0.0) {
                    double r = b.mag[i] - mpred;
                    msum += r * r / (merr * merr);
                    mcount++;
                }
            }
        }
        msum = wsum(msum);
        for (int k = 16; k; k >>= 1) mcount += __shfl_xor_sync(FULL, mcount, k);
    }
    if (lane == 0) {
        for (int j = 0; j < np; j++) { o.mu[j] = mu[j]; o.log_sigma[j] = ls[j]; }
        o.mag_chi2 = mcount > 0 ? msum / (double)mcount : NAN;
    }
}

void launch_refine(const DeviceBatch& d, cudaStream_t s) {
    if (d.n_bands == 0) return;
    int64_t threads = (int64_t)d.n_bands * 32;
    refine_kernel<<<(int)((threads + LCF_REFINE_BLOCK - 1) / LCF_REFINE_BLOCK), LCF_REFINE_BLOCK, 0, s>>>(d);
}
// The MetzgerKN bands of the refinements: one block per SM (the tables take
// half of its shared memory), the grid draining band_order's MetzgerKN bands.
void launch_refine_metzger(const DeviceBatch& d, cudaStream_t s) {
    if (d.n_bands == 0) return;
    refine_metzger_kernel<<<std::min(d.n_bands, d.num_sms), MZ_BLOCK, sizeof(MzTables), s>>>(d);
}
int finalize_init_attributes() {
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const cudaFuncAttribute split = cudaFuncAttributePreferredSharedMemoryCarveout;  // as the SVI kernels (polish.cu)
    cudaError_t e = cudaFuncSetAttribute(refine_metzger_kernel, a, (int)sizeof(MzTables));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(laplace_metzger_kernel, a, (int)sizeof(MzTables));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(refine_metzger_kernel, split, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(laplace_metzger_kernel, split, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(refine_kernel, split, cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(laplace_kernel, split, cudaSharedmemCarveoutMaxShared);
    return (int)e;
}
int64_t mz_lum_doubles(int num_sms) { return (int64_t)num_sms * MZ_LUM; }

// ---------------------------------------------------------------------------
// Profile t0 search (SVI mode, rank-0 band): task builders and pickers.
// Coarse: 5 runs on linspace(t0_min, t0_max, 5); fine: 3 runs on
// linspace(best_t0 -/+ 0.5 clipped); results in t0 slots (band * 8 + k).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double lin_at(double a, double b, int n, int i) {
    return n <= 1 ? a : a + (double)i * ((b - a) / (double)(n - 1));
}

__global__ void t0_build_kernel(DeviceBatch d, int slot, int fine, int64_t t0_base) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= d.n_bands) return;
    BandStats bs = d.stats[b];
    BandOut& o = d.out[b];
    if (!bs.valid || bs.rank != 0 || o.model < 0 || bs.joint) return;  // no t0 search in the joint fit
    int m = o.model, t0i = t0_idx_of(m);
    double* ts = d.t0_state + 3 * (int64_t)b;
    if (!fine) {
        double pilot = o.pso_params[t0i];
        ts[0] = fmax(pilot - 5.0, bs.t_first - 10.0);
        ts[1] = pilot + 5.0;
        ts[2] = pilot;
    }
    double t0_min = ts[0], t0_max = ts[1];
    int cnt = fine ? 3 : 5;
    double a = t0_min, z = t0_max;
    if (fine) {
        a = fmax(ts[2] - 0.5, t0_min);
        z = fmin(ts[2] + 0.5, t0_max);
    }
    int base = atomicAdd(&d.ctr->task_count[slot], cnt);
    for (int k = 0; k < cnt; k++) {
        PsoTask t;
        t.band = b;
        t.kind = (int16_t)m;
        t.restart = 0;
        t.flags = TASK_T0_FIXED;
        t.out = (int)(t0_base + (int64_t)b * 8 + (fine ? 5 : 0) + k);
        t.aux = -1;
        t.t0_fixed = lin_at(a, z, cnt, k);
        d.tasks[slot][base + k] = t;
    }
}

__global__ void t0_pick_kernel(DeviceBatch d, int fine, int64_t t0_base) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= d.n_bands) return;
    BandStats bs = d.stats[b];
    BandOut& o = d.out[b];
    if (!bs.valid || bs.rank != 0 || o.model < 0 || bs.joint) return;
    int m = o.model, np = n_params_of(m), t0i = t0_idx_of(m);
    double* ts = d.t0_state + 3 * (int64_t)b;
    double t0_min = ts[0], t0_max = ts[1];
    double best_c = o.pso_cost;
    double best_t0 = ts[2];
    double a = t0_min, z = t0_max;
    int cnt = fine ? 3 : 5;
    if (fine) { a = fmax(best_t0 - 0.5, t0_min); z = fmin(best_t0 + 0.5, t0_max); }
    int best_k = -1;
    for (int k = 0; k < cnt; k++) {
        const PsoResult& R = d.pso_res[t0_base + (int64_t)b * 8 + (fine ? 5 : 0) + k];
        if (R.cost < best_c) { best_c = R.cost; best_k = k; if (!fine) best_t0 = lin_at(a, z, cnt, k); }
    }
    if (!fine) ts[2] = best_t0;
    if (best_k >= 0) {
        const PsoResult& R = d.pso_res[t0_base + (int64_t)b * 8 + (fine ? 5 : 0) + best_k];
        double t0v = lin_at(a, z, cnt, best_k);
        int fi = 0;
        for (int i = 0; i < np - 1; i++) {
            if (i == t0i) o.pso_params[fi++] = t0v;
            o.pso_params[fi++] = pso_param(R, i);
        }
        if (t0i >= np - 1) o.pso_params[fi] = t0v;
        o.pso_cost = best_c;
    }
}

void launch_t0_build(const DeviceBatch& d, int slot, int fine, cudaStream_t s) {
    if (d.n_bands == 0) return;
    t0_build_kernel<<<(d.n_bands + 127) / 128, 128, 0, s>>>(d, slot, fine, d.t0_slot_base);
}
void launch_t0_pick(const DeviceBatch& d, int slot, int fine, cudaStream_t s) {
    (void)slot;
    if (d.n_bands == 0) return;
    t0_pick_kernel<<<(d.n_bands + 127) / 128, 128, 0, s>>>(d, fine, d.t0_slot_base);
}

// Bazin gate of fit_all_models == false (src/parametric.rs:2037): the bands
// whose polished Bazin cost is >= 2 get the remaining seven models.
__global__ void gate_build_kernel(DeviceBatch d, int slot) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= d.n_bands) return;
    BandStats bs = d.stats[b];
    if (!bs.valid) return;
    if (!(d.fits[b * 8 + BAZIN].cost >= 2.0)) return;
    int base = atomicAdd(&d.ctr->task_count[slot], 21);
    int k = 0;
    for (int mi = 1; mi < 8; mi++) {
        int m = c_select_order[mi];
        for (int r = 0; r < 3; r++) {
            PsoTask t;
            t.band = b;
            t.kind = (int16_t)m;
            t.restart = (int8_t)r;
            t.flags = TASK_PRIOR | TASK_T0_BOUNDS | (r > 0 ? TASK_SEEDED : 0);
            t.out = (b * 8 + m) * 3 + r;
            t.aux = -1;
            t.t0_fixed = 0.0;
            d.tasks[slot][base + k++] = t;
        }
    }
}
void launch_gate_build(const DeviceBatch& d, int slot, cudaStream_t s) {
    if (d.n_bands == 0) return;
    gate_build_kernel<<<(d.n_bands + 127) / 128, 128, 0, s>>>(d, slot);
}

// ---------------------------------------------------------------------------
// MultiBazin (fit_multi_bazin, src/parametric.rs:1008-1157) on rank-0 bands
// with n >= 5.  Results of K live in slots mb_base + (band * 4 + K - 1) * 3 + r.
// ---------------------------------------------------------------------------
__device__ double mb_eval(const double* p, int k, double t) {
    double sum = 0.0;
    for (int c = 0; c < k; c++) {
        const double* q = p + 4 * c;
        double dt = t - q[1];
        sum += exp(q[0]) * exp(-dt / exp(q[3])) * (1.0 / (1.0 + exp(-dt / exp(q[2]))));
    }
    return sum + p[4 * k];
}

__global__ void mb_pick_kernel(DeviceBatch d, int k, int64_t mb_base) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= d.n_bands) return;
    BandStats bs = d.stats[b];
    if (!bs.valid || bs.rank != 0 || bs.n < 5) return;
    MbState& S = d.mb[b];
    if (k == 1) {
        S.best_k = 1; S.done = 0; S.k_done = 0;
        S.best_cost = INFINITY; S.best_bic = INFINITY;
        for (int i = 0; i < LCF_MB_MAX_K; i++) { S.per_k_cost[i] = NAN; S.per_k_bic[i] = NAN; }
    }
    if (S.done) return;
    const PsoResult* R = d.pso_res + mb_base + ((int64_t)b * 4 + (k - 1)) * 3;
    int np = 4 * k + 2;
    int best = 0;
    double c1 = R[0].cost;
    if (k > 1 && R[1].cost < c1) { c1 = R[1].cost; best = 1; }
    if (R[2].cost < c1) { c1 = R[2].cost; best = 2; }
    double nf = (double)bs.n;
    double kb = 2.0 * c1 * nf + (double)np * log(nf);
    S.per_k_cost[k - 1] = c1;
    S.per_k_bic[k - 1] = kb;
    if (kb < S.best_bic) {
        S.best_bic = kb;
        S.best_cost = c1;
        S.best_k = k;
        for (int j = 0; j < MB_MAXP; j++) S.best_params[j] = j < np ? pso_param(R[best], j) : NAN;
    }
    for (int j = 0; j < MB_MAXP; j++) S.prev_params[j] = j < np ? pso_param(R[best], j) : NAN;
    S.k_done = k;
    if (k > 1 && kb > S.per_k_bic[k - 2] + 2.0) S.done = 1;
}

// Builds the K tasks (K >= 2): the seed particle extends the K-1 fit with a
// component at the largest positive residual of a detection.
__global__ void mb_build_kernel(DeviceBatch d, int slot, int k, int64_t mb_base) {
    int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (warp >= d.n_bands) return;
    int b = warp;
    BandStats bs = d.stats[b];
    if (!bs.valid || bs.rank != 0 || bs.n < 5) return;
    MbState& S = d.mb[b];
    if (S.done || S.k_done != k - 1) return;
    BandView v = band_view(d, bs);
    const double* prev = S.prev_params;
    double best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = lane; i < v.n; i += 32) {
        if (v.up[i]) continue;
        double res = v.f[i] - mb_eval(prev, k - 1, v.t[i]);
        if (res > best) { best = res; bi = i; }
    }
    for (int s = 16; s; s >>= 1) {
        double ob = __shfl_xor_sync(FULL, best, s);
        int oi = __shfl_xor_sync(FULL, bi, s);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
    }
    if (lane != 0) return;
    if (bi == 0x7fffffff) bi = 0;
    int np = 4 * k + 2, pn = 4 * (k - 1);
    double init[MB_MAXP];
    for (int j = 0; j < pn; j++) init[j] = prev[j];
    init[pn] = log(fmax(best, 1e-10));
    init[pn + 1] = v.t[bi];
    init[pn + 2] = 1.0;
    init[pn + 3] = 1.0;
    init[pn + 4] = prev[pn];
    init[pn + 5] = prev[pn + 1];
    for (int c = 0; c < k; c++) {
        const double lo[4] = {-3.0, bs.t_first - 30.0, -2.0, -2.0}, hi[4] = {3.0, bs.t_last + 30.0, 5.0, 6.0};
        for (int q = 0; q < 4; q++) init[4 * c + q] = fmin(fmax(init[4 * c + q], lo[q]), hi[q]);
    }
    init[4 * k] = fmin(fmax(init[4 * k], -0.3), 0.3);
    init[4 * k + 1] = fmin(fmax(init[4 * k + 1], -5.0), 0.0);
    for (int j = 0; j < MB_MAXP; j++) S.seed[j] = j < np ? init[j] : 0.0;
    int base = atomicAdd(&d.ctr->task_count[slot], 3);
    for (int r = 0; r < 3; r++) {
        PsoTask t;
        t.band = b;
        t.kind = (int16_t)(KIND_MB1 + k - 1);
        t.restart = (int8_t)r;
        t.flags = r == 1 ? TASK_SEEDED : 0;
        t.out = (int)(mb_base + ((int64_t)b * 4 + (k - 1)) * 3 + r);
        t.aux = r == 1 ? b : -1;
        t.t0_fixed = 0.0;
        d.tasks[slot][base + r] = t;
    }
}

void launch_mb_pick(const DeviceBatch& d, int k, cudaStream_t s) {
    if (d.n_bands == 0) return;
    mb_pick_kernel<<<(d.n_bands + 127) / 128, 128, 0, s>>>(d, k, d.mb_slot_base);
}
void launch_mb_build(const DeviceBatch& d, int slot, int k, cudaStream_t s) {
    if (d.n_bands == 0) return;
    int64_t threads = (int64_t)d.n_bands * 32;
    mb_build_kernel<<<(int)((threads + 127) / 128), 128, 0, s>>>(d, slot, k, d.mb_slot_base);
}

}  // namespace lcf
