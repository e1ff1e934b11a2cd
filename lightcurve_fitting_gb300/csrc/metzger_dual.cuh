// metzger_dual.cuh — MetzgerKN prediction and its derivatives with respect to
// (log10 M_ej, log10 v_ej, log10 kappa, t0) by forward-mode differentiation in
// FP32 (dual numbers).
//
// The reference differentiates MetzgerKN for SVI by forward differences of
// its FP64 model with step 1e-5 (metzger_kn_grad_batch_into,
// src/parametric.rs:843-860): five sequential ODE solves per sample.  In FP32
// a 1e-5 difference would lose the derivative to rounding, so the sweep of
// models_f32.cuh (MetzgerF::sweep) is carried out on dual numbers instead: the
// tangents give the derivative of the same piecewise formula (grid, Euler
// recurrence with its clamps, linear interpolation, peak normalisation) that
// the forward difference approximates to O(1e-5).
#pragma once

#include <math.h>

namespace lcf {

// A value with K tangents (forward-mode dual number).
template <int K>
struct DN {
    float v, d[K];
    __device__ DN() {}
    __device__ explicit DN(float x) : v(x) {
#pragma unroll
        for (int k = 0; k < K; k++) d[k] = 0.0f;
    }
};
template <int K>
__device__ __forceinline__ DN<K> mk(float v, float s, const DN<K>& a) {  // v with tangent s * a.d
    DN<K> r;
    r.v = v;
#pragma unroll
    for (int k = 0; k < K; k++) r.d[k] = s * a.d[k];
    return r;
}
template <int K>
__device__ __forceinline__ DN<K> operator+(const DN<K>& a, const DN<K>& b) {
    DN<K> r; r.v = a.v + b.v;
#pragma unroll
    for (int k = 0; k < K; k++) r.d[k] = a.d[k] + b.d[k];
    return r;
}
template <int K>
__device__ __forceinline__ DN<K> operator-(const DN<K>& a, const DN<K>& b) {
    DN<K> r; r.v = a.v - b.v;
#pragma unroll
    for (int k = 0; k < K; k++) r.d[k] = a.d[k] - b.d[k];
    return r;
}
template <int K>
__device__ __forceinline__ DN<K> operator*(const DN<K>& a, const DN<K>& b) {
    DN<K> r; r.v = a.v * b.v;
#pragma unroll
    for (int k = 0; k < K; k++) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
    return r;
}
template <int K>
__device__ __forceinline__ DN<K> operator/(const DN<K>& a, const DN<K>& b) {
    DN<K> r; float ib = 1.0f / b.v; r.v = a.v * ib;
#pragma unroll
    for (int k = 0; k < K; k++) r.d[k] = (a.d[k] - r.v * b.d[k]) * ib;
    return r;
}
template <int K>
__device__ __forceinline__ DN<K> operator+(const DN<K>& a, float c) { DN<K> r = a; r.v += c; return r; }
template <int K>
__device__ __forceinline__ DN<K> operator-(const DN<K>& a, float c) { DN<K> r = a; r.v -= c; return r; }
template <int K>
__device__ __forceinline__ DN<K> operator*(const DN<K>& a, float c) { return mk(a.v * c, c, a); }
template <int K>
__device__ __forceinline__ DN<K> operator*(float c, const DN<K>& a) { return mk(a.v * c, c, a); }
template <int K>
__device__ __forceinline__ DN<K> dexp(const DN<K>& a) { float e = expf(a.v); return mk(e, e, a); }
template <int K>
__device__ __forceinline__ DN<K> dlog(const DN<K>& a) { return mk(logf(a.v), 1.0f / a.v, a); }
template <int K>
__device__ __forceinline__ DN<K> dlog1p(const DN<K>& a) { return mk(log1pf(a.v), 1.0f / (1.0f + a.v), a); }
template <int K>
__device__ __forceinline__ DN<K> dsqrt(const DN<K>& a) { float s = sqrtf(a.v); return mk(s, 0.5f / s, a); }
template <int K>
__device__ __forceinline__ DN<K> dpowc(const DN<K>& a, float c) {  // a^c, a > 0
    float p = exp2f(c * log2f(a.v));
    return mk(p, c * p / a.v, a);
}
template <int K>
__device__ __forceinline__ DN<K> datan(const DN<K>& a) { return mk(atanf(a.v), 1.0f / (1.0f + a.v * a.v), a); }

// ---------------------------------------------------------------------------
// The sweep by a warp (the SVI's steps, and lcf_svi_elbo_grad).  Of a grid
// step's ~300 instructions all but the energy, velocity and radius recursion
// depend on the grid time alone: the lanes first form the 200 grid rows and
// their t0 tangents, then lanes 0..3 run the recursion (lane k with the tangent
// of parameter k), and the lanes interpolate the observations.  The recursion's
// 200 dependent steps are what is left of the chain.
// ---------------------------------------------------------------------------
// a * b with the tangent's two products rounded in a fixed order: the first
// form rounds a'b before the sum, the second ab'.  Whichever product is fused,
// the tangent is good to an ulp, but the recursion amplifies an ulp, so the
// order is written down at the places that feed it: a fit keeps its bits
// whatever the compiler would contract there.
__device__ __forceinline__ DN<1> mul_round_first(const DN<1>& a, const DN<1>& b) {
    DN<1> r;
    r.v = a.v * b.v;
    r.d[0] = __fmaf_rn(a.v, b.d[0], __fmul_rn(a.d[0], b.v));
    return r;
}
__device__ __forceinline__ DN<1> mul_round_second(const DN<1>& a, const DN<1>& b) {
    DN<1> r;
    r.v = a.v * b.v;
    r.d[0] = __fmaf_rn(a.d[0], b.v, __fmul_rn(a.v, b.d[0]));
    return r;
}
// Keeps a value's own rounding: the compiler must not contract the product
// behind it into a later sum.
__device__ __forceinline__ void keep_rounded(DN<1>& a) {
    asm volatile("" : "+f"(a.v), "+f"(a.d[0]));
}
struct MzWarp {
    float row[200][6];  // grid time, heating rate per mass, 0.8 - neutron fraction; each with its t0 tangent
    float lum[200][5];  // l_rad and its four tangents
};

__device__ __forceinline__ void metzger_dual_row(int i, const DN<1>& dl, float lmin, float* row) {
    using D = DN<1>;
    const float SPD = 86400.0f, PI_F = 3.14159265358979f;
    const float xn0 = 0.8f;
    D t_day = i == 0 ? D(0.01f) : dexp(dl * (float)i + lmin);
    D t_sec = t_day * SPD;
    D ef = dpowc(t_day, 0.74f) * 0.34f;
    D eth = (dexp(t_day * -0.56f) + (ef.v > 1e-10f ? dlog1p(ef) / ef : D(1.0f))) * 0.36f;
    D xn = dexp(t_sec * (-1.0f / 900.0f)) * xn0;
    D tt = datan(D(0.11f) / (t_sec - 1.3f)) * (1.0f / PI_F);
    if (tt.v < 1e-30f) tt = D(1e-30f);
    D eps_rp = mul_round_second(eth, dpowc(tt, 1.3f)) * 2e18f;
    D heat = xn * 3.2e14f + eps_rp;
    D q = D(xn0) - xn;
    row[0] = t_day.v; row[1] = t_day.d[0];
    row[2] = heat.v; row[3] = heat.d[0];
    row[4] = q.v; row[5] = q.d[0];
}

// One sample's normalised predictions and derivatives of the band to
// out[j * 5 + {0..4}], for observation times in ascending order; pv is uniform
// over the warp.  All zeros where the reference returns zeros (phase_max <=
// 0.01, or a non-positive or non-finite peak).
template <class Times>
__device__ __forceinline__ void metzger_dual_warp(MzWarp& W, const float* pv, float t_last, const Times& t, int n,
                                                  float* out) {
    using D = DN<1>;
    const float MSUN30 = 1.989e3f, C = 2.998e10f, SPD = 86400.0f, PI_F = 3.14159265358979f, LN10F = 2.302585093f;
    const int lane = threadIdx.x & 31;
    const float lmin = -4.605170185988091f;
    const float pm = t_last - pv[3];
    bool ok = pm > 0.01f;
    D t0(pv[3]);
    float lp_v = 0.0f, lp_d = 0.0f;
    if (ok) {
        t0.d[0] = 1.0f;
        {
            D phase_max = (t0 * -1.0f) + t_last;
            D lmax = dlog(phase_max * 1.05f);
            D dl = (lmax - lmin) * (1.0f / 199.0f);
            for (int i = lane; i < 200; i += 32) metzger_dual_row(i, dl, lmin, W.row[i]);
        }
        __syncwarp();
        if (lane < 4) {
            D p0(pv[0]), p1(pv[1]), p2(pv[2]);
            if (lane == 0) p0.d[0] = 1.0f;
            if (lane == 1) p1.d[0] = 1.0f;
            if (lane == 2) p2.d[0] = 1.0f;
            D m30 = dexp(p0 * LN10F) * MSUN30;
            D v = dexp(p1 * LN10F) * C;
            D kappa_r = dexp(p2 * LN10F);
            const float xr = 0.2f;
            D vs = v * 1e-5f;
            D e_th = m30 * vs * vs * 0.5f;
            D e_kin = e_th;
            D t_day = D(0.01f);
            D r = t_day * v * SPD;
            D mos = m30 * 1e-10f;
            D diff_k = m30 * (3.0f / (4.0f * PI_F * C) * 1e30f);
            D l_peak = D(-INFINITY);
            auto tangent = [&](float d) { return lane == 3 ? d : 0.0f; };
            for (int i = 0; i < 200; i++) {
                const float* row = W.row[i];
                D heat(row[2]), q(row[4]);
                heat.d[0] = tangent(row[3]);
                q.d[0] = tangent(row[5]);
                D t_sec = t_day * SPD;
                D l_heat = mos * heat;
                D kappa_eff = q * 0.4f + kappa_r * xr;
                D t_diff = kappa_eff * diff_k / mul_round_first(v, t_sec) + r * (1.0f / C);
                D l_rad = (e_th.v > 0.0f && t_diff.v > 0.0f) ? e_th / t_diff : D(0.0f);
                if (l_rad.v > l_peak.v) l_peak = l_rad;
                if (lane == 0) W.lum[i][0] = l_rad.v;
                W.lum[i][1 + lane] = l_rad.d[0];
                D l_pdv = r.v > 0.0f ? e_th * v / r : D(0.0f);
                if (i < 199) {
                    D t_next(W.row[i + 1][0]);
                    t_next.d[0] = tangent(W.row[i + 1][1]);
                    D dts = (t_next - t_day) * SPD;
                    e_th = e_th + mul_round_first(l_heat - l_pdv - l_rad, dts);
                    if (e_th.v < 0.0f) e_th = D(0.0f);
                    e_kin = e_kin + mul_round_first(l_pdv, dts);
                    D vn = dsqrt(e_kin * 2.0f / mos);
                    v = vn.v < C ? vn : D(C);
                    r = r + mul_round_first(v, dts);
                    t_day = t_next;
                }
            }
            lp_v = l_peak.v;
            lp_d = l_peak.d[0];
        }
        __syncwarp();
        lp_v = __shfl_sync(0xffffffffu, lp_v, 0);
        ok = lp_v > 0.0f && isfinite(lp_v);
    }
    // lane 4 q + k: tangent k of observations q, q + 8, ...
    const int k = lane & 3;
    const float lpd = __shfl_sync(0xffffffffu, lp_d, k);
    const float ip = 1.0f / lp_v;
    auto tangent = [&](float d) { return k == 3 ? d : 0.0f; };
    for (int j = lane >> 2; j < n; j += 8) {
        D l(0.0f);
        const float phv = t(j) - pv[3];
        if (ok && !(phv <= 0.0f)) {
            // the first grid point not before the phase (a NaN phase: NaN from the first interval)
            int i = 0;
            for (int step = 128; step; step >>= 1)
                if (i + step <= 200 && phv > W.row[i + step - 1][0]) i += step;
            if (i == 0 && !(phv <= W.row[0][0])) i = 1;
            if (i == 0 || i == 200) {
                const int g = i == 0 ? 0 : 199;
                l.v = W.lum[g][0];
                l.d[0] = W.lum[g][1 + k];
            } else {
                D tk(pv[3]), prev_t(W.row[i - 1][0]), t_day(W.row[i][0]), prev_l(W.lum[i - 1][0]), l_rad(W.lum[i][0]);
                tk.d[0] = tangent(1.0f);
                prev_t.d[0] = tangent(W.row[i - 1][1]);
                t_day.d[0] = tangent(W.row[i][1]);
                prev_l.d[0] = W.lum[i - 1][1 + k];
                l_rad.d[0] = W.lum[i][1 + k];
                D ph = (tk * -1.0f) + t(j);
                l = prev_l + (ph - prev_t) / (t_day - prev_t) * (l_rad - prev_l);
            }
        }
        keep_rounded(l);
        // normalise by the peak, its tangent included
        const float y = l.v * ip;
        out[j * 5 + 1 + k] = ok ? (l.d[0] - y * lpd) * ip : 0.0f;
        if (k == 0) out[j * 5] = ok ? y : 0.0f;
    }
    __syncwarp();
}

}  // namespace lcf
