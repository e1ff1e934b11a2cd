// metzger_block.cuh — MetzgerKN evaluations of one band by a block: many
// parameter vectors at once, one per lane, in FP64 with the arithmetic of
// metzger_sweep64 (models_f64.cuh).
//
// An Euler step of the sweep is ~500 FP64 instructions (two powers, three
// exponentials, a logarithm, an arctangent, eight divisions), and the FP64
// pipe takes a warp instruction per 16 cycles and SM.  All but ~130 of them
// depend on the grid time alone, that is on t0 and the band: the heating rate
// and the neutron fraction.  A block therefore tabulates each t0's 200 grid
// rows once, its threads over the rows, and the lanes' sweeps read them: the
// scans of the refinements use 25 values of t0 for 75 sweeps and 16 for 61,
// the Laplace stencil 7 for 41.  The sweeps keep their 200 luminosities, so
// that the predictions, which need the grid's peak, are interpolated without
// integrating a second time.
#pragma once

#include "models_f64.cuh"

namespace lcf {

constexpr int MZ_NG = 200;      // grid points
constexpr int MZ_SLOTS = 25;    // t0 values tabulated at once
constexpr int MZ_LANES = 64;    // sweeps whose luminosities are kept
constexpr int MZ_BLOCK = 128;

struct MzTables {
    double row[MZ_NG][3][MZ_SLOTS];   // grid time, neutron fraction, heating rate per mass
    double pm[MZ_SLOTS];              // phase_max of each t0
    // l_rad of each kept sweep, in the block's slice of global memory (L2): in
    // shared memory the block would fill its SM and run beside no other kernel
    double (*lum)[MZ_LANES];
};
constexpr size_t MZ_LUM = (size_t)MZ_NG * MZ_LANES;  // doubles a block

// One grid row: the terms of metzger_sweep64's step that depend on time alone.
__device__ __forceinline__ void mz_row(int i, double pm, double& t_day, double& xn, double& heat) {
    const double SPD = 86400.0, PI = 3.14159265358979323846;
    const double lmin = log(0.01), lmax = log(pm * 1.05);
    t_day = i == 0 ? exp(lmin) : exp(lmin + (lmax - lmin) * (double)i / (double)(MZ_NG - 1));
    const double t_sec = t_day * SPD;
    const double ef = 0.34 * pow(t_day, 0.74);
    const double eth = 0.36 * (exp(-0.56 * t_day) + (ef > 1e-10 ? log(1.0 + ef) / ef : 1.0));
    xn = 0.8 * exp(-t_sec / 900.0);
    const double tt = fmax(0.5 - atan((t_sec - 1.3) / 0.11) / PI, 1e-30);
    const double eps_rp = 2e18 * eth * pow(tt, 1.3);
    heat = 3.2e14 * xn + eps_rp;
}

// Tabulates t0_of(0 .. n_slots - 1), the block's threads over the rows.  The
// caller synchronises before (the tables' last readers) and after.
template <class F>
__device__ void mz_tabulate(MzTables& T, int n_slots, double t_last, F&& t0_of, int tid, int n_threads, int slot0 = 0) {
    for (int q = tid; q < n_slots * MZ_NG; q += n_threads) {
        const int i = q / n_slots, s = q - i * n_slots;
        const double pm = fmax(0.01, t_last - t0_of(s));
        if (i == 0) T.pm[slot0 + s] = pm;
        double t, xn, h;
        mz_row(i, pm, t, xn, h);
        T.row[i][0][slot0 + s] = t;
        T.row[i][1][slot0 + s] = xn;
        T.row[i][2][slot0 + s] = h;
    }
}

// The sweep of one lane over table `slot`, its luminosities to column `col`.
// False when the reference returns zeros before integrating.
__device__ __forceinline__ bool mz_sweep(MzTables& T, const double* p, int slot, int col, double& l_peak) {
    const double MSUN = 1.989e33, C = 2.998e10, SPD = 86400.0, PI = 3.14159265358979323846;
    double m_ej = pow(10.0, p[0]) * MSUN, v_ej = pow(10.0, p[1]) * C, kappa_r = pow(10.0, p[2]);
    l_peak = -INFINITY;
    if (T.pm[slot] <= 0.01) return false;
    double e0 = 0.5 * m_ej * v_ej * v_ej;
    double e_th = e0 / 1e40, e_kin = e0 / 1e40, v = v_ej;
    double t_day = T.row[0][0][slot];
    double r = t_day * SPD * v;
    for (int i = 0; i < MZ_NG; i++) {
        const double xn = T.row[i][1][slot], heat = T.row[i][2][slot];
        double t_sec = t_day * SPD;
        double l_heat = m_ej * heat / 1e40;
        double kappa_eff = 0.4 * (0.8 - xn) + kappa_r * 0.2;
        double t_diff = 3.0 * kappa_eff * m_ej / (4.0 * PI * C * v * t_sec) + r / C;
        double l_rad = (e_th > 0.0 && t_diff > 0.0) ? e_th / t_diff : 0.0;
        l_peak = fmax(l_peak, l_rad);
        T.lum[i][col] = l_rad;
        double l_pdv = r > 0.0 ? e_th * v / r : 0.0;
        if (i < MZ_NG - 1) {
            const double t_next = T.row[i + 1][0][slot];
            double dts = (t_next - t_day) * SPD;
            e_th += (l_heat - l_pdv - l_rad) * dts;
            if (e_th < 0.0) e_th = 0.0;
            e_kin += l_pdv * dts;
            v = fmin(sqrt(2.0 * e_kin * 1e40 / m_ej), C);
            r += v * dts;
            t_day = t_next;
        }
    }
    return true;
}

// The luminosity at phase ph > 0: the grid interval is the first whose end is
// not before the phase, searched from `i` on (phases ascend).
__device__ __forceinline__ double mz_interp(const MzTables& T, int slot, int col, double ph, int& i) {
    while (i < MZ_NG && ph > T.row[i][0][slot]) i++;
    if (i == MZ_NG) return T.lum[MZ_NG - 1][col];
    if (i == 0) {
        if (ph <= T.row[0][0][slot]) return T.lum[0][col];
        i = 1;  // a NaN phase: NaN from the first interval, as in metzger_sweep64
    }
    const double l_rad = T.lum[i][col];
    const double prev_t = T.row[i - 1][0][slot], prev_l = T.lum[i - 1][col];
    double frac = (ph - prev_t) / (T.row[i][0][slot] - prev_t);
    return prev_l + frac * (l_rad - prev_l);
}

// visit(j, l) at every observation after t0, in order; j_start = the first.
template <class V>
__device__ __forceinline__ void mz_visit(const MzTables& T, int slot, int col, double t0, const double* times, int n,
                                         int& j_start, V& visit) {
    int j = 0, i = 0;
    while (j < n && times[j] - t0 <= 0.0) j++;
    j_start = j;
    for (; j < n; j++) visit(j, mz_interp(T, slot, col, times[j] - t0, i));
}

}  // namespace lcf
