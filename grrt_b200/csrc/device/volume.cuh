// Volumetric Shakura-Sunyaev disk queries on the device: radial and
// per-column z-normalised profile interpolation, soft photosphere edge, ISCO
// taper, simplex-noise fBm turbulence, emitter four-velocities, and the
// opacity / Planck lookups of the radiative transfer.
//
// Restates src/volumetric_disk.cpp:97-273, src/noise.cpp:38-115 and
// src/opacity.cpp:209-345 with the same operation order. The one planned
// difference is the absorption table, stored as ln(max(kappa, 1e-100)) at
// scene build (the values the reference takes the log of at every lookup), so
// each lookup needs one exp instead of eight logs and an exp.
//
// A physics step is a long chain on few lanes, and a warp waits for it. A
// division by the operator is ~140 cycles and a branch that nothing is
// scheduled across; there were about twenty. The same quotients come from a
// reciprocal (the scene's, or one shared by several quotients) and the exact
// residual, the tables' cells are formed once, and roundings are written out as
// the compiler fused them, so every caller has the same bits (Kerr a=0.9,
// 512x512 on B200: RGB mixed form 31 -> 23 ms, 32 bins FP64 37 -> 33 ms).
#pragma once

#include "integrate.cuh"
#include "scene.h"

namespace grrt_b200 {

__device__ __forceinline__ double vmax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double vmin(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double vclamp(double v, double lo, double hi) {
    return (v < lo) ? lo : (hi < v) ? hi : v;
}
__device__ __forceinline__ int iclamp(int v, int lo, int hi) { return (v < lo) ? lo : (hi < v) ? hi : v; }

// Integer part of a table coordinate, safe for NaN and huge values.
__device__ __forceinline__ int table_index(double t, int lo, int hi) {
    if (!(t >= static_cast<double>(lo))) return lo;
    if (t >= static_cast<double>(hi)) return hi;
    return static_cast<int>(t);
}

// One body of each library function that a physics step calls at several
// places: what stalls the volumetric kernels' full phase is instruction fetch
// (44% of a warp's cycles on the 512x512 spectral frame), and a physics step's
// code is cold each time. (Out of line as well, the geometry's sincos cost the
// frames' long rays more than it saved.)
static __device__ __noinline__ double exp_call(double x) { return exp(x); }
static __device__ __noinline__ double log10_call(double x) { return log10(x); }
static __device__ __noinline__ double2 sincos_call(double x) {
    double2 r;
    sincos(x, &r.x, &r.y);
    return r;
}

// lo (1 - t) + hi t
__device__ __forceinline__ double v_lerp(double lo, double hi, double t) {
    return __fma_rn(hi, t, __dmul_rn(lo, __dadd_rn(1.0, -t)));
}

// (1 - t) lo + t hi, the first product fused
__device__ __forceinline__ double v_mix(double lo, double hi, double t) {
    return __fma_rn(__dadd_rn(1.0, -t), lo, __dmul_rn(t, hi));
}

// Cell and fraction of the radial tables at r; every radial table and profile
// shares it. Outside the tables it is their end, the start first (a disk whose
// outer edge lies at or inside r_min has no other cells).
struct VolCell {
    int i;
    double t;
};
__device__ __forceinline__ VolCell v_cell(const DevVolume& V, double r) {
    const double last = static_cast<double>(V.n_r - 1);
    double frac = __dmul_rn(div_by(__dadd_rn(r, -V.r_min), V.span, V.inv_span), last);
    frac = (r >= V.r_outer) ? last : frac;
    frac = (r <= V.r_min) ? 0.0 : frac;
    const int i = table_index(frac, 0, V.n_r - 2);
    return VolCell{i, __dadd_rn(frac, -static_cast<double>(i))};
}
__device__ __forceinline__ double v_radial(const double* lut, const VolCell& c) {
    return v_lerp(__ldg(lut + c.i), __ldg(lut + c.i + 1), c.t);
}

__device__ __forceinline__ double v_scale_height(const DevVolume& V, double r) {
    return v_radial(V.H, v_cell(V, r));
}
__device__ __forceinline__ double v_zmax(const DevVolume& V, double r) { return v_radial(V.z_max, v_cell(V, r)); }

// Cells of the vertical profiles at height z of the two columns beside a
// radius, each over its own photosphere height; a column that ends below z
// counts as 0.
struct VolColumns {
    bool lo_ok, hi_ok;
    int lo, hi;          // profile elements
    double t_lo, t_hi;
};
__device__ __forceinline__ VolColumns v_columns(const DevVolume& V, const VolCell& c, double z) {
    const double zl = __ldg(V.z_max + c.i), zh = __ldg(V.z_max + c.i + 1);
    VolColumns k;
    k.lo_ok = zl > 0.0 && z < zl;
    k.hi_ok = zh > 0.0 && z < zh;
    const double n = static_cast<double>(V.n_z - 1);
    const double fl = __dmul_rn(div_by(z, zl, __ldg(V.inv_z_max + c.i)), n);
    const double fh = __dmul_rn(div_by(z, zh, __ldg(V.inv_z_max + c.i + 1)), n);
    const int il = table_index(fl, 0, V.n_z - 2), ih = table_index(fh, 0, V.n_z - 2);
    k.lo = c.i * V.n_z + il;
    k.hi = k.lo - il + V.n_z + ih;
    k.t_lo = __dadd_rn(fl, -static_cast<double>(il));
    k.t_hi = __dadd_rn(fh, -static_cast<double>(ih));
    return k;
}
__device__ __forceinline__ double v_profile(const double* lut, const VolCell& c, const VolColumns& k) {
    const double lo = k.lo_ok ? v_mix(__ldg(lut + k.lo), __ldg(lut + k.lo + 1), k.t_lo) : 0.0;
    const double hi = k.hi_ok ? v_mix(__ldg(lut + k.hi), __ldg(lut + k.hi + 1), k.t_hi) : 0.0;
    return v_mix(lo, hi, c.t);
}

__device__ __forceinline__ bool v_inside(const DevVolume& V, double r, double z) {
    if (r <= V.r_horizon || r > V.r_outer) return false;
    return fabs(z) < __fma_rn(1.5, v_scale_height(V, r), v_zmax(V, r));
}

// 3D simplex noise (src/noise.cpp:38-96): skewed cell, corner ranking, 12 edge
// gradients, (0.6 - r^2)^4 kernel, scaled by 32.
// The gradient has two components of +-1: its product is a sum of two
// coordinates with signs.
__device__ __forceinline__ double simplex_corner(double x, double y, double z, int gi) {
    double t0 = __fma_rn(-z, z, __fma_rn(-y, y, __fma_rn(-x, x, 0.6)));
    // gradients to the midpoints of the 12 cube edges: (x, y), (x, z), (y, z)
    const int g = gi % 12;
    const double u = (g < 8) ? x : y, v = (g < 4) ? y : z;
    const double su = (g & 1) ? -u : u, sv = (g & 2) ? -v : v;
    const double dot = __dadd_rn(su, sv);
    t0 = __dmul_rn(t0, t0 < 0.0 ? 0.0 : t0);
    return __dmul_rn(__dmul_rn(t0, t0), dot);
}

__device__ __forceinline__ double simplex3(const int* __restrict__ P, double x, double y, double z) {
    constexpr double F3 = 1.0 / 3.0, G3 = 1.0 / 6.0;
    const double sum = __dadd_rn(__dadd_rn(x, y), z);
    const int i = static_cast<int>(floor(__fma_rn(sum, F3, x))), j = static_cast<int>(floor(__fma_rn(sum, F3, y))),
              k = static_cast<int>(floor(__fma_rn(sum, F3, z)));
    const double n = i + j + k;
    const double x0 = x - __fma_rn(-n, G3, i), y0 = y - __fma_rn(-n, G3, j), z0 = z - __fma_rn(-n, G3, k);
    int i1, j1, k1, i2, j2, k2;
    if (x0 >= y0) {
        if (y0 >= z0) { i1 = 1; j1 = 0; k1 = 0; i2 = 1; j2 = 1; k2 = 0; }
        else if (x0 >= z0) { i1 = 1; j1 = 0; k1 = 0; i2 = 1; j2 = 0; k2 = 1; }
        else { i1 = 0; j1 = 0; k1 = 1; i2 = 1; j2 = 0; k2 = 1; }
    } else {
        if (y0 < z0) { i1 = 0; j1 = 0; k1 = 1; i2 = 0; j2 = 1; k2 = 1; }
        else if (x0 < z0) { i1 = 0; j1 = 1; k1 = 0; i2 = 0; j2 = 1; k2 = 1; }
        else { i1 = 0; j1 = 1; k1 = 0; i2 = 1; j2 = 1; k2 = 0; }
    }
    const double x1 = x0 - i1 + G3, y1 = y0 - j1 + G3, z1 = z0 - k1 + G3;
    const double x2 = x0 - i2 + 2 * G3, y2 = y0 - j2 + 2 * G3, z2 = z0 - k2 + 2 * G3;
    const double x3 = x0 - 1 + 3 * G3, y3 = y0 - 1 + 3 * G3, z3 = z0 - 1 + 3 * G3;
    const int ii = i & 255, jj = j & 255, kk = k & 255;
    const double n0 = simplex_corner(x0, y0, z0, P[ii + P[jj + P[kk]]]);
    const double n1 = simplex_corner(x1, y1, z1, P[ii + i1 + P[jj + j1 + P[kk + k1]]]);
    const double n2 = simplex_corner(x2, y2, z2, P[ii + i2 + P[jj + j2 + P[kk + k2]]]);
    const double n3 = simplex_corner(x3, y3, z3, P[ii + 1 + P[jj + 1 + P[kk + 1]]]);
    return 32.0 * (n0 + n1 + n2 + n3);
}

// Density with the soft photosphere edge, ISCO taper and fBm turbulence, and
// temperature from the vertical profile, its surface value in the soft edge
// (src/volumetric_disk.cpp:228-273), at a point inside the volume's bounds
// (r_h < r <= r_outer, |z| < zm + 1.5 H). H, zm: the scale and photosphere
// heights at r. P is the 512-entry permutation.
__device__ __forceinline__ void v_density_temperature(const DevVolume& V, const int* __restrict__ P, double r,
                                                      double z, double phi, double H, double zm, double& rho,
                                                      double& T) {
    const double z_abs = fabs(z);
    const double z_top = __dmul_rn(zm, 0.9999);
    const double z_T = vmin(z_abs, z_top);
    double edge = 1.0, z_look = z_abs;
    bool dense = true;
    if (z_abs >= zm) {
        const double dz = __dadd_rn(z_abs, -zm);
        dense = !(dz >= __dmul_rn(1.5, H));
        const double d = div_f64(dz, H);
        edge = exp_call(__dmul_rn(__dmul_rn(-2.0, d), d));
        z_look = z_top;
    }
    const VolCell c = v_cell(V, r);
    VolColumns k = v_columns(V, c, z_look);
    const double rho_mid = v_radial(V.rho_mid, c);
    const double rho_norm = v_profile(V.rho_prof, c, k);
    if (z_T != z_look) k = v_columns(V, c, z_T);
    T = v_profile(V.T_prof, c, k);
    double taper = 1.0;
    if (r < V.r_isco) {
        const double dr = __dadd_rn(V.r_isco, -r);
        taper = exp_call(div_by(-__dmul_rn(dr, dr), V.taper_w2, V.inv_taper_w2));
    }
    const double base = __dmul_rn(
        __dmul_rn(__dmul_rn(__dmul_rn(rho_mid, rho_norm), V.rho_scale), taper), edge);
    const double2 sc = sincos_call(phi);
    const double sp = sc.x, cp = sc.y;
    const double nx = div_by(__dmul_rn(r, cp), V.noise_scale, V.inv_noise);
    const double ny = div_by(__dmul_rn(r, sp), V.noise_scale, V.inv_noise);
    const double nz = div_by(z, V.noise_scale, V.inv_noise);
    double n = 0.0, amp = 1.0, freq = 1.0;
    for (int o = 0; o < V.octaves; ++o) {
        n = __fma_rn(amp, simplex3(P, nx * freq, ny * freq, nz * freq), n);
        amp *= 0.5;
        freq *= 2.0;
    }
    rho = dense ? vmax(0.0, __dmul_rn(base, __fma_rn(V.turbulence, n, 1.0))) : 0.0;
}

// Emitter four-velocity (circular orbit outside the ISCO, plunging geodesic
// with ISCO constants inside; src/volumetric_disk.cpp:97-137) and the redshift
// g = (p.u)_emit / (p.u)_obs (src/geodesic_tracer.cpp:279-292). ct: cos(theta).
__device__ __forceinline__ void v_redshift(const DevVolume& V, double pt, double pr, double pph, double r,
                                           double ct, double& g, double& pue) {
    const double M = V.M, a = V.a;
    const double ri = recip_f64(r);
    const double m2 = 2.0 * M;
    double ut, ur = 0.0, uphi;
    if (r >= V.r_isco) {
        const double Omg = div_f64(V.sqrt_M, __fma_rn(r, sqrt(r), __dmul_rn(a, V.sqrt_M)));
        const double g_tt = -__dadd_rn(1.0, -div_by(m2, r, ri));
        const double g_tphi = div_by(__dmul_rn(-m2, a), r, ri);
        const double g_phph =
            __dadd_rn(__fma_rn(r, r, __dmul_rn(a, a)), div_by(__dmul_rn(__dmul_rn(m2, a), a), r, ri));
        const double den = -__fma_rn(__dmul_rn(g_phph, Omg), Omg, __fma_rn(2.0 * g_tphi, Omg, g_tt));
        ut = recip_f64(sqrt(vmax(den, 1e-30)));
        uphi = __dmul_rn(Omg, ut);
    } else {
        const double E = V.E_isco, L = V.L_isco;
        const double a2 = __dmul_rn(a, a), r2 = __dmul_rn(r, r), m2a = __dmul_rn(m2, a);
        const double ra = __dadd_rn(r2, a2);
        const double Delta = __dadd_rn(__fma_rn(-m2, r, r2), a2);
        const double Sigma = __fma_rn(__dmul_rn(a2, ct), ct, r2);
        const double sum = __dadd_rn(ra, __ddiv_rn(__dmul_rn(m2a, a), r));
        ut = __ddiv_rn(__fma_rn(E, sum, -__ddiv_rn(__dmul_rn(m2a, L), r)), Delta);
        uphi = __ddiv_rn(__fma_rn(L, __dadd_rn(1.0, -__ddiv_rn(m2, r)), __ddiv_rn(__dmul_rn(m2a, E), r)), Delta);
        const double EaL = __fma_rn(E, ra, -__dmul_rn(a, L));
        const double LaE = __fma_rn(-a, E, L);
        const double R = __fma_rn(EaL, EaL, -__dmul_rn(Delta, __fma_rn(LaE, LaE, r2)));
        ur = __ddiv_rn(-__dsqrt_rn(vmax(0.0, R)), Sigma);
    }
    pue = __fma_rn(pph, uphi, __fma_rn(pt, ut, __dmul_rn(pr, ur)));
    g = div_f64(pue, __dmul_rn(pt, V.ut_obs));
}

// Table coordinate of a log-spaced axis of length len (src/opacity.cpp:218-224).
// The distance from the axis' start is clamped before the quotient, which has
// to be finite: a frequency bin of 0 or infinity has an infinite lv.
__device__ __forceinline__ void log_locate(double lv, double lo, double len, double inv_len, int n, int& idx,
                                           double& frac) {
    const double d = vmin(vmax(__dadd_rn(lv, -lo), 0.0), len);
    const double t = vmin(__dmul_rn(div_by(d, len, inv_len), static_cast<double>(n - 1)), static_cast<double>(n - 2));
    idx = table_index(t, 0, n - 2);
    frac = __dadd_rn(t, -static_cast<double>(idx));
}

// Electron-scattering opacity, bilinear in the (rho, T) cell.
__device__ __forceinline__ double v_kappa_es(const DevVolume& V, int ir, double fr, int iT, double fT) {
    const double* L = V.kes;
    const int nt = V.n_T;
    const double v00 = __ldg(L + ir * nt + iT), v01 = __ldg(L + ir * nt + iT + 1);
    const double v10 = __ldg(L + (ir + 1) * nt + iT), v11 = __ldg(L + (ir + 1) * nt + iT + 1);
    const double gr = __dadd_rn(1.0, -fr), gT = __dadd_rn(1.0, -fT);
    double k = __fma_rn(__dmul_rn(v00, gr), gT, __dmul_rn(__dmul_rn(v01, gr), fT));
    k = __fma_rn(__dmul_rn(v10, fr), gT, k);
    return __fma_rn(__dmul_rn(v11, fr), fT, k);
}

// Absorption opacity: trilinear in ln kappa over (nu, rho, T), then exp.
__device__ __forceinline__ double v_kappa_abs(const DevVolume& V, double nu, int ir, double fr, int iT, double fT) {
    int inu;
    double fnu;
    log_locate(log10_call(nu), V.log_nu_min, V.len_nu, V.inv_len_nu, V.n_nu, inu, fnu);
    const size_t s0 = static_cast<size_t>(V.n_rho) * V.n_T;
    const double* L0 = V.ln_kabs + inu * s0 + ir * V.n_T + iT;
    const double* L1 = L0 + s0;
    const int nt = V.n_T;
    const double l00 = v_mix(__ldg(L0), __ldg(L0 + 1), fT);
    const double l01 = v_mix(__ldg(L0 + nt), __ldg(L0 + nt + 1), fT);
    const double l10 = v_mix(__ldg(L1), __ldg(L1 + 1), fT);
    const double l11 = v_mix(__ldg(L1 + nt), __ldg(L1 + nt + 1), fT);
    return exp_call(v_mix(v_mix(l00, l01, fr), v_mix(l10, l11, fr), fnu));
}

// One frequency's transfer over a physics step (src/geodesic_tracer.cpp:300-325):
// opacity, optical depth and Planck emission (CGS, src/opacity.cpp:209-214) at
// emitter frequency nu.
struct BinStep {
    double ka, dtau, src, e;  // kappa_abs, optical depth, source B eps / nu^3, exp_call(-dtau)
};
__device__ __forceinline__ BinStep v_bin_step(const DevVolume& V, double nu, double T, double rho, double dsp,
                                              double ke, int ir, double fr, int iT, double fT) {
    constexpr double h = 6.626070e-27, k = 1.380649e-16, c = 2.997924e10;
    BinStep s;
    s.ka = v_kappa_abs(V, nu, ir, fr, iT, fT);
    const double kt = __dadd_rn(s.ka, ke);
    const double eps = (kt > 0.0) ? div_by(s.ka, kt, recip_f64(kt)) : 1.0;  // ka >= 1e-100
    s.dtau = __dmul_rn(__dmul_rn(kt, rho), dsp);
    double B = 0.0;
    if (!(nu <= 0.0 || T <= 0.0)) {
        const double x = div_f64(__dmul_rn(h, nu), __dmul_rn(k, T));
        if (!(x > 500.0)) {
            const double n3 = __dmul_rn(__dmul_rn(__dmul_rn(2.0 * h, nu), nu), nu);
            B = div_f64(div_by(n3, c * c, 1.0 / (c * c)), __dadd_rn(exp_call(x), -1.0));
        }
    }
    s.src = div_f64(__dmul_rn(eps, B), __dmul_rn(__dmul_rn(nu, nu), nu));
    s.e = exp_call(-s.dtau);
    return s;
}

}  // namespace grrt_b200
