// Pieces of the volumetric trace shared by the volumetric kernels: the
// near-disk clamp at the start of an outer step, the hand-over test from the
// outer DP45 loop to the ray-march, the march's starting step, and the
// per-launch counters (src/geodesic_tracer.cpp:71-153 and 495-603).
#pragma once

#include "integrate.cuh"
#include "shading.cuh"
#include "volume.cuh"

namespace grrt_b200 {

struct VolCounters {  // one lane's counts: 32 bits hold hours of steps
    unsigned attempts = 0, accepted = 0, rays = 0, horizon = 0, escaped = 0, maxsteps = 0;
    unsigned clamp = 0, march = 0, physics = 0, fp64 = 0;
    unsigned long long bins = 0;
};

// Order in which the spectral kernel takes its work items: within each full
// block of kVolSpread^2 items the order is transposed, so the 32 items a warp
// takes at once lie kVolSpread items apart in the image. Neighbouring pixels
// trace alike, and the costliest rays (near the photon orbit, grazing the
// volume for thousands of clamped steps) come in clusters; a cluster taken by
// one warp serves its lanes' physics steps one after another, while spread
// over different warps the long rays run side by side. Items past the last
// full block keep their index. A bijection on [0, total).
#ifndef GRRT_VOL_SPREAD
#define GRRT_VOL_SPREAD 64
#endif
constexpr unsigned kVolSpread = GRRT_VOL_SPREAD;
__host__ __device__ __forceinline__ unsigned vol_spread_order(unsigned k, unsigned total) {
    constexpr unsigned kBlock = kVolSpread * kVolSpread;
    if (k >= (total / kBlock) * kBlock) return k;
    const unsigned base = k - k % kBlock, j = k % kBlock;
    return base + (j % kVolSpread) * kVolSpread + j / kVolSpread;
}

// Warp sum of the counters, one atomic per counter per warp.
__device__ __forceinline__ void flush_vol(DevStats* st, const VolCounters& c, bool cancelled) {
    unsigned long long v[11] = {c.attempts, c.accepted, c.rays, c.horizon, c.escaped, c.maxsteps,
                                c.clamp, c.march, c.physics, c.bins, c.fp64};
#pragma unroll
    for (int k = 0; k < 11; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&st->attempts, v[0]);
        atomicAdd(&st->accepted, v[1]);
        atomicAdd(&st->rays, v[2]);
        atomicAdd(&st->horizon, v[3]);
        atomicAdd(&st->escaped, v[4]);
        atomicAdd(&st->max_steps, v[5]);
        atomicAdd(&st->clamp_evals, v[6]);
        atomicAdd(&st->march_steps, v[7]);
        atomicAdd(&st->physics_steps, v[8]);
        atomicAdd(&st->bin_updates, v[9]);
        atomicAdd(&st->fp64_attempts, v[10]);
        if (cancelled && threadIdx.x == 0) atomicAdd(&st->cancelled, 1ull);
    }
}

// Pixel sum += J nu^3 (I_obs = J nu^3, src/geodesic_tracer.cpp:598-600), each
// operation rounded on its own (no contraction into a fused multiply-add), so
// every spectral kernel and the mixed form's resolve produce the same bits.
__device__ __forceinline__ double add_intensity(double sum, double J, double f) {
    return __dadd_rn(sum, __dmul_rn(__dmul_rn(__dmul_rn(J, f), f), f));
}

// Where a state lies relative to the volume: the sine and cosine of its
// colatitude, its height z, and the disk's scale height and photosphere height
// at its radius. The clamp, the hand-over and the march's start need it of the
// same two states of a step, so a trace keeps the one of its current state
// instead of looking it up up to three times.
struct VolGeo {
    double st, ct, z, H, zm;
};
__device__ __forceinline__ VolGeo vol_geo(const DevVolume& V, double r, double th) {
    VolGeo g;
    sincos(th, &g.st, &g.ct);
    g.z = __dmul_rn(r, g.ct);
    const VolCell c = v_cell(V, r);
    g.H = v_radial(V.H, c);
    g.zm = v_radial(V.z_max, c);
    return g;
}

// v_inside of a state whose geometry is known.
__device__ __forceinline__ bool geo_inside(const DevVolume& V, double r, const VolGeo& g) {
    return !(r <= V.r_horizon || r > V.r_outer) && fabs(g.z) < __fma_rn(1.5, g.H, g.zm);
}

// Radii whose outer steps the clamp and the hand-over look at.
__device__ __forceinline__ bool vol_near_radius(const DevVolume& V, double r) {
    return r >= V.r_horizon * 0.9 && r <= V.r_outer * 1.5;
}

// Near-disk clamp at the start of an outer step (src/geodesic_tracer.cpp:71-95):
// for r in [0.9 r_h, 1.5 r_outer] (vol_near_radius, the caller's test) and
// |z| < z_max + 6 H, dlambda is capped at max(H / (4 |dz/dlambda|), H / 64).
// d = f(y), the right-hand side the step's first DP45 stage uses too (the
// reference evaluates it here once more); g = the geometry of y. Returns
// whether the clamp applied (the clamp counter).
__device__ __forceinline__ bool vol_clamp(const Vec5<double>& d, double r, const VolGeo& g, double& dlambda) {
    if (!(fabs(g.z) < __fma_rn(6.0, g.H, g.zm))) return false;
    const double dz_dl = fabs(__fma_rn(g.ct, d.r, -__dmul_rn(__dmul_rn(r, g.st), d.th)));
    if (dz_dl > 1e-20) {
        const double dl_max = vmax(div_f64(0.25 * g.H, dz_dl), g.H * (1.0 / 64.0));
        dlambda = vmin(dlambda, dl_max);
    }
    return true;
}

// Whether an accepted outer step between these radii can hand over at all: its
// radii reach [r_h, r_outer] from a start inside [0.9 r_h, 1.5 r_outer].
__device__ __forceinline__ bool vol_may_enter(const DevVolume& V, double r_prev, double r_new) {
    const double r_lo = vmin(r_prev, r_new), r_hi = vmax(r_prev, r_new);
    return r_hi >= V.r_horizon && r_lo <= V.r_outer && vol_near_radius(V, r_prev);
}

// Hand-over after an accepted outer step prev -> y (src/geodesic_tracer.cpp:105-153)
// that vol_may_enter: the step crossed the equator, ends inside the volume, or
// either end is within z_max + 2H of the plane over the disk's radii. The march
// then starts from prev. gp, g: the geometry of the two ends.
__device__ __forceinline__ bool vol_enters(const DevVolume& V, const Vec5<double>& prev, const VolGeo& gp,
                                           const Vec5<double>& y, const VolGeo& g) {
    const double hp = kHalfPi;
    const double d_prev = prev.th - hp, d_new = y.th - hp;
    const bool crossed = (d_prev * d_new < 0.0) && fabs(d_prev - d_new) > 1e-12;
    const bool near = (fabs(g.z) < __fma_rn(2.0, g.H, g.zm) || fabs(gp.z) < __fma_rn(2.0, gp.H, gp.zm)) &&
                      y.r >= V.r_horizon && y.r <= V.r_outer;
    return crossed || near || geo_inside(V, y.r, g);
}

// First march step length from the start state s of geometry g: H/16 inside
// the volume, else min(|z|/8, 2H).
__device__ __forceinline__ double vol_march_start(const DevVolume& V, double r, const VolGeo& g, bool& been_inside) {
    been_inside = geo_inside(V, r, g);
    return been_inside ? g.H / 16.0 : vmin(fabs(g.z) / 8.0, g.H * 2.0);
}

// Observer-frame RGB frequencies (450, 550, 650 nm) of the RGB transfer.
__device__ __forceinline__ double rgb_nu(int ch) {
    constexpr double c = 2.997924e10;
    return ch == 0 ? c / 450e-7 : (ch == 1 ? c / 550e-7 : c / 650e-7);
}

// The RGB ray-march's work at a new state ns of geometry g, reached by a step
// of length ds (src/geodesic_tracer.cpp:183-337): inside the volume the three
// channels' emission and absorption update J and Tt and the next ds follows
// the optical depth and the radius; outside it ds approaches the volume (never
// inside yet) or holds at H/4 (after being inside). Returns whether the march
// ends here: outside [r_h, r_outer], all channels opaque, or beyond z_max + 3H
// after being inside. The 4096-step cap is the caller's.
__device__ __forceinline__ bool vol_march_rgb(const DevScene& S, double pt, double pph, const Vec5<double>& ns,
                                              const VolGeo& g, double& ds, bool& been_inside, double* J, double* Tt,
                                              VolCounters& cnt) {
    const DevVolume& V = S.vol;
    ++cnt.march;
    const double r = ns.r;
    const double z = g.z, H = g.H;
    if (r < V.r_horizon || r > V.r_outer) return true;
    if (Tt[0] < 1e-6 && Tt[1] < 1e-6 && Tt[2] < 1e-6) return true;
    if (!geo_inside(V, r, g)) {
        if (been_inside && fabs(z) > __fma_rn(3.0, H, g.zm)) return true;
        ds = been_inside ? vclamp(H / 4.0, H / 64.0, H) : vmax(vmin(fabs(z) / 8.0, H * 2.0), H / 64.0);
        return false;
    }
    been_inside = true;
    double rho, Tl;
    v_density_temperature(V, V.perm, r, z, ns.ph, H, g.zm, rho, Tl);
    if (rho > 0.0 && Tl > 0.0) {
        ++cnt.physics;
        double gs, pue;
        v_redshift(V, pt, ns.pr, pph, r, g.ct, gs, pue);
        const double dsp = fabs(pue) * fabs(ds);
        int ir, iT;
        double fr, fT;
        log_locate(log10(rho), V.log_rho_min, V.len_rho, V.inv_len_rho, V.n_rho, ir, fr);
        log_locate(log10(Tl), V.log_T_min, V.len_T, V.inv_len_T, V.n_T, iT, fT);
        const double ke = v_kappa_es(V, ir, fr, iT, fT);
        const double ag = fabs(gs);
        double ka_med = 0.0;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const BinStep s = v_bin_step(V, ag * rgb_nu(b), Tl, rho, dsp, ke, ir, fr, iT, fT);
            if (b == 1) ka_med = s.ka;
            J[b] = __fma_rn(__dmul_rn(Tt[b], s.src), __dadd_rn(1.0, -s.e), J[b]);
            Tt[b] *= s.e;
        }
        cnt.bins += 3;
        const double at = (ka_med + ke) * rho;
        const double ds_tau = (at > 0.0) ? div_f64(0.05, at) : ds * 2.0;
        const double ds_geo = 0.1 * vmax(r - V.r_horizon, 0.5);
        ds = vclamp(vmin(ds_tau, ds_geo), H / 64.0, H);
    }
    return false;
}

}  // namespace grrt_b200
