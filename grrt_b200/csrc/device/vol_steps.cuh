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

// Order in which the kernels take many work items: within each full
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

// Lanes of a warp that take work items: all 32 of them where the items keep the
// grid's lanes busy; where there are fewer items than lanes, their number
// spread over the warps, since a warp runs its lanes' different phases one
// after another and a ray alone in its warp runs fastest.
__device__ __forceinline__ int vol_lanes_in_use(unsigned total) {
    const unsigned warps = gridDim.x * (blockDim.x >> 5);
    const unsigned per = (total + warps - 1) / warps;
    return per < 32u ? static_cast<int>(per) : 32;
}

// The item of a grid's k-th take where most items have a lane from the start:
// blocks of one item a lane (`lanes` of each of `warps` warps; the last block
// what remains) are dealt out over the warps, so the numbers a warp takes at
// once lie a warp count of items apart and clusters of long rays end up in
// different warps. A bijection on [0, total).
__host__ __device__ __forceinline__ unsigned vol_deal_order(unsigned k, unsigned total, unsigned lanes,
                                                            unsigned warps) {
    const unsigned block = lanes * warps;
    const unsigned base = k - k % block, j = k % block;
    const unsigned m = total - base < block ? total - base : block;
    const unsigned q = m / lanes, r = m % lanes;  // the first r rows hold one more
    if (j >= q * lanes) return base + (j - q * lanes) * (q + 1) + q;
    const unsigned row = j % lanes;
    return base + row * q + (row < r ? row : r) + j / lanes;
}

// The item of the k-th take. Up to two items a lane they are dealt out: the
// frame then waits for its longest rays, which run fastest with short-lived
// neighbours (Kerr a=0.9 on B200, over disk seeds: 512x512 RGB mixed, 58 k
// listed rays on 56,832 lanes, 195 -> 185 ms for six frames, 19.4 -> 14.8 at
// best; 101x75, 16 bins, mixed: 11.8 -> 9.3). Beyond that the spread order,
// which starts a frame's long rays nearly in their own order, is as good or
// better (512x512, 32 bins, FP64, three frames: 101 against 106 ms dealt).
__device__ __forceinline__ unsigned vol_take_order(unsigned k, unsigned total) {
    const unsigned warps = gridDim.x * (blockDim.x >> 5);
    if (total > 64u * warps) return vol_spread_order(k, total);
    return vol_deal_order(k, total, vol_lanes_in_use(total), warps);
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
    return !((r <= V.r_horizon) | (r > V.r_outer)) & (fabs(g.z) < __fma_rn(1.5, g.H, g.zm));
}

// Radii whose outer steps the clamp and the hand-over look at.
__device__ __forceinline__ bool vol_near_radius(const DevVolume& V, double r) {
    return (r >= V.r_horizon * 0.9) & (r <= V.r_outer * 1.5);
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
    return (r_hi >= V.r_horizon) & (r_lo <= V.r_outer) & vol_near_radius(V, r_prev);
}

// Hand-over after an accepted outer step prev -> y (src/geodesic_tracer.cpp:105-153)
// that vol_may_enter: the step crossed the equator, ends inside the volume, or
// either end is within z_max + 2H of the plane over the disk's radii. The march
// then starts from prev. gp, g: the geometry of the two ends.
__device__ __forceinline__ bool vol_enters(const DevVolume& V, const Vec5<double>& prev, const VolGeo& gp,
                                           const Vec5<double>& y, const VolGeo& g) {
    const double hp = kHalfPi;
    const double d_prev = prev.th - hp, d_new = y.th - hp;
    const bool crossed = (d_prev * d_new < 0.0) & (fabs(d_prev - d_new) > 1e-12);
    const bool near = ((fabs(g.z) < __fma_rn(2.0, g.H, g.zm)) | (fabs(gp.z) < __fma_rn(2.0, gp.H, gp.zm))) &
                      (y.r >= V.r_horizon) & (y.r <= V.r_outer);
    return crossed | near | geo_inside(V, y.r, g);
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

// The ray-march at a new state of radius r and geometry g
// (src/geodesic_tracer.cpp:183-337): it ends outside [r_h, r_outer], when
// opaque, or beyond z_max + 3H after being inside; inside the volume the step's
// physics comes next; elsewhere the next step length ds approaches the volume
// (never inside yet) or holds at H/4 (after being inside). The 4096-step cap is
// the caller's.
enum MarchState { kMarchOn, kMarchEnd, kMarchInside };
__device__ __forceinline__ MarchState vol_march_state(const DevVolume& V, double r, const VolGeo& g, bool opaque,
                                                      bool& been_inside, double& ds) {
    const bool in = geo_inside(V, r, g);
    const bool end = (r < V.r_horizon) | (r > V.r_outer) | opaque |
                     (!in & been_inside & (fabs(g.z) > __fma_rn(3.0, g.H, g.zm)));
    const double approach = vmax(vmin(fabs(g.z) / 8.0, g.H * 2.0), g.H / 64.0);
    const double hold = vclamp(g.H / 4.0, g.H / 64.0, g.H);
    if (end) return kMarchEnd;
    if (in) {
        been_inside = true;
        return kMarchInside;
    }
    ds = been_inside ? hold : approach;
    return kMarchOn;
}

// The frequency-independent part of a physics step.
struct PhysStep {
    double ag, rho, T, dsp, ke, fr, fT;  // |g|, density, temperature, path, kappa_es, table fractions
    int ir, iT;                          // table cell
};
// At the march's state y of geometry g inside the volume, reached by a step of
// length ds; false where there is no matter.
__device__ __forceinline__ bool vol_physics(const DevVolume& V, double pt, double pph, const Vec5<double>& y,
                                            const VolGeo& g, double ds, PhysStep& p) {
    v_density_temperature(V, V.perm, y.r, g.z, y.ph, g.H, g.zm, p.rho, p.T);
    if (!(p.rho > 0.0 && p.T > 0.0)) return false;
    double gs, pue;
    v_redshift(V, pt, y.pr, pph, y.r, g.ct, gs, pue);
    p.ag = fabs(gs);
    p.dsp = fabs(pue) * fabs(ds);
    log_locate(log10_call(p.rho), V.log_rho_min, V.len_rho, V.inv_len_rho, V.n_rho, p.ir, p.fr);
    log_locate(log10_call(p.T), V.log_T_min, V.len_T, V.inv_len_T, V.n_T, p.iT, p.fT);
    p.ke = v_kappa_es(V, p.ir, p.fr, p.iT, p.fT);
    return true;
}

// The next march step length after a physics step: an optical depth of 0.05 at
// the median frequency (opacity ka + ke), a tenth of the distance to the
// horizon, between H/64 and H.
__device__ __forceinline__ double vol_next_ds(const DevVolume& V, double r, double H, double ka, double ke,
                                              double rho, double ds) {
    const double at = (ka + ke) * rho;
    const double ds_tau = (at > 0.0) ? div_f64(0.05, at) : ds * 2.0;
    const double ds_geo = 0.1 * vmax(r - V.r_horizon, 0.5);
    return vclamp(vmin(ds_tau, ds_geo), H / 64.0, H);
}

// One frequency's transfer: J += T S (1 - e), T *= e.
__device__ __forceinline__ void vol_transfer(const BinStep& s, double& J, double& T) {
    J = __fma_rn(__dmul_rn(T, s.src), __dadd_rn(1.0, -s.e), J);
    T = __dmul_rn(T, s.e);
}

// Physics steps of a warp's lanes staged in shared memory by rank, for the
// per-frequency part that the whole warp does.
struct PhysStage {
    double ag[32], rho[32], T[32], dsp[32], ke[32], fr[32], fT[32];
    int ir[32], iT[32], src[32];  // table cell, the lane
    __device__ __forceinline__ void put(int k, const PhysStep& p, int lane) {
        ag[k] = p.ag;
        rho[k] = p.rho;
        T[k] = p.T;
        dsp[k] = p.dsp;
        ke[k] = p.ke;
        fr[k] = p.fr;
        fT[k] = p.fT;
        ir[k] = p.ir;
        iT[k] = p.iT;
        src[k] = lane;
    }
    __device__ __forceinline__ BinStep bin(const DevVolume& V, int k, double freq) const {
        return v_bin_step(V, __dmul_rn(ag[k], freq), T[k], rho[k], dsp[k], ke[k], ir[k], fr[k], iT[k], fT[k]);
    }
};

}  // namespace grrt_b200
