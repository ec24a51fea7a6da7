// Device build of FP64 building blocks beside the plain operations they stand
// for, at the ends of their ranges, so a GPU test can compare the bits.
// Test-only.
#include <vector>

#include "../../grrt_b200/csrc/device/volume.cuh"

using namespace grrt_b200;

namespace {

// x -> reciprocal, and the quotient a / x through it
__global__ void recip_kernel(const double* in, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = in[2 * i], x = in[2 * i + 1];
    fast[2 * i] = recip_f64(x);
    plain[2 * i] = 1.0 / x;
    fast[2 * i + 1] = div_f64(a, x);
    plain[2 * i + 1] = a / x;
}

// five |numerators| and five |y| -> the largest quotient's numerator and denominator
__global__ void quotient_kernel(const double* in, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* e = in + 10 * i;
    const double* y = e + 5;
    const Vec5<double> zero{0.0, 0.0, 0.0, 0.0, 0.0};
    const ErrQuotient q = error_quotient(Vec5<double>{y[0], y[1], y[2], y[3], y[4]}, 1.0, zero,
                                         Vec5<double>{e[0], e[1], e[2], e[3], e[4]});
    fast[2 * i] = q.num;
    fast[2 * i + 1] = q.den;
    double num = 0.0, den = 1.0;
    for (int k = 0; k < 5; ++k) {
        const double nk = fabs(e[k]), dk = __dadd_rn(fabs(y[k]), 1e-10);
        if (__dmul_rn(num, dk) < __dmul_rn(nk, den)) {
            num = nk;
            den = dk;
        }
    }
    plain[2 * i] = num;
    plain[2 * i + 1] = den;
}

// (lv, lo, hi, axis points) -> table cell and fraction
__global__ void locate_kernel(const double* in, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double lv = in[4 * i], lo = in[4 * i + 1], hi = in[4 * i + 2];
    const int m = static_cast<int>(in[4 * i + 3]);
    int idx;
    double frac;
    const double len = __dadd_rn(hi, -lo);
    log_locate(lv, lo, len, 1.0 / len, m, idx, frac);
    fast[2 * i] = idx;
    fast[2 * i + 1] = frac;
    const double t = vclamp(__dmul_rn(__dadd_rn(lv, -lo) / len, static_cast<double>(m - 1)), 0.0,
                            static_cast<double>(m - 2));
    idx = table_index(t, 0, m - 2);
    plain[2 * i] = idx;
    plain[2 * i + 1] = __dadd_rn(t, -static_cast<double>(idx));
}

// (r, theta, p_r, p_theta) with a NaN in r or theta -> how many of the five
// derivatives are NaN
__global__ void rhs_kernel(const double* in, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* y = in + 4 * i;
    const double a = 0.9;
    const Vec5<double> d =
        kerr_rhs_f64(KerrHole{1.0, a, a * a, 2.0}, -1.0, 2.0, y[0], y[1], y[2], y[3]);
    fast[2 * i] = isnan(d.r) + isnan(d.th) + isnan(d.ph) + isnan(d.pr) + isnan(d.pth);
    plain[2 * i] = 5.0;
    fast[2 * i + 1] = plain[2 * i + 1] = 0.0;
}

constexpr int kNodes = 17;

// (r, r_min, r_outer) -> scale height from a table of kNodes radii
__global__ void radial_kernel(const double* in, int n, const double* lut, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    DevVolume V;
    V.n_r = kNodes;
    V.H = lut;
    const double r = in[3 * i];
    V.r_min = in[3 * i + 1];
    V.r_outer = in[3 * i + 2];
    V.span = __dadd_rn(V.r_outer, -V.r_min);
    V.inv_span = 1.0 / V.span;
    fast[2 * i] = v_scale_height(V, r);
    fast[2 * i + 1] = plain[2 * i + 1] = 0.0;
    if (r <= V.r_min) {
        plain[2 * i] = lut[0];
    } else if (r >= V.r_outer) {
        plain[2 * i] = lut[kNodes - 1];
    } else {
        const double frac = __dmul_rn(__dadd_rn(r, -V.r_min) / V.span, static_cast<double>(kNodes - 1));
        const int idx = table_index(frac, 0, kNodes - 2);
        plain[2 * i] = v_lerp(lut[idx], lut[idx + 1], __dadd_rn(frac, -static_cast<double>(idx)));
    }
}

}  // namespace

// kind: 0 reciprocal, 1 largest quotient, 2 table cell, 3 radial table, 4
// right-hand side. in: n rows of 2, 10, 4, 3, 4 values; fast, plain: n rows of 2.
extern "C" int f64_edges(int kind, const double* in, int n, double* fast, double* plain) {
    const int cols[5] = {2, 10, 4, 3, 4};
    const size_t bytes_in = sizeof(double) * cols[kind] * n, bytes_out = sizeof(double) * 2 * n;
    std::vector<double> table(kNodes);
    for (int k = 0; k < kNodes; ++k) table[k] = 0.3 + 0.11 * k * k;
    double *d_in = nullptr, *d_fast = nullptr, *d_plain = nullptr, *lut = nullptr;
    bool ok = cudaMalloc(&d_in, bytes_in) == cudaSuccess && cudaMalloc(&d_fast, bytes_out) == cudaSuccess &&
              cudaMalloc(&d_plain, bytes_out) == cudaSuccess &&
              cudaMalloc(&lut, sizeof(double) * kNodes) == cudaSuccess &&
              cudaMemcpy(lut, table.data(), sizeof(double) * kNodes, cudaMemcpyHostToDevice) == cudaSuccess &&
              cudaMemcpy(d_in, in, bytes_in, cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok) {
        const int g = (n + 127) / 128;
        if (kind == 0) recip_kernel<<<g, 128>>>(d_in, n, d_fast, d_plain);
        else if (kind == 1) quotient_kernel<<<g, 128>>>(d_in, n, d_fast, d_plain);
        else if (kind == 2) locate_kernel<<<g, 128>>>(d_in, n, d_fast, d_plain);
        else if (kind == 3) radial_kernel<<<g, 128>>>(d_in, n, lut, d_fast, d_plain);
        else rhs_kernel<<<g, 128>>>(d_in, n, d_fast, d_plain);
        ok = cudaMemcpy(fast, d_fast, bytes_out, cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(plain, d_plain, bytes_out, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    for (double* p : {d_in, d_fast, d_plain, lut}) cudaFree(p);
    return ok ? 0 : -1;
}
