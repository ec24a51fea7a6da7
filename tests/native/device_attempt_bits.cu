// Device build of the right-hand sides, the DP45 attempt in its forms and the
// RK4 step beside the generic bodies (device_attempt_generic.cu), so a GPU test
// can compare the bits. Test-only.
#include "../../grrt_b200/csrc/device/integrate.cuh"
#include "device_attempt_bits.cuh"

using namespace grrt_b200;

namespace {

// kind: 0 FP32 right-hand side, 1 FP64 right-hand side, 2 attempt, 3 RK4 step
// (2 and 3 from shared stages with `shared`, the attempt's last stages as a loop
// with `rolled`)
__global__ void device_kernel(int kind, bool shared, bool rolled, const AttemptRow* rows, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const AttemptRow& w = rows[i];
    double* o = out + static_cast<size_t>(kAttemptOut) * i;
    for (int k = 0; k < kAttemptOut; ++k) o[k] = 0.0;
    const Vec5<double> y{w.r, w.th, w.ph, w.pr, w.pth};
    if (kind == 0) {
        const Vec5<float> d =
            kerr_rhs_f32(static_cast<float>(w.M), static_cast<float>(w.a), static_cast<float>(w.pt),
                         static_cast<float>(w.pph), static_cast<float>(y.r), static_cast<float>(y.th),
                         static_cast<float>(y.pr), static_cast<float>(y.pth));
        o[0] = d.r, o[1] = d.th, o[2] = d.ph, o[3] = d.pr, o[4] = d.pth;
        return;
    }
    auto f = [&](const Vec5<double>& s) {
        return kerr_rhs_f64(KerrHole{w.M, w.a, w.a * w.a, 2.0 * w.M}, w.pt, w.pph, s.r, s.th, s.pr, s.pth);
    };
    const Vec5<double> k1 = f(y);
    Vec5<double> e = k1, k7{}, k2, k3, k4;
    if (kind >= 2 && shared) shared_stages_f64(f, kind == 3, y, w.h, k1, k2, k3, k4);
    if (kind == 2) {
        ErrQuotient q;
        if (!shared) q = dp45_attempt_f64(f, y, w.h, k1, e, k7);
        else if (rolled) q = dp45_tail_rolled_f64(f, y, w.h, k1, k2, k3, k4, e, k7);
        else q = dp45_tail_f64(f, y, w.h, k1, k2, k3, k4, e, k7);
        o[10] = q.num / q.den;
    }
    if (kind == 3) e = shared ? rk4_end_f64(y, w.h, k1, k2, k3, k4) : rk4_step<double>(w.M, w.a, w.pt, w.pph, y, w.h);
    o[0] = e.r, o[1] = e.th, o[2] = e.ph, o[3] = e.pr, o[4] = e.pth;
    o[5] = k7.r, o[6] = k7.th, o[7] = k7.ph, o[8] = k7.pr, o[9] = k7.pth;
}

}  // namespace

// rows: n x 10 values (AttemptRow); fast, plain: n x kAttemptOut.
extern "C" int attempt_bits(int kind, int shared, int rolled, const double* rows, int n, double* fast, double* plain) {
    const size_t in = sizeof(AttemptRow) * n, out = sizeof(double) * kAttemptOut * n;
    AttemptRow* d_rows = nullptr;
    double *d_fast = nullptr, *d_plain = nullptr;
    bool ok = cudaMalloc(&d_rows, in) == cudaSuccess && cudaMalloc(&d_fast, out) == cudaSuccess &&
              cudaMalloc(&d_plain, out) == cudaSuccess &&
              cudaMemcpy(d_rows, rows, in, cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok) {
        device_kernel<<<(n + 127) / 128, 128>>>(kind, shared != 0, rolled != 0, d_rows, n, d_fast);
        launch_generic(kind, d_rows, n, d_plain);
        ok = cudaMemcpy(fast, d_fast, out, cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(plain, d_plain, out, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFree(d_rows);
    cudaFree(d_fast);
    cudaFree(d_plain);
    return ok ? 0 : -1;
}
