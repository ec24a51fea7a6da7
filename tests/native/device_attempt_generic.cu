// The generic right-hand sides and attempt; test-only (device_attempt_bits.cu).
#define GRRT_RHS_GENERIC 1
#define GRRT_RHS_CALL_F64 1
#include "../../grrt_b200/csrc/device/integrate.cuh"
#include "device_attempt_bits.cuh"

using namespace grrt_b200;

namespace {

__global__ void generic_kernel(int kind, const AttemptRow* rows, int n, double* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const AttemptRow& w = rows[i];
    double* o = out + static_cast<size_t>(kAttemptOut) * i;
    for (int k = 0; k < kAttemptOut; ++k) o[k] = 0.0;
    const Vec5<double> y{w.r, w.th, w.ph, w.pr, w.pth};
    if (kind == 0) {
        const Vec5<float> yf{static_cast<float>(y.r), static_cast<float>(y.th), static_cast<float>(y.ph),
                             static_cast<float>(y.pr), static_cast<float>(y.pth)};
        const Vec5<float> d = kerr_rhs<float>(static_cast<float>(w.M), static_cast<float>(w.a),
                                              static_cast<float>(w.pt), static_cast<float>(w.pph), yf);
        o[0] = d.r, o[1] = d.th, o[2] = d.ph, o[3] = d.pr, o[4] = d.pth;
        return;
    }
    const Vec5<double> k1 = kerr_rhs<double>(w.M, w.a, w.pt, w.pph, y);
    Vec5<double> e = k1, k7{};
    if (kind == 2) o[10] = dp45_attempt_k1<double>(w.M, w.a, w.pt, w.pph, y, w.h, k1, e, k7);
    if (kind == 3) e = rk4_step<double>(w.M, w.a, w.pt, w.pph, y, w.h);
    o[0] = e.r, o[1] = e.th, o[2] = e.ph, o[3] = e.pr, o[4] = e.pth;
    o[5] = k7.r, o[6] = k7.th, o[7] = k7.ph, o[8] = k7.pr, o[9] = k7.pth;
}

}  // namespace

void launch_generic(int kind, const AttemptRow* rows, int n, double* out) {
    generic_kernel<<<(n + 127) / 128, 128>>>(kind, rows, n, out);
}
