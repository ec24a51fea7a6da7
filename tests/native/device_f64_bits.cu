// Device build of the FP64 right-hand side's building blocks beside the plain
// operations they stand for, so a GPU test can compare the bits. Test-only.
#include "../../grrt_b200/csrc/device/integrate.cuh"

using namespace grrt_b200;

namespace {

__global__ void sincos_kernel(const double* x, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s, c;
    sincos_clamped_f64(x[i], s, c);
    fast[2 * i] = s;
    fast[2 * i + 1] = c;
    fast_sincos(x[i], s, c);
    if (fabs(s) < 1e-10) s = (s >= 0.0) ? 1e-10 : -1e-10;
    plain[2 * i] = s;
    plain[2 * i + 1] = c;
}

__global__ void divide_kernel(const double* a, const double* b, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    fast[2 * i] = recip_f64(b[i]);
    plain[2 * i] = 1.0 / b[i];
    fast[2 * i + 1] = div_f64(a[i], b[i]);
    plain[2 * i + 1] = a[i] / b[i];
}

__global__ void control_kernel(const double* num, const double* den, const double* dl, const int* retry,
                               const double* r, double tol, int n, double* fast, double* plain) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const StepDecision a = pi_control_q(ErrQuotient{num[i], den[i]}, tol, dl[i], retry[i], r[i]);
    const StepDecision b = pi_control(num[i] / den[i], tol, dl[i], retry[i], r[i]);
    fast[2 * i] = a.next;
    fast[2 * i + 1] = a.accept;
    plain[2 * i] = b.next;
    plain[2 * i + 1] = b.accept;
}

// Device copies of host arrays, freed at the end of a call.
struct Buffers {
    void* p[8];
    int n = 0;
    bool ok = true;
    template <typename T>
    T* make(const T* host, size_t count) {
        void* d = nullptr;
        ok = ok && cudaMalloc(&d, count * sizeof(T)) == cudaSuccess;
        if (ok && host) ok = cudaMemcpy(d, host, count * sizeof(T), cudaMemcpyHostToDevice) == cudaSuccess;
        p[n++] = d;
        return static_cast<T*>(d);
    }
    int finish(const double* d_fast, const double* d_plain, int n_out, double* fast, double* plain) {
        ok = ok && cudaMemcpy(fast, d_fast, n_out * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess &&
             cudaMemcpy(plain, d_plain, n_out * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess;
        return ok ? 0 : -1;
    }
    ~Buffers() {
        for (int i = 0; i < n; ++i) cudaFree(p[i]);
    }
};

}  // namespace

extern "C" {

int f64_sincos(const double* x, int n, double* fast, double* plain) {
    Buffers b;
    const double* dx = b.make(x, n);
    double* f = b.make<double>(nullptr, 2 * n);
    double* q = b.make<double>(nullptr, 2 * n);
    if (b.ok) sincos_kernel<<<(n + 127) / 128, 128>>>(dx, n, f, q);
    return b.finish(f, q, 2 * n, fast, plain);
}

int f64_divide(const double* a, const double* d, int n, double* fast, double* plain) {
    Buffers b;
    const double *da = b.make(a, n), *dd = b.make(d, n);
    double* f = b.make<double>(nullptr, 2 * n);
    double* q = b.make<double>(nullptr, 2 * n);
    if (b.ok) divide_kernel<<<(n + 127) / 128, 128>>>(da, dd, n, f, q);
    return b.finish(f, q, 2 * n, fast, plain);
}

int f64_control(const double* num, const double* den, const double* dl, const int* retry, const double* r, double tol,
                int n, double* fast, double* plain) {
    Buffers b;
    const double *dn = b.make(num, n), *dd = b.make(den, n), *dh = b.make(dl, n), *dr = b.make(r, n);
    const int* dt = b.make(retry, n);
    double* f = b.make<double>(nullptr, 2 * n);
    double* q = b.make<double>(nullptr, 2 * n);
    if (b.ok) control_kernel<<<(n + 127) / 128, 128>>>(dn, dd, dh, dt, dr, tol, n, f, q);
    return b.finish(f, q, 2 * n, fast, plain);
}

}  // extern "C"
