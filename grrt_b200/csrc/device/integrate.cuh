// Dormand-Prince 5(4) attempt and the PI step controller, one attempt per
// call, so a warp advances all its rays in lock-step at attempt granularity.
//
// Method and constants follow RK4::step_kerr_rkdp45
// (include/grrt/geodesic/rk4.h:73-177) and RK4::adaptive_step_kerr_dp45
// (src/rk4.cpp:87-136): Butcher tableau of Dormand & Prince (1980), the
// 5th-order solution is kept, the error is y5 - y4 evaluated with k7 = f(y5),
// the norm is the max over r, theta, phi, p_r, p_theta of |e|/(|y5|+1e-10)
// (the p_t and p_phi terms of the reference norm are identically zero).
#pragma once

#include "kerr.cuh"

namespace grrt_b200 {

// Dormand-Prince (1980) tableau.
namespace dp {
constexpr double a21 = 1.0 / 5.0;
constexpr double a31 = 3.0 / 40.0, a32 = 9.0 / 40.0;
constexpr double a41 = 44.0 / 45.0, a42 = -56.0 / 15.0, a43 = 32.0 / 9.0;
constexpr double a51 = 19372.0 / 6561.0, a52 = -25360.0 / 2187.0, a53 = 64448.0 / 6561.0,
                 a54 = -212.0 / 729.0;
constexpr double a61 = 9017.0 / 3168.0, a62 = -355.0 / 33.0, a63 = 46732.0 / 5247.0,
                 a64 = 49.0 / 176.0, a65 = -5103.0 / 18656.0;
constexpr double b1 = 35.0 / 384.0, b3 = 500.0 / 1113.0, b4 = 125.0 / 192.0,
                 b5 = -2187.0 / 6784.0, b6 = 11.0 / 84.0;
constexpr double e1 = 71.0 / 57600.0, e3 = -71.0 / 16695.0, e4 = 71.0 / 1920.0,
                 e5 = -17253.0 / 339200.0, e6 = 22.0 / 525.0, e7 = -1.0 / 40.0;
}  // namespace dp

template <typename T>
GRRT_HD Vec5<T> axpy(const Vec5<T>& y, T h, const Vec5<T>& k) {
#ifdef GRRT_RHS_PINNED
    if constexpr (sizeof(T) == sizeof(double))
        return Vec5<T>{__fma_rn(h, k.r, y.r), __fma_rn(h, k.th, y.th), __fma_rn(h, k.ph, y.ph),
                       __fma_rn(h, k.pr, y.pr), __fma_rn(h, k.pth, y.pth)};
#endif
    return Vec5<T>{y.r + h * k.r, y.th + h * k.th, y.ph + h * k.ph, y.pr + h * k.pr, y.pth + h * k.pth};
}

#if defined(__CUDACC__) && !defined(GRRT_RHS_GENERIC)
struct DpConst {
    double a21, a31, a32, a41, a42, a43, a51, a52, a53, a54, a61, a62, a63, a64, a65;
    double b1, b3, b4, b5, b6, e1, e3, e4, e5, e6, e7, floor;
    double next[2], err[2];  // a65, b6 and e5, e6
};
static __constant__ DpConst kDp = {dp::a21, dp::a31, dp::a32, dp::a41, dp::a42, dp::a43, dp::a51, dp::a52, dp::a53,
                                   dp::a54, dp::a61, dp::a62, dp::a63, dp::a64, dp::a65, dp::b1, dp::b3, dp::b4,
                                   dp::b5, dp::b6, dp::e1, dp::e3, dp::e4, dp::e5, dp::e6, dp::e7, 1e-10,
                                   {dp::a65, dp::b6}, {dp::e5, dp::e6}};

// n / d, correctly rounded, from inv = the rounded 1 / d: the quotient
// corrected by its exact residual (Markstein, as recip_f64). For numbers far
// from the range's ends.
__device__ __forceinline__ double div_by(double n, double d, double inv) {
    const double q = __dmul_rn(n, inv);
    return __fma_rn(__fma_rn(-d, q, n), inv, q);
}

// n / d, correctly rounded: by the reciprocal for 2^-450 <= |n|, |d| < 2^450
// or n = 0, by the division operator elsewhere.
static __device__ __noinline__ double div_call(double n, double d) { return n / d; }
__device__ __forceinline__ double div_f64(double n, double d) {
    const int hn = __double2hiint(n) & 0x7fffffff, hd = __double2hiint(d) & 0x7fffffff;
    const bool n_ok = static_cast<unsigned>(hn - 0x23d00000) < 0x38400000u || (hn | __double2loint(n)) == 0;
    if (!n_ok || static_cast<unsigned>(hd - 0x23d00000) >= 0x38400000u) return div_call(n, d);
    return div_by(n, d, recip_f64(d));
}

// One DP45 attempt on the device (dp45_attempt_k1 below), roundings written out
// as the compiler fuses the generic form's sums: the first product of each.
// What a stage no longer needs is folded into the sums of the later stages as
// soon as it is known (the terms enter in the tableau's order), so fewer
// registers live through the right-hand sides; phi does not feed the right-hand
// side, so its stage states are not formed.
struct ErrQuotient {
    double num, den;  // error norm = num / den
};

// The error norm of dp45_attempt_k1 as the quotient it is, the largest one
// picked by a tree. Where the products of the comparisons cannot overflow, the
// order of the comparisons does not matter but for quotients within a rounding
// of each other, where either may be taken. qe: the error sum up to the sixth
// stage.
__device__ __forceinline__ ErrQuotient error_quotient(const Vec5<double>& y5, double h, const Vec5<double>& k7,
                                                      const Vec5<double>& qe) {
    const DpConst& C = kDp;
#define GRRT_N(f) fabs(__dmul_rn(h, __fma_rn(C.e7, k7.f, qe.f)))
#define GRRT_D(f) __dadd_rn(fabs(y5.f), C.floor)
    const ErrQuotient q[5] = {{GRRT_N(r), GRRT_D(r)},
                              {GRRT_N(th), GRRT_D(th)},
                              {GRRT_N(ph), GRRT_D(ph)},
                              {GRRT_N(pr), GRRT_D(pr)},
                              {GRRT_N(pth), GRRT_D(pth)}};
#undef GRRT_N
#undef GRRT_D
    auto larger = [](const ErrQuotient& u, const ErrQuotient& v) {
        const bool gt = __dmul_rn(u.num, v.den) < __dmul_rn(v.num, u.den);
        return ErrQuotient{gt ? v.num : u.num, gt ? v.den : u.den};
    };
    unsigned top = 0;  // unsigned: the device's NaN has its sign set, through fabs too
#pragma unroll
    for (int i = 0; i < 5; ++i)
        top = max(top, max(static_cast<unsigned>(__double2hiint(q[i].num)),
                           static_cast<unsigned>(__double2hiint(q[i].den))));
    if (top >= 0x5ff00000u) {  // 2^512, an infinity or a NaN: the terms in order, a NaN skipped
        ErrQuotient m{0.0, 1.0};
        for (int i = 0; i < 5; ++i) m = larger(m, q[i]);
        return m;
    }
    return larger(larger(larger(q[0], q[1]), larger(q[2], q[3])), q[4]);
}

#define GRRT_V4(s) {s(r), s(th), 0.0, s(pr), s(pth)}
#define GRRT_V5(s) {s(r), s(th), s(ph), s(pr), s(pth)}
__device__ __forceinline__ double sum2_f64(double c1, double x1, double c2, double x2) {
    return __fma_rn(c1, x1, __dmul_rn(c2, x2));
}

// The attempt from its fourth stage on.
template <typename F>
__device__ __forceinline__ ErrQuotient dp45_tail_f64(const F& f, const Vec5<double>& y, double h,
                                                     const Vec5<double>& k1, const Vec5<double>& k2,
                                                     const Vec5<double>& k3, const Vec5<double>& k4, Vec5<double>& y5,
                                                     Vec5<double>& k7) {
    const DpConst& C = kDp;
#define GRRT_Q6(f) __fma_rn(C.a64, k4.f, __fma_rn(C.a63, k3.f, sum2_f64(C.a61, k1.f, C.a62, k2.f)))
    const Vec5<double> q6 GRRT_V4(GRRT_Q6);
#define GRRT_QB(f) __fma_rn(C.b4, k4.f, sum2_f64(C.b1, k1.f, C.b3, k3.f))
    Vec5<double> qb GRRT_V5(GRRT_QB);
#define GRRT_QE(f) __fma_rn(C.e4, k4.f, sum2_f64(C.e1, k1.f, C.e3, k3.f))
    Vec5<double> qe GRRT_V5(GRRT_QE);
#define GRRT_S5(f) \
    __fma_rn(h, __fma_rn(C.a54, k4.f, __fma_rn(C.a53, k3.f, sum2_f64(C.a51, k1.f, C.a52, k2.f))), y.f)
    const Vec5<double> k5 = f(Vec5<double> GRRT_V4(GRRT_S5));
#define GRRT_QB5(f) __fma_rn(C.b5, k5.f, qb.f)
    qb = GRRT_V5(GRRT_QB5);
#define GRRT_QE5(f) __fma_rn(C.e5, k5.f, qe.f)
    qe = GRRT_V5(GRRT_QE5);
#define GRRT_S6(f) __fma_rn(h, __fma_rn(C.a65, k5.f, q6.f), y.f)
    const Vec5<double> k6 = f(Vec5<double> GRRT_V4(GRRT_S6));
#define GRRT_Y5(f) __fma_rn(h, __fma_rn(C.b6, k6.f, qb.f), y.f)
    y5 = GRRT_V5(GRRT_Y5);
#define GRRT_QE6(f) __fma_rn(C.e6, k6.f, qe.f)
    qe = GRRT_V5(GRRT_QE6);
    k7 = f(y5);
#undef GRRT_S5
#undef GRRT_S6
#undef GRRT_Q6
#undef GRRT_QB
#undef GRRT_QE
#undef GRRT_QB5
#undef GRRT_QE5
#undef GRRT_QE6
#undef GRRT_Y5
    return error_quotient(y5, h, k7, qe);
}

// dp45_tail_f64 with its last three stages as one loop body, for kernels whose
// code must stay small: sums of no later use are formed as well.
template <typename F>
__device__ __forceinline__ ErrQuotient dp45_tail_rolled_f64(const F& f, const Vec5<double>& y, double h,
                                                            const Vec5<double>& k1, const Vec5<double>& k2,
                                                            const Vec5<double>& k3, const Vec5<double>& k4,
                                                            Vec5<double>& y5, Vec5<double>& k7) {
    const DpConst& C = kDp;
#define GRRT_S5(f) \
    __fma_rn(h, __fma_rn(C.a54, k4.f, __fma_rn(C.a53, k3.f, sum2_f64(C.a51, k1.f, C.a52, k2.f))), y.f)
    Vec5<double> s GRRT_V4(GRRT_S5);
#define GRRT_Q6(f) __fma_rn(C.a64, k4.f, __fma_rn(C.a63, k3.f, sum2_f64(C.a61, k1.f, C.a62, k2.f)))
    Vec5<double> qa GRRT_V4(GRRT_Q6);
#define GRRT_QB(f) __fma_rn(C.b4, k4.f, sum2_f64(C.b1, k1.f, C.b3, k3.f))
    const Vec5<double> qb GRRT_V5(GRRT_QB);
#define GRRT_QE(f) __fma_rn(C.e4, k4.f, sum2_f64(C.e1, k1.f, C.e3, k3.f))
    Vec5<double> qe GRRT_V5(GRRT_QE);
#undef GRRT_S5
#undef GRRT_Q6
#undef GRRT_QB
#undef GRRT_QE
#pragma unroll 1
    for (int i = 0;; ++i) {
        k7 = f(s);
        if (i == 2) break;
        const double ca = C.next[i], ce = C.err[i];
#define GRRT_NEXT(f) __fma_rn(h, __fma_rn(ca, k7.f, qa.f), y.f)
        s = GRRT_V5(GRRT_NEXT);
#define GRRT_SB(f) __fma_rn(C.b5, k7.f, qb.f)
        qa = GRRT_V5(GRRT_SB);
#define GRRT_SE(f) __fma_rn(ce, k7.f, qe.f)
        qe = GRRT_V5(GRRT_SE);
#undef GRRT_NEXT
#undef GRRT_SB
#undef GRRT_SE
    }
    y5 = s;
    return error_quotient(y5, h, k7, qe);
}

// f: the right-hand side of a state (its phi unused).
template <typename F>
__device__ __forceinline__ ErrQuotient dp45_attempt_f64(const F& f, const Vec5<double>& y, double h,
                                                        const Vec5<double>& k1, Vec5<double>& y5, Vec5<double>& k7) {
    const DpConst& C = kDp;
#define GRRT_S2(f) __fma_rn(h, __dmul_rn(C.a21, k1.f), y.f)
    const Vec5<double> k2 = f(Vec5<double> GRRT_V4(GRRT_S2));
#define GRRT_S3(f) __fma_rn(h, sum2_f64(C.a31, k1.f, C.a32, k2.f), y.f)
    const Vec5<double> k3 = f(Vec5<double> GRRT_V4(GRRT_S3));
#define GRRT_S4(f) __fma_rn(h, __fma_rn(C.a43, k3.f, sum2_f64(C.a41, k1.f, C.a42, k2.f)), y.f)
    const Vec5<double> k4 = f(Vec5<double> GRRT_V4(GRRT_S4));
#undef GRRT_S2
#undef GRRT_S3
#undef GRRT_S4
    return dp45_tail_f64(f, y, h, k1, k2, k3, k4, y5, k7);
}

// Stages 2 to 4 of an attempt, or of a classic RK4 step (rk4_step: its stage
// coefficients 1/2, 1/2, 1 in the same sums, where a zero coefficient leaves
// the bits), so that lanes of both kinds evaluate these right-hand sides
// together.
template <typename F>
__device__ __forceinline__ void shared_stages_f64(const F& f, bool rk4, const Vec5<double>& y, double h,
                                                  const Vec5<double>& k1, Vec5<double>& k2, Vec5<double>& k3,
                                                  Vec5<double>& k4) {
    const double c21 = rk4 ? 0.5 : kDp.a21, c31 = rk4 ? 0.0 : kDp.a31, c32 = rk4 ? 0.5 : kDp.a32;
    const double c41 = rk4 ? 0.0 : kDp.a41, c42 = rk4 ? 0.0 : kDp.a42, c43 = rk4 ? 1.0 : kDp.a43;
#define GRRT_S2(f) __fma_rn(h, __dmul_rn(c21, k1.f), y.f)
    k2 = f(Vec5<double> GRRT_V4(GRRT_S2));
#define GRRT_S3(f) __fma_rn(h, sum2_f64(c31, k1.f, c32, k2.f), y.f)
    k3 = f(Vec5<double> GRRT_V4(GRRT_S3));
#define GRRT_S4(f) __fma_rn(h, __fma_rn(c43, k3.f, sum2_f64(c41, k1.f, c42, k2.f)), y.f)
    k4 = f(Vec5<double> GRRT_V4(GRRT_S4));
#undef GRRT_S2
#undef GRRT_S3
#undef GRRT_S4
}

// The end state of an RK4 step of length h from its four right-hand sides.
__device__ __forceinline__ Vec5<double> rk4_end_f64(const Vec5<double>& y, double h, const Vec5<double>& k1,
                                                    const Vec5<double>& k2, const Vec5<double>& k3,
                                                    const Vec5<double>& k4) {
    const double w = div_f64(h, 6.0);
#define GRRT_R4(f) __fma_rn(__dadd_rn(__fma_rn(2.0, k3.f, __fma_rn(2.0, k2.f, k1.f)), k4.f), w, y.f)
    return Vec5<double> GRRT_V5(GRRT_R4);
#undef GRRT_R4
}
#undef GRRT_V4
#undef GRRT_V5
#endif

// Classic RK4 step (include/grrt/geodesic/rk4.h:34-52).
template <typename T>
GRRT_HD Vec5<T> rk4_step(T M, T a, T pt, T pph, const Vec5<T>& y, T h) {
    const Vec5<T> k1 = kerr_rhs<T>(M, a, pt, pph, y);
    const Vec5<T> k2 = kerr_rhs<T>(M, a, pt, pph, axpy(y, h * T(0.5), k1));
    const Vec5<T> k3 = kerr_rhs<T>(M, a, pt, pph, axpy(y, h * T(0.5), k2));
    const Vec5<T> k4 = kerr_rhs<T>(M, a, pt, pph, axpy(y, h, k3));
#ifdef GRRT_RHS_PINNED
    if constexpr (sizeof(T) == sizeof(double)) return rk4_end_f64(y, h, k1, k2, k3, k4);
#endif
    const T w = h / T(6);
#define GRRT_RK4C(f) y.f + (k1.f + T(2) * k2.f + T(2) * k3.f + k4.f) * w
    return Vec5<T>{GRRT_RK4C(r), GRRT_RK4C(th), GRRT_RK4C(ph), GRRT_RK4C(pr), GRRT_RK4C(pth)};
#undef GRRT_RK4C
}

// One DP45 attempt with k1 = f(y) given by the caller: returns the error
// norm, the 5th-order state in y5 and k7 = f(y5). The reference evaluates
// f(y) afresh at every attempt; mathematically it is the previous accepted
// attempt's k7 (same state, same constants) or the rejected attempt's k1
// (same state), so a caller that keeps it evaluates six right-hand sides per
// attempt instead of seven. The kept value has the bits of a fresh one: on the
// host without FMA contraction, on the device with the roundings written out
// (not under GRRT_RHS_GENERIC, where each inlined copy is contracted by itself).
template <typename T>
GRRT_HD T dp45_attempt_k1(T M, T a, T pt, T pph, const Vec5<T>& y, T h, const Vec5<T>& k1, Vec5<T>& y5,
                          Vec5<T>& k7_out) {
#ifdef GRRT_RHS_PINNED
    if constexpr (sizeof(T) == sizeof(double)) {
        auto f = [&](const Vec5<double>& s) { return kerr_rhs<double>(M, a, pt, pph, s); };
        const ErrQuotient q = dp45_attempt_f64(f, y, h, k1, y5, k7_out);
        return div_f64(q.num, q.den);
    }
#endif
    using namespace dp;
#define GRRT_S2(f) y.f + h * (T(a21) * k1.f)
    const Vec5<T> k2 = kerr_rhs<T>(M, a, pt, pph, Vec5<T>{GRRT_S2(r), GRRT_S2(th), GRRT_S2(ph), GRRT_S2(pr), GRRT_S2(pth)});
#define GRRT_S3(f) y.f + h * (T(a31) * k1.f + T(a32) * k2.f)
    const Vec5<T> k3 = kerr_rhs<T>(M, a, pt, pph, Vec5<T>{GRRT_S3(r), GRRT_S3(th), GRRT_S3(ph), GRRT_S3(pr), GRRT_S3(pth)});
#define GRRT_S4(f) y.f + h * (T(a41) * k1.f + T(a42) * k2.f + T(a43) * k3.f)
    const Vec5<T> k4 = kerr_rhs<T>(M, a, pt, pph, Vec5<T>{GRRT_S4(r), GRRT_S4(th), GRRT_S4(ph), GRRT_S4(pr), GRRT_S4(pth)});
#define GRRT_S5(f) y.f + h * (T(a51) * k1.f + T(a52) * k2.f + T(a53) * k3.f + T(a54) * k4.f)
    const Vec5<T> k5 = kerr_rhs<T>(M, a, pt, pph, Vec5<T>{GRRT_S5(r), GRRT_S5(th), GRRT_S5(ph), GRRT_S5(pr), GRRT_S5(pth)});
#define GRRT_S6(f) y.f + h * (T(a61) * k1.f + T(a62) * k2.f + T(a63) * k3.f + T(a64) * k4.f + T(a65) * k5.f)
    const Vec5<T> k6 = kerr_rhs<T>(M, a, pt, pph, Vec5<T>{GRRT_S6(r), GRRT_S6(th), GRRT_S6(ph), GRRT_S6(pr), GRRT_S6(pth)});
#define GRRT_Y5(f) y.f + h * (T(b1) * k1.f + T(b3) * k3.f + T(b4) * k4.f + T(b5) * k5.f + T(b6) * k6.f)
    y5 = Vec5<T>{GRRT_Y5(r), GRRT_Y5(th), GRRT_Y5(ph), GRRT_Y5(pr), GRRT_Y5(pth)};
#define GRRT_E6(f) (T(e1) * k1.f + T(e3) * k3.f + T(e4) * k4.f + T(e5) * k5.f + T(e6) * k6.f)
    Vec5<T> e = Vec5<T>{GRRT_E6(r), GRRT_E6(th), GRRT_E6(ph), GRRT_E6(pr), GRRT_E6(pth)};
#undef GRRT_S2
#undef GRRT_S3
#undef GRRT_S4
#undef GRRT_S5
#undef GRRT_S6
#undef GRRT_Y5
#undef GRRT_E6
    const Vec5<T> k7 = kerr_rhs<T>(M, a, pt, pph, y5);
    k7_out = k7;
    // err = max |h (sum e_i k_i)| / (|y5| + 1e-10); max written as the
    // standard library's (a < b) ? b : a so a NaN term is skipped as there.
    // The largest quotient is picked by cross-multiplied comparisons
    // (numerators >= 0, denominators > 0) and divided once: the same value as
    // dividing each and taking the maximum, but for quotients within a rounding
    // of each other, where either may be taken. A NaN term fails every
    // comparison and is skipped.
    T num = T(0), den = T(1);
#define GRRT_ERR(f)                                            \
    {                                                          \
        const T n_ = fabs(h * (e.f + T(e7) * k7.f));           \
        const T d_ = fabs(y5.f) + T(1e-10);                    \
        if (num * d_ < n_ * den) {                             \
            num = n_;                                          \
            den = d_;                                          \
        }                                                      \
    }
    GRRT_ERR(r) GRRT_ERR(th) GRRT_ERR(ph) GRRT_ERR(pr) GRRT_ERR(pth)
#undef GRRT_ERR
    return num / den;
}

// One DP45 attempt from scratch: returns the 5th-order state in y5 and the error norm.
template <typename T>
GRRT_HD T dp45_attempt(T M, T a, T pt, T pph, const Vec5<T>& y, T h, Vec5<T>& y5) {
    const Vec5<T> k1 = kerr_rhs<T>(M, a, pt, pph, y);
    Vec5<T> k7;
    return dp45_attempt_k1<T>(M, a, pt, pph, y, h, k1, y5, k7);
}

// f(y) in FP32 as the mixed-precision attempt forms it (state rounded to FP32).
GRRT_HD Vec5<float> mixed_k1(float M, float a, float pt, float pph, const Vec5<double>& y) {
    const Vec5<float> yf{static_cast<float>(y.r), static_cast<float>(y.th), static_cast<float>(y.ph),
                         static_cast<float>(y.pr), static_cast<float>(y.pth)};
    return kerr_rhs<float>(M, a, pt, pph, yf);
}

// 1/x of the FP32 error norm (x > 0, far from the range's ends).
GRRT_HD float recip_err(float x) {
#ifdef GRRT_RHS_PINNED
    return rcp_approx(x);
#else
    return recip(x);
#endif
}

// Packed FP32 pairs: sm_100's two-wide FP32 fused multiply-add and multiply,
// one instruction for two lanes, each lane rounded as fmaf / the float
// product (elsewhere the lanes are computed one by one, with the same results).
GRRT_HD float2 pk(float x, float y) { return make_float2(x, y); }
GRRT_HD float2 pk_fma(float2 a, float2 b, float2 c) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __ffma2_rn(a, b, c);
#else
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#endif
}
GRRT_HD float2 pk_mul(float2 a, float2 b) {
#if defined(__CUDA_ARCH__) && __CUDA_ARCH__ >= 1000
    return __fmul2_rn(a, b);
#else
    return make_float2(a.x * b.x, a.y * b.y);
#endif
}

// The four components that feed the right-hand side as two packed pairs
// (r, theta), (p_r, p_theta); phi is kept apart, its stage states are not formed.
struct Pk4 {
    float2 a, b;
};
GRRT_HD Pk4 pack4(const Vec5<float>& v) { return Pk4{pk(v.r, v.th), pk(v.pr, v.pth)}; }
// c * v, and c * v + w, per component
GRRT_HD Pk4 pk4_mul(float c, const Pk4& v) { return Pk4{pk_mul(pk(c, c), v.a), pk_mul(pk(c, c), v.b)}; }
GRRT_HD Pk4 pk4_fma(float c, const Pk4& v, const Pk4& w) {
    return Pk4{pk_fma(pk(c, c), v.a, w.a), pk_fma(pk(c, c), v.b, w.b)};
}

// Mixed-precision attempt: the seven right-hand sides and the stage sums in
// FP32, the state and its update in FP64 (y5 = y + double(h * sum b_i k_i)),
// so round-off does not accumulate along the ray. The error norm is formed in
// FP32; its noise floor (about 1e-7 of |h k|/|y|) is why FP32 steps are
// controlled against their own tolerance (DevScene::tol_fp32). The stage sums
// run on packed pairs: each stage state is y + h * (sum_j a_sj k_j), the sum
// accumulated in the tableau's order with fused multiply-adds.
// k1 = mixed_k1(y) is given by the caller (the previous accepted attempt's
// k7, which is f at float(y5) = float(new y), or the rejected attempt's k1).
// mixed_attempt_yf also takes Y = float(y) and gives Y5 = float(y5), so a
// caller that keeps it converts each state once.
GRRT_HD double mixed_attempt_yf(float M, float a, float pt, float pph, const Vec5<double>& y, const Pk4& Y, double dl,
                                const Vec5<float>& k1v, Vec5<double>& y5, Pk4& Y5, Vec5<float>& k7_out) {
    using namespace dp;
    const float h = static_cast<float>(dl);
    // f(y + h * sum), packed, and the phi component
    auto stage = [&](const Pk4& sum, float& ph) {
        const Pk4 v = pk4_fma(h, sum, Y);
        const Vec5<float> k = kerr_rhs<float>(M, a, pt, pph, Vec5<float>{v.a.x, v.a.y, 0.0f, v.b.x, v.b.y});
        ph = k.ph;
        return pack4(k);
    };
    float p2, p3, p4, p5, p6;
    const float p1 = k1v.ph;
    const Pk4 K1 = pack4(k1v);
    const Pk4 K2 = stage(pk4_mul(float(a21), K1), p2);
    const Pk4 K3 = stage(pk4_fma(float(a32), K2, pk4_mul(float(a31), K1)), p3);
    const Pk4 K4 = stage(pk4_fma(float(a43), K3, pk4_fma(float(a42), K2, pk4_mul(float(a41), K1))), p4);
    const Pk4 K5 = stage(
        pk4_fma(float(a54), K4, pk4_fma(float(a53), K3, pk4_fma(float(a52), K2, pk4_mul(float(a51), K1)))), p5);
    const Pk4 K6 = stage(
        pk4_fma(float(a65), K5,
                pk4_fma(float(a64), K4, pk4_fma(float(a63), K3, pk4_fma(float(a62), K2, pk4_mul(float(a61), K1))))),
        p6);
    const Pk4 B = pk4_fma(float(b6), K6,
                          pk4_fma(float(b5), K5, pk4_fma(float(b4), K4, pk4_fma(float(b3), K3, pk4_mul(float(b1), K1)))));
    const float Bp = fmaf(float(b6), p6, fmaf(float(b5), p5, fmaf(float(b4), p4, fmaf(float(b3), p3, float(b1) * p1))));
    const Pk4 I = pk4_mul(h, B);
    y5 = Vec5<double>{y.r + double(I.a.x), y.th + double(I.a.y), y.ph + double(h * Bp), y.pr + double(I.b.x),
                      y.pth + double(I.b.y)};
    const Pk4 E = pk4_fma(float(e6), K6,
                          pk4_fma(float(e5), K5, pk4_fma(float(e4), K4, pk4_fma(float(e3), K3, pk4_mul(float(e1), K1)))));
    const float Ep = fmaf(float(e6), p6, fmaf(float(e5), p5, fmaf(float(e4), p4, fmaf(float(e3), p3, float(e1) * p1))));
    const Vec5<float> y5f{static_cast<float>(y5.r), static_cast<float>(y5.th), static_cast<float>(y5.ph),
                          static_cast<float>(y5.pr), static_cast<float>(y5.pth)};
    const Vec5<float> k7 = kerr_rhs<float>(M, a, pt, pph, y5f);
    k7_out = k7;
    Y5 = pack4(y5f);
    const Pk4 e4v = pk4_fma(float(e7), pack4(k7), E);
    const float ep = fmaf(float(e7), k7.ph, Ep);
    float err = 0.0f;
    auto term = [&](float e, float yv) {
        const float v = fabsf(h * e) * recip_err(fabsf(yv) + 1e-10f);
        err = (err < v) ? v : err;
    };
    term(e4v.a.x, y5f.r);
    term(e4v.a.y, y5f.th);
    term(ep, y5f.ph);
    term(e4v.b.x, y5f.pr);
    term(e4v.b.y, y5f.pth);
    return static_cast<double>(err);
}

GRRT_HD Pk4 pack_state(const Vec5<double>& y) {
    return Pk4{pk(static_cast<float>(y.r), static_cast<float>(y.th)),
               pk(static_cast<float>(y.pr), static_cast<float>(y.pth))};
}

GRRT_HD double mixed_attempt_k1(float M, float a, float pt, float pph, const Vec5<double>& y, double dl,
                                const Vec5<float>& k1v, Vec5<double>& y5, Vec5<float>& k7_out) {
    Pk4 Y5;
    return mixed_attempt_yf(M, a, pt, pph, y, pack_state(y), dl, k1v, y5, Y5, k7_out);
}

GRRT_HD double mixed_attempt_impl(float M, float a, float pt, float pph, const Vec5<double>& y, double dl,
                                  Vec5<double>& y5, Vec5<float>& k7_out) {
    return mixed_attempt_k1(M, a, pt, pph, y, dl, mixed_k1(M, a, pt, pph, y), y5, k7_out);
}

// Outcome of the controller after one attempt (src/rk4.cpp:87-136).
struct StepDecision {
    bool accept;    // take y5 and start a new outer step
    double next;    // accepted: step size for the next outer step; rejected: the new trial size
};

// (tol/err)^0.2 for the step-size factor. The factor only sets the next trial
// step, on which the solution depends through the truncation error (a relative
// change d in the step moves the result by about 5 d times the local error), so
// single precision (2^-22 relative) is ample and avoids an FP64 pow per attempt.
GRRT_HD double step_factor_pow(double x) {
#ifdef __CUDA_ARCH__
    return static_cast<double>(__powf(static_cast<float>(x), 0.2f));
#else
    return static_cast<double>(powf(static_cast<float>(x), 0.2f));
#endif
}

GRRT_HD double step_quotient(double tol, double err) {
#ifdef GRRT_RHS_PINNED
    return div_f64(tol, err);
#else
    return tol / err;
#endif
}

// retry = number of rejected attempts so far in this outer step (0..20). The
// 21st attempt (retry == 20) is taken unconditionally with next = dl, as the
// reference's "exhausted retries" path.
GRRT_HD StepDecision pi_control(double err, double tol, double dl, int retry,
                                                   double r5) {
    constexpr double safety = 0.9, grow_max = 5.0, shrink_max = 0.2, dl_min = 1e-6;
    StepDecision d;
    const double ar = fabs(r5);
    const double cap = 5.0 * ((ar < 1.0) ? 1.0 : ar);
    if (retry >= 20) {
        d.accept = true;
        d.next = dl;
        return d;
    }
    if (err <= tol) {
        double f = (err > 1e-30) ? safety * step_factor_pow(step_quotient(tol, err)) : grow_max;
        f = (f < 1.0) ? 1.0 : (grow_max < f) ? grow_max : f;
        const double nx = dl * f;
        d.accept = true;
        d.next = (cap < nx) ? cap : nx;
        return d;
    }
    double f = safety * step_factor_pow(step_quotient(tol, err));
    f = (f < shrink_max) ? shrink_max : (1.0 < f) ? 1.0 : f;
    const double ndl = dl * f;
    if (ndl < dl_min) {
        d.accept = true;
        d.next = (cap < dl_min) ? cap : dl_min;
        return d;
    }
    d.accept = false;
    d.next = ndl;
    return d;
}

#if defined(__CUDACC__) && !defined(GRRT_RHS_GENERIC)
// pi_control of the error norm q.num / q.den, with the same decision and the
// same step to the bit but without its two divisions in sequence: the factor
// needs (tol / err) rounded to single precision only, so tol * den * (1 / num),
// a few ulp off, rounds alike unless it lies that close to a rounding boundary,
// and err <= tol is the same as that quotient >= 1 unless it is as close to 1.
// Those cases (1 in 10^7), numbers near the range's ends and tolerances
// where the 1e-30 rule could matter take pi_control. Positive doubles are
// compared as integers, off the FP64 pipe.
static __device__ __noinline__ StepDecision pi_control_call(double num, double den, double tol, double dl, int retry,
                                                            double r5) {
    return pi_control(num / den, tol, dl, retry, r5);
}

__device__ __forceinline__ StepDecision pi_control_q(const ErrQuotient& q, double tol, double dl, int retry,
                                                     double r5) {
    constexpr double safety = 0.9, grow_max = 5.0, shrink_max = 0.2, dl_min = 1e-6;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q.num));
    const double e = __fma_rn(-q.num, y, 1.0);
    y = __fma_rn(y, __fma_rn(e, e, e), y);
    const double ratio = __dmul_rn(__dmul_rn(tol, q.den), y);  // tol / err
    const long long rb = __double_as_longlong(ratio);
    // 2^-450 <= num, den < 2^450 (a negative or NaN num fails as well)
    const bool in_range = static_cast<unsigned>(__double2hiint(q.num) - 0x23d00000) < 0x38400000u &&
                          static_cast<unsigned>(__double2hiint(q.den) - 0x23d00000) < 0x38400000u;
    const bool near_half = ((static_cast<unsigned>(rb) - 0x10000000u + 16u) & 0x1fffffffu) <= 32u;
    const bool near_one = static_cast<unsigned long long>(rb - 0x3ff0000000000000ll + 64) <= 128ull;
    if (!in_range || near_half || near_one || !(tol >= 1e-20 && tol <= 1e20))
        return pi_control_call(q.num, q.den, tol, dl, retry, r5);
    auto less = [](double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); };
    const bool ok = rb >= 0x3ff0000000000000ll;
    double f = __dmul_rn(safety, static_cast<double>(__powf(static_cast<float>(ratio), 0.2f)));
    const double lo = ok ? 1.0 : shrink_max, hi = ok ? grow_max : 1.0;
    f = less(f, lo) ? lo : less(hi, f) ? hi : f;
    const double ar = fabs(r5);
    const double cap = __dmul_rn(5.0, less(ar, 1.0) ? 1.0 : ar);
    const double nx = __dmul_rn(dl, f);
    const bool tiny = !ok && less(nx, dl_min);
    StepDecision d;
    d.accept = ok || tiny || retry >= 20;
    d.next = tiny ? dl_min : nx;
    if ((ok || tiny) && less(cap, d.next)) d.next = cap;
    if (retry >= 20) d.next = dl;
    return d;
}
#endif

// The FP32 pass's controller: pi_control with (tol/err)^0.2 formed from a
// single-precision quotient (the FP32 error norm carries no more digits).
GRRT_HD double step_factor_ratio(double tol, double err) {
#ifdef __CUDA_ARCH__
    return static_cast<double>(__powf(__fdividef(static_cast<float>(tol), static_cast<float>(err)), 0.2f));
#else
    return static_cast<double>(powf(static_cast<float>(tol) / static_cast<float>(err), 0.2f));
#endif
}

// err is a single-precision value. Selects in place of branches: a warp nearly
// always holds both outcomes.
GRRT_HD StepDecision pi_control_f32(double err, double tol, double dl, int retry,
                                                   double r5) {
    constexpr double safety = 0.9, grow_max = 5.0, shrink_max = 0.2, dl_min = 1e-6;
    const bool ok = err <= tol;
    const double lo = ok ? 1.0 : shrink_max, hi = ok ? grow_max : 1.0;
    double f = safety * step_factor_ratio(tol, err);
    f = (f < lo) ? lo : (hi < f) ? hi : f;
    if (ok && !(err > 1e-30)) f = grow_max;
    const double ar = fabs(r5);
    const double cap = 5.0 * ((ar < 1.0) ? 1.0 : ar);
    const double nx = dl * f;
    const bool tiny = !ok && nx < dl_min;
    StepDecision d;
    d.accept = ok || tiny || retry >= 20;
    d.next = tiny ? dl_min : nx;
    if ((ok || tiny) && cap < d.next) d.next = cap;
    if (retry >= 20) d.next = dl;
    return d;
}

}  // namespace grrt_b200
