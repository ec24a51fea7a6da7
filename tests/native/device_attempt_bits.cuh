// Right-hand sides and attempts of rows of states, for the two translation units
// of the attempt test: the device code as the kernels use it, and the generic
// bodies (GRRT_RHS_GENERIC) that it stands for. Test-only.
#pragma once

struct AttemptRow {
    double M, a, pt, pph;
    double r, th, ph, pr, pth, h;
};
constexpr int kAttemptOut = 11;  // y5, k7 and the error norm

void launch_generic(int kind, const AttemptRow* rows, int n, double* out);
