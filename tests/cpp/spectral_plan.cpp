// The rule of csrc/spectral_plan.h and the recurrence of k_zcr, compiled for the host (tests/test_spectral_plan.py).
#include "spectral_plan.h"

extern "C" int takes(int nx, int ny, float dxi, float dyi, float dzi) { return vof::sp_takes(nx, ny, dxi, dyi, dzi); }
extern "C" int most_steps(void) { return vof::SP_ZCR_STEPS; }
extern "C" double least_ratio(void) { return vof::SP_LEAST_RATIO; }

// Steps until alpha is at most 2^-60, from the column of eigenvalue sg; `limit` if it takes more.
extern "C" int steps(double az, double sg, int contracted, int limit) {
    double al = az / (2.0 * az + sg);
    int n = 0;
    for (; n < limit && al > 0x1p-60; ++n) {
        const double m = contracted ? fma(-2.0 * al, al, 1.0) : 1.0 - 2.0 * al * al;
        al = al * al / m;
    }
    return n;
}
