// spectral_plan.h -- which systems the direct solve takes (spectral.cu), in plain C++.
#pragma once
#include <math.h>

namespace vof {

// Most steps k_zcr takes.  A column whose alpha is still above 2^-60 then has
// alpha = 1/2 in FP64, where the recurrence stays for ever.
constexpr int SP_ZCR_STEPS = 48;

// Least eigenvalue of a column along x and y, over 1/h^2 along z, that the
// direct solve takes: alpha = 1 / (2 + ratio) keeps 13 bits of the ratio, and
// its 25 or so steps are far from the limit above.  A cube of 905 cells a side
// has 1.2e-5, and flat boxes pass down to planes some thousand times closer
// than the cells of a row.
constexpr double SP_LEAST_RATIO = 0x1p-40;

// Whether that holds for a grid (dxi, dyi, dzi: cells per unit length).
inline bool sp_takes(int nx, int ny, float dxi, float dyi, float dzi) {
    const double az = (double)dzi * dzi;
    if (!(az > 0.0 && isfinite(az))) return false;
    const int n[2] = {nx, ny};
    const double inv_h2[2] = {(double)dxi * dxi, (double)dyi * dyi};
    for (int q = 0; q < 2; ++q) {
        if (n[q] == 1) continue;  // (no column but the constant one)
        const double sn = sin(3.14159265358979323846 / (2.0 * n[q])), least = 4.0 * inv_h2[q] * sn * sn;
        if (!(least >= SP_LEAST_RATIO * az && isfinite(4.0 * inv_h2[q]))) return false;
    }
    return true;
}

}  // namespace vof
