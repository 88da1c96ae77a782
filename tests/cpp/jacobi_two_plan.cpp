// The tiling of csrc/jacobi_two_plan.h, compiled for the host (tests/test_jacobi_two_plan.py).
#include "jacobi_two_plan.h"

// Of every grid of sides from[q], from[q] + step[q] .. to[q]: how many tilings
// break a limit of the launch; the first such grid in bad[0 .. 2].
extern "C" int check_plans(const int* from, const int* to, const int* step, int* bad) {
    int broken = 0;
    for (int nx = from[0]; nx <= to[0]; nx += step[0])
        for (int ny = from[1]; ny <= to[1]; ny += step[1])
            for (int nz = from[2]; nz <= to[2]; nz += step[2]) {
                const vof::J2Plan p = vof::j2_plan(nx, ny, nz);
                const int quads = (nx + 1) / 4 + 1;
                const bool fine = 4 * p.nq <= 256 && p.rows + 2 <= 256 && p.rows >= 3 && p.nq >= 1 + 2 * p.hq &&
                                  p.nq * p.rows <= p.threads && p.threads <= vof::J2_THREADS && p.threads % 32 == 0 &&
                                  p.smem == vof::j2_smem(p.nq, p.rows) && p.smem <= vof::J2_SMEM &&
                                  p.tx * p.wq >= quads && (p.tx == 1 || p.hq == 1) && p.wq == p.nq - 2 * p.hq &&
                                  p.ty * (p.rows - 2) >= ny && p.ty <= 65535 && p.kc >= 1 &&
                                  (nz + p.kc - 1) / p.kc <= 65535;
                if (!fine && broken++ == 0) {
                    bad[0] = nx;
                    bad[1] = ny;
                    bad[2] = nz;
                }
            }
    return broken;
}

extern "C" int chosen(int nx, int ny, int nz, int iters, int forced) {
    return vof::j2_chosen(nx, ny, nz, iters, forced);
}
