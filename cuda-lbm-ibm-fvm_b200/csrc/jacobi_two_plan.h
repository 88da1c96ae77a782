// jacobi_two_plan.h -- the tiling of a two-sweep Jacobi launch (jacobi_two.cu), in plain C++.
#pragma once
#include <math.h>
#include <stdint.h>

namespace vof {

constexpr int J2_THREADS = 512, J2_STAGES = 4, J2_SMEM = 220 * 1024;
constexpr int J2_BOX = 256;  // most elements a side of a TMA box may have

// Whether `iters` sweeps of a grid run two per launch where nothing else takes
// them (forced: 1 one per launch, 2 two, 0 by size).  From 2^19 cells: below,
// the march of two sweeps is too short to pay for its halo (64^3: 30 steps 4.56
// against 4.45 ms, 32^3 1.65 against 1.59; from 128^3 up two are faster).  A
// launch cannot end in the buffer it reads, where two sweeps have to end.
inline bool j2_chosen(int nx, int ny, int nz, int iters, int forced) {
    if (iters <= 2 || forced == 1) return false;
    return forced == 2 || (long long)nx * ny * nz >= 1 << 19;
}

// Tiling of one launch: blocks of nq x rows quads (four cells of a row) march
// kc planes; the outermost hq quads (where tiles neighbour along x) and the
// first and last row are halo.
struct J2Plan {
    int nq, rows, hq, wq;  // quads per row of the tile, rows, halo quads a side, quads a tile writes
    int tx, ty, kc;        // tiles along x and y, planes per block
    int threads, smem;
};

inline int j2_smem(int nq, int rows) {
    const int plane = (((rows + 2) * 4 * nq * 4 + 127) & ~127);
    return (2 * J2_STAGES + 2) * plane + J2_STAGES * (int)sizeof(uint64_t);
}

// The tiling with the least estimated time in units of microseconds: waves of
// one block per SM, times the planes a block marches (its own, two of the halo
// and about 1.5 to start), times a plane's cost (its warps' issue slots, not
// below its latency).  At 200^3, one column of 29 x 5 tiles of 51 quads x 9
// rows (7 of them written) and 40 planes.  A plane is loaded as one TMA box of
// 4 nq x (rows + 2) elements, which bounds both: rows of one quad (nx of 1 or
// 2) would otherwise take up to 512 rows.
inline J2Plan j2_plan(int nx, int ny, int nz) {
    const int all = (nx + 1) / 4 + 1;  // quads covering columns 0 .. nx + 1
    J2Plan best = {};
    double least = 1e30;
    for (int tx = 1; tx <= all; ++tx) {
        J2Plan p = {};
        p.tx = tx;
        p.wq = (all + tx - 1) / tx;
        p.hq = tx > 1 ? 1 : 0;
        p.nq = p.wq + 2 * p.hq;
        if ((tx - 1) * p.wq >= all) continue;  // an empty tile
        if (4 * p.nq > J2_BOX) continue;
        if (p.nq < 10 && tx > 1) break;
        for (p.rows = ny < 12 ? 3 : 8; p.rows <= ny + 2 && p.rows * p.nq <= J2_THREADS && p.rows + 2 <= J2_BOX;
             ++p.rows) {
            p.smem = j2_smem(p.nq, p.rows);
            if (p.smem > J2_SMEM) break;
            p.ty = (ny + p.rows - 3) / (p.rows - 2);
            p.threads = (p.nq * p.rows + 31) / 32 * 32;
            const double plane = fmax(0.45, 0.15 + 0.04 * (p.threads / 32));
            const int tiles = p.tx * p.ty;
            for (int waves = (tiles + 147) / 148, last = waves + 12; waves <= last; ++waves) {
                int nch = waves * 148 / tiles;
                if (nch > nz) nch = nz;
                p.kc = (nz + nch - 1) / nch;
                const int blocks = tiles * ((nz + p.kc - 1) / p.kc);
                const double cost = (double)((blocks + 147) / 148) * (p.kc + 3.5) * plane;
                if (cost < least) {
                    least = cost;
                    best = p;
                }
                if (p.kc <= 8 || nch == nz) break;
            }
        }
    }
    return best;
}

}  // namespace vof
