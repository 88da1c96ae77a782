// spectral.h -- direct solve of the Neumann pressure system by cosine
// transforms along x and y and cyclic reduction along z (spectral.cu), the
// inner solve of the convergent modes.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <new>

#include "spectral_plan.h"
#include "vof_device.cuh"

namespace vof {

// One transformed axis of n cells.  The cosine basis c_a(i) = s_a cos(pi a
// (i + 1/2) / n) is even (a even) or odd (a odd) about the middle, so a
// transform of length n is two products of half the size: h0 = ceil(n/2) rows
// for the even modes (part 0) and h1 = floor(n/2) for the odd ones (part 1);
// the spectrum is stored even modes first.  fwd / inv hold the two matrices of
// each direction in the order the tensor-core fragments read them: mt row
// tiles of 16, kt steps of 8.
struct SpAxis {
    int n, h0, h1, mt, kt;
    const double* fwd[2];
    const double* inv[2];
    const double* lam;  // eigenvalues of the second difference, 4/h^2 sin^2(pi a / (2n)) (sign changed)
};

struct SpSolver {
    SpAxis ax[2];
    double az;        // 1/h^2 along z
    void* mem[2][5];  // the device arrays of each axis (fwd 0/1, inv 0/1, lam)
};

// Host tables of one axis: the four fragment-ordered matrices (forward parts
// 0 and 1, back parts 0 and 1; sp_table_doubles(n) values each) and the n
// eigenvalues.  cosine: room for 4n values.
size_t sp_table_doubles(int n);
void sp_tables(int n, double inv_h2, double* tables, double* lam, double* cosine);

void sp_destroy(SpSolver* m);

// The kernels do nothing when sqrt(norms[0] / norms[1]) <= tol on the device
// as they start (norms null: they always run).
struct SpStop {
    const double* norms;
    double tol;
};

// p64 (padded layout) += the mean-free solution e of A e = r - mean(r).  r:
// compact array (i fastest, no ghosts), overwritten.  launches += kernels enqueued.
cudaError_t sp_correct(const Geom& g, const SpSolver& m, double* r, double* p64, const SpStop& stop, cudaStream_t s,
                       int& launches);

// Build the tables for grid g.  alloc(void**, bytes): the caller's device allocator.
template <typename Alloc>
cudaError_t sp_create(const Geom& g, SpSolver* m, cudaStream_t s, Alloc&& alloc) {
    const int n[2] = {g.nx, g.ny};
    const double a[2] = {(double)g.dxi * g.dxi, (double)g.dyi * g.dyi};
    m->az = (double)g.dzi * g.dzi;
    for (int q = 0; q < 2; ++q) {
        SpAxis& x = m->ax[q];
        x.n = n[q];
        x.h0 = (n[q] + 1) / 2;
        x.h1 = n[q] / 2;
        x.mt = (x.h0 + 15) / 16;
        x.kt = (x.h0 + 7) / 8;
        const size_t nt = sp_table_doubles(n[q]);
        double* h = new (std::nothrow) double[4 * nt + 5 * (size_t)n[q]];
        if (!h) return cudaErrorMemoryAllocation;
        sp_tables(n[q], a[q], h, h + 4 * nt, h + 4 * nt + n[q]);
        for (int t = 0; t < 5; ++t) {
            const size_t nb = sizeof(double) * (t < 4 ? nt : (size_t)n[q]);
            cudaError_t e = alloc(&m->mem[q][t], nb);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // (alloc clears the array on s)
            if (e == cudaSuccess) e = cudaMemcpy(m->mem[q][t], h + t * nt, nb, cudaMemcpyHostToDevice);
            if (e != cudaSuccess) {
                delete[] h;
                return e;
            }
        }
        delete[] h;
        x.fwd[0] = static_cast<const double*>(m->mem[q][0]);
        x.fwd[1] = static_cast<const double*>(m->mem[q][1]);
        x.inv[0] = static_cast<const double*>(m->mem[q][2]);
        x.inv[1] = static_cast<const double*>(m->mem[q][3]);
        x.lam = static_cast<const double*>(m->mem[q][4]);
    }
    return cudaSuccess;
}

}  // namespace vof
