// spectral.cu -- direct solve of the Neumann pressure system: the inner solve
// of the convergent modes (an extension; the reference runs 10 Jacobi sweeps,
// voftrial1.cu:1371-1375).
//
// The operator (Sigma over the non-wall neighbours of (p_nb - p)/h^2 on a
// uniform box) is diagonal in the cosine basis cos(pi a (i + 1/2) / n) along
// x and y (the DCT-II; G. Strang, "The discrete cosine transform", SIAM
// Review 41(1), 1999), with eigenvalues -4/h^2 sin^2(pi a / (2n)).  Forward
// transforms along x and y leave one tridiagonal system along z per column;
// after solving those the transforms back give the solution, to rounding.
//
// Transforms (k_dct).  A transform of length n is a product with a dense
// n x n matrix.  The basis functions are even or odd about the middle, so
// folding a line (x_i + x_{n-1-i}, x_i - x_{n-1-i}) makes it two products of
// half the size, n/2 FP64 multiply-adds per value, at any n.  They run on the
// FP64 tensor cores (mma.sync m16n8k8).  A block owns TN neighbouring lines
// over their full length: the lines are copied to shared memory
// asynchronously (all of them in flight at once: by registers, 8 loads a
// thread, a 200^3 pass took 15 us longer), folded there, each warp forms 16
// rows of both parts for all TN lines, and the results go back in place.  At
// 200^3 a pass takes 85 to 105 us with the tensor pipe 62 to 68 % busy (its
// floor is 51 us: 1.86 GFLOP with the padding of 100 rows to 112 x 104); the
// rest is the blocks' load and store phases, which three blocks an SM overlap
// in part.  The matrices come in fragment order straight from L2 (coalesced,
// one step ahead).  The last transform (along x) adds into the pressure.
//
// Columns (k_zcr).  With the column's equation scaled to
//   e_k - alpha (e_{k-1} + e_{k+1}) = q_k,   0 < alpha < 1/2 (in FP64 too: sp_takes),
// and the zero-gradient ends mirrored (an even sequence of period 2 nz), one
// step of cyclic reduction (R. W. Hockney, J. ACM 12(1), 1965) applied to
// every row keeps that form with stride 2 s,
//   q_k += alpha (q_{k-s} + q_{k+s}),  alpha' = alpha^2 / (1 - 2 alpha^2),
// up to the factor 1 / (1 - 2 alpha^2), which is collected and applied at
// the end.  alpha falls quadratically: the loop ends when it is below 2^-60
// in every column of the block, after some 5 steps for most columns and 13
// for the slowest at nz = 200 (SP_ZCR_STEPS at most).  All terms of a step have the sign of their
// q's weights (no cancellation).  At 200^3 it takes 76 us; two more dense
// transforms and the division took 225.  The constant column's system is singular:
// one warp sums it twice and removes the mean.
#include "spectral.h"

#include <math.h>

#include "pdl.cuh"

namespace vof {

namespace {

struct SpArgs {
    int nx, ny, nz, lines;
    SpAxis ax;
    double* p;  // pressure of the last pass (padded layout)
    int px, plane;
    SpStop stop;
};

__device__ __forceinline__ bool reached(const SpStop& s) {
    return s.norms && (s.norms[1] > 0.0 ? sqrt(s.norms[0] / s.norms[1]) : 0.0) <= s.tol;
}

__device__ __forceinline__ void copy8(double* dst, const double* src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = in ? 8 : 0;  // (0: the word is zeroed, src is not read)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], double b0, double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}

__device__ __forceinline__ void load_a(const double* __restrict__ f, int step, int lane, double (&a)[4]) {
    const double2* q = reinterpret_cast<const double2*>(f + ((size_t)step * 32 + lane) * 4);
    const double2 u = __ldg(q), v = __ldg(q + 1);
    a[0] = u.x;
    a[1] = u.y;
    a[2] = v.x;
    a[3] = v.y;
}

// c = M x of row tile m of one part; X: [kt * 8][P] in shared memory.
template <int NT, int P>
__device__ __forceinline__ void gemm(const double* __restrict__ f, int m, int kt, const double* X,
                                     double (&c)[NT][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[q][e] = 0.0;
    double a[4];
    load_a(f, m * kt, lane, a);
    const double* x = X + t * P + g;
    for (int k = 0; k < kt; ++k) {
        double n[4];
        load_a(f, m * kt + (k + 1 < kt ? k + 1 : k), lane, n);
#pragma unroll
        for (int q = 0; q < NT; ++q) dmma(c[q], a, x[q * 8], x[4 * P + q * 8]);
        x += 8 * P;
#pragma unroll
        for (int q = 0; q < 4; ++q) a[q] = n[q];
    }
}

// AXIS 0 (x) or 1 (y); BACK: the transform back (along x: added into p).
template <int AXIS, bool BACK, int TN, bool WIDE>
__global__ void __launch_bounds__(WIDE ? 512 : 256, WIDE ? 1 : 3) k_dct(SpArgs A, double* w) {
    pdl_enter();
    if (reached(A.stop)) return;
    constexpr int NT = TN / 8, P = TN + 4;  // P = 4 (mod 16): a B fragment's words are on distinct banks
    extern __shared__ __align__(16) double X[];
    const int n = A.ax.n, h0 = A.ax.h0, h1 = A.ax.h1, kt = A.ax.kt, kp = kt * 8;
    const int nw = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int c0 = blockIdx.x * TN;
    const int st = AXIS == 0 ? 1 : A.nx;
    auto base = [&](int c) { return AXIS == 0 ? c * A.nx : (c / A.nx) * A.nx * A.ny + c % A.nx; };
    double* X1 = X + kp * P;
    // row r of part 0 and of part 1: positions r and n-1-r (to be folded), or the modes 2r and 2r + 1
    auto second = [&](int r) { return BACK ? h0 + r : n - 1 - r; };
    if (AXIS == 0) {  // 8 lines x 4 positions per warp: 32-byte pieces of each line, distinct banks
        const int groups = TN / 8, chunks = kp / 4;
        for (int q = warp; q < groups * chunks; q += nw) {
            const int l = (q % groups) * 8 + g, r = (q / groups) * 4 + t;
            const double* x = w + base(min(c0 + l, A.lines - 1));
            const bool in = c0 + l < A.lines;
            copy8(X + r * P + l, x + min(r, h0 - 1), in && r < h0);
            copy8(X1 + r * P + l, x + (r < h1 ? second(r) : 0), in && r < h1);
        }
    } else {
        const int l = lane % TN;
        const bool in = c0 + l < A.lines;
        const double* x = w + base(min(c0 + l, A.lines - 1));
        for (int r = warp * (32 / TN) + lane / TN; r < kp; r += nw * (32 / TN)) {
            copy8(X + r * P + l, x + (size_t)min(r, h0 - 1) * st, in && r < h0);
            copy8(X1 + r * P + l, x + (size_t)(r < h1 ? second(r) : 0) * st, in && r < h1);
        }
    }
    copy_wait();
    __syncthreads();
    if (!BACK) {
        for (int q = threadIdx.x; q < h1 * TN; q += blockDim.x) {
            const int at = (q / TN) * P + q % TN;
            const double lo = X[at], hi = X1[at];
            X[at] = lo + hi;
            X1[at] = lo - hi;
        }
        __syncthreads();
    }
    const double* const* F = BACK ? A.ax.inv : A.ax.fwd;
    for (int m = warp; m < A.ax.mt; m += nw) {
        const int r0 = m * 16 + g;
        if (!BACK) {
#pragma unroll 1
            for (int part = 0; part < 2; ++part) {
                double c[NT][4];
                gemm<NT, P>(F[part], m, kt, part ? X1 : X, c);
#pragma unroll
                for (int q = 0; q < NT; ++q)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int col = c0 + q * 8 + 2 * t + (e & 1), r = r0 + (e & 2) * 4;
                        if (col < A.lines && r < (part ? h1 : h0))
                            w[base(col) + (size_t)(part ? h0 + r : r) * st] = c[q][e];
                    }
            }
            continue;
        }
        // (half of the columns at a time: the accumulators of both parts are live together)
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            constexpr int NH = NT / 2;
            const int h = half * NH * 8;
            double c[2][NH][4];
            gemm<NH, P>(F[0], m, kt, X + h, c[0]);
            gemm<NH, P>(F[1], m, kt, X1 + h, c[1]);
            double* x[NH][2];
            double old[NH][2][4];
#pragma unroll
            for (int q = 0; q < NH; ++q)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = min(c0 + h + q * 8 + 2 * t + e, A.lines - 1);
                    if (AXIS == 0)
                        x[q][e] = A.p + ((size_t)(col / A.ny + 1) * A.plane + (size_t)(col % A.ny + 1) * A.px + 1);
                    else
                        x[q][e] = w + base(col);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {  // along x: the pressure's old values, all in flight together
                        const int r = min(r0 + u * 8, h0 - 1);
                        old[q][0][2 * u + e] = AXIS == 0 ? x[q][e][r] : 0.0;
                        old[q][1][2 * u + e] = AXIS == 0 ? x[q][e][n - 1 - r] : 0.0;
                    }
                }
#pragma unroll
            for (int q = 0; q < NH; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int col = c0 + h + q * 8 + 2 * t + (e & 1), r = r0 + (e & 2) * 4;
                    if (col >= A.lines || r >= h0) continue;
                    double* y = x[q][e & 1];
                    y[(size_t)r * st] = old[q][0][e] + (c[0][q][e] + c[1][q][e]);
                    if (2 * r != n - 1) y[(size_t)(n - 1 - r) * st] = old[q][1][e] + (c[0][q][e] - c[1][q][e]);
                }
        }
    }
}

// The systems along z of TN columns (two buffers of nz x TN in shared memory).
constexpr int ZCR_THREADS = 512;

template <int TN>
__global__ void __launch_bounds__(ZCR_THREADS, 2) k_zcr(int nx, int ny, int nz, double az, const double* lx,
                                             const double* ly, double* w, SpStop stop) {
    pdl_enter();
    if (reached(stop)) return;
    extern __shared__ __align__(16) double Z[];
    constexpr int ROWS = ZCR_THREADS / TN;
    const int lines = nx * ny, c0 = blockIdx.x * TN, l = threadIdx.x % TN, row = threadIdx.x / TN;
    const int col = min(c0 + l, lines - 1);
    const bool in = c0 + l < lines;
    double* cur = Z;
    double* nxt = Z + nz * TN;
    for (int k = row; k < nz; k += ROWS) copy8(cur + k * TN + l, w + (size_t)k * lines + col, in);
    const double sg = lx[col % nx] + ly[col / nx];
    const bool constant = col == 0;  // the mode of the (x, y) mean: eigenvalue 0
    const double d = 2.0 * az + sg;
    double al = constant ? 0.0 : az / d, f = constant ? 1.0 : -1.0 / d;
    copy_wait();
    __syncthreads();
    if (c0 == 0) {
        // singular column: az (e_{k+1} - 2 e_k + e_{k-1}) = q_k - mean, summed
        // twice by one warp, each lane over its own piece of the column
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x, len = (nz + 31) / 32, k0 = min(nz, lane * len), k1 = min(nz, k0 + len);
            double sum = 0.0;
            for (int k = k0; k < k1; ++k) sum += cur[k * TN];
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const double mean = sum / nz, raz = 1.0 / az;
            // twice: q -> flux (inclusive sums), flux -> e (exclusive sums)
            for (int pass = 0; pass < 2; ++pass) {
                double own = 0.0;
                for (int k = k0; k < k1; ++k) own += pass ? cur[k * TN] : (cur[k * TN] - mean) * raz;
                double run = own;
                for (int o = 1; o < 32; o <<= 1) {
                    const double up = __shfl_up_sync(0xffffffffu, run, o);
                    if (lane >= o) run += up;
                }
                run -= own;
                for (int k = k0; k < k1; ++k) {
                    const double v = pass ? cur[k * TN] : (cur[k * TN] - mean) * raz;
                    cur[k * TN] = pass ? run : run + v;
                    run += v;
                }
            }
            sum = 0.0;
            for (int k = k0; k < k1; ++k) sum += cur[k * TN];
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            sum /= nz;
            for (int k = k0; k < k1; ++k) cur[k * TN] -= sum;
        }
        __syncthreads();
    }
    int s = 1;  // stride modulo the period 2 nz
    for (int step = 0; step < SP_ZCR_STEPS && __syncthreads_or(al > 0x1p-60); ++step) {
#pragma unroll 4
        for (int k = row; k < nz; k += ROWS) {
            int a = k - s, b = k + s;  // mirrored into 0 .. nz-1: the sequence is even about -1/2 with period 2 nz
            if (a < 0) a = -1 - a;
            if (a >= nz) a = 2 * nz - 1 - a;
            if (b >= 2 * nz) b -= 2 * nz;
            if (b >= nz) b = 2 * nz - 1 - b;
            nxt[k * TN + l] = fma(al, cur[a * TN + l] + cur[b * TN + l], cur[k * TN + l]);
        }
        const double m = 1.0 - 2.0 * al * al;
        f /= m;
        al = al * al / m;
        s = 2 * s % (2 * nz);
        double* x = cur;
        cur = nxt;
        nxt = x;
    }
    if (in)
        for (int k = row; k < nz; k += ROWS) w[(size_t)k * lines + col] = f * cur[k * TN + l];
}

template <int TN>
size_t dct_smem(const SpAxis& a) {
    return sizeof(double) * 2 * (size_t)(a.kt * 8) * (TN + 4);
}

template <int AXIS, bool BACK, int TN, bool WIDE>
cudaError_t launch_dct(const SpArgs& A, double* w, cudaStream_t s) {
    auto* k = k_dct<AXIS, BACK, TN, WIDE>;
    const size_t smem = dct_smem<TN>(A.ax);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int most = WIDE ? 16 : 8, warps = A.ax.mt < most ? A.ax.mt : most;
    return pdl_launch(k, dim3((A.lines + TN - 1) / TN), dim3(warps * 32), smem, s, A, w);
}

template <int AXIS, bool BACK>
cudaError_t dct(const Geom& g, const SpSolver& m, double* w, double* p, const SpStop& stop, cudaStream_t s) {
    SpArgs A;
    A.nx = g.nx;
    A.ny = g.ny;
    A.nz = g.nz;
    A.ax = m.ax[AXIS];
    A.lines = AXIS == 0 ? g.ny * g.nz : g.nx * g.nz;
    A.p = p;
    A.px = g.px;
    A.plane = g.plane;
    A.stop = stop;
    if (A.ax.mt <= 8) return launch_dct<AXIS, BACK, 32, false>(A, w, s);
    return dct_smem<32>(A.ax) <= 200 * 1024 ? launch_dct<AXIS, BACK, 32, true>(A, w, s)
                                            : launch_dct<AXIS, BACK, 16, true>(A, w, s);
}

template <int TN>
cudaError_t launch_zcr(const Geom& g, const SpSolver& m, double* w, const SpStop& stop, cudaStream_t s) {
    const size_t smem = sizeof(double) * 2 * (size_t)g.nz * TN;
    cudaError_t e = cudaFuncSetAttribute(k_zcr<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return pdl_launch(k_zcr<TN>, dim3((g.nx * g.ny + TN - 1) / TN), dim3(ZCR_THREADS), smem, s, g.nx, g.ny, g.nz, m.az,
                      m.ax[0].lam, m.ax[1].lam, w, stop);
}

}  // namespace

cudaError_t sp_correct(const Geom& g, const SpSolver& m, double* r, double* p64, const SpStop& stop, cudaStream_t s,
                       int& launches) {
    cudaError_t e;
    launches += 5;
    if ((e = dct<0, false>(g, m, r, p64, stop, s)) != cudaSuccess) return e;
    if ((e = dct<1, false>(g, m, r, p64, stop, s)) != cudaSuccess) return e;
    // (two buffers of nz x columns in shared memory, two blocks per SM)
    e = g.nz <= 208 ? launch_zcr<32>(g, m, r, stop, s) : g.nz <= 416 ? launch_zcr<16>(g, m, r, stop, s) : launch_zcr<8>(g, m, r, stop, s);
    if (e != cudaSuccess) return e;
    if ((e = dct<1, true>(g, m, r, p64, stop, s)) != cudaSuccess) return e;
    return dct<0, true>(g, m, r, p64, stop, s);
}

void sp_destroy(SpSolver* m) {
    for (int q = 0; q < 2; ++q)
        for (int t = 0; t < 5; ++t)
            if (m->mem[q][t]) cudaFree(m->mem[q][t]);
    *m = SpSolver{};
}

size_t sp_table_doubles(int n) {
    const size_t h0 = (n + 1) / 2;
    return ((h0 + 15) / 16) * ((h0 + 7) / 8) * 128;
}

void sp_tables(int n, double inv_h2, double* tables, double* lam, double* cosine) {
    const int h[2] = {(n + 1) / 2, n / 2};
    const int mt = (h[0] + 15) / 16, kt = (h[0] + 7) / 8;
    const long double pi = 3.14159265358979323846264338327950288L;
    // c_a(i): the argument reduced exactly, a (2i + 1) modulo 4n in units of pi / (2n)
    for (int q = 0; q < 4 * n; ++q) cosine[q] = (double)(sqrtl(2.0L / n) * cosl(pi * q / (2.0L * n)));
    const double first = (double)sqrtl(1.0L / n);
    auto basis = [&](int a, int i) { return a == 0 ? first : cosine[((long long)a * (2 * i + 1)) % (4LL * n)]; };
    const size_t nt = sp_table_doubles(n);
    for (int part = 0; part < 2; ++part)
        for (int m = 0; m < mt; ++m)
            for (int k = 0; k < kt; ++k)
                for (int lane = 0; lane < 32; ++lane)
                    for (int e = 0; e < 4; ++e) {
                        // element e of lane: row m*16 + lane/4 (+8 for odd e), column k*8 + lane%4 (+4 for e >= 2)
                        const int row = m * 16 + lane / 4 + (e & 1) * 8, col = k * 8 + lane % 4 + (e >> 1) * 4;
                        const size_t at = ((size_t)(m * kt + k) * 32 + lane) * 4 + e;
                        const bool in = row < h[part] && col < h[part];
                        // forward: mode 2 row + part from position col; back: position row from mode 2 col + part
                        tables[part * nt + at] = in ? basis(2 * row + part, col) : 0.0;
                        tables[(2 + part) * nt + at] = in ? basis(2 * col + part, row) : 0.0;
                    }
    for (int q = 0; q < n; ++q) {  // even modes first, as the spectrum is stored
        const int a = q < h[0] ? 2 * q : 2 * (q - h[0]) + 1;
        const long double sn = sinl(pi * a / (2.0L * n));
        lam[q] = (double)(4.0L * inv_h2 * sn * sn);
    }
}

}  // namespace vof
