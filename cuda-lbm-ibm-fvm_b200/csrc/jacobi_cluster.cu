// jacobi_cluster.cu -- all Jacobi sweeps of a small grid in one launch
// (solve_p_jacobi_kernel, voftrial1.cu:401-439, with the ping-pong of
// voftrial1.cu:1371-1375).
//
// Compiled with -fmad=false: each cell keeps the reference's operand order and
// the IEEE quotient (div_rn_pre), so the bits are those of separate sweeps.
//
// On a small grid a sweep of its own is all launch and latency (1.8 to 2.0 us).
// Here one thread-block cluster holds the pressure in its shared
// memories from the first sweep to the last: each block owns some z planes in
// two buffers (the ping-pong's), a thread a pair of cells with their right-hand
// sides and coefficients in registers.  After a sweep a block stores its first
// and last plane into its neighbours' halo planes (distributed shared memory)
// and the cluster meets at its barrier.  Each buffer starts with what the
// global one holds, ghost cells included, so that the products of ghosts are
// the same as well.
//
// What bounds it: per sweep the chain of loads, six subtractions and the
// quotient, the store to the neighbour and the barrier (0.7 us with a few warps
// a block), plus 0.4 us of instruction issue with 32 warps; a kernel's start
// and the first loads, once.  Measured on a B200: 32^3, 30 steps of 10 sweeps,
// 1.15 -> 1.03 ms; 24 x 20 x 16, six steps one call at a time, 482 -> 388 us.
#include "jacobi_cluster.h"

#include "pdl.cuh"

namespace vof {

#if defined(__CUDA_ARCH__) && !defined(VOF_FMAD_FALSE)
#error "jacobi_cluster.cu must be compiled with -fmad=false -DVOF_FMAD_FALSE"
#endif

namespace {

constexpr int JC_THREADS = 1024, JC_SMEM = 200 * 1024, JC_LOADS = 6;

__host__ __device__ __forceinline__ int jc_row(const Geom& g) { return (g.nx + 5) & ~1; }

__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// x / n for 0 <= x < 2^18 and rn = RN(1/n): x + 1/2 is at least 1/(2n) of the
// quotient away from an integer, the two roundings move it by x/n 2^-22.
__device__ __forceinline__ int quot(int x, float rn) { return (int)(((float)x + 0.5f) * rn); }

__device__ __forceinline__ void store_remote(unsigned local, unsigned rank, float2 v) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}

}  // namespace

// A pair of cells (2m + 1, 2m + 2 of a row) per thread; block r of the cluster
// owns planes 1 + r pl .. (r + 1) pl.  In shared memory column i of a row is at
// i + 1, so that a pair is an aligned 8-byte word; rows are of `row` values.
__global__ void __launch_bounds__(JC_THREADS, 1) k_jacobi_cluster(Geom g, const float* pin, const float* other,
                                                                  const float* rhs, float* out, int iters, int pl) {
    extern __shared__ __align__(16) float sm[];
    pdl_enter(pin, other, rhs, out);
    const int row = jc_row(g), slot = row * (g.ny + 2), size = (pl + 2) * slot;
    const int rank = blockIdx.x, ka = 1 + rank * pl, np = min(g.nz, ka + pl - 1) - ka + 1;  // own planes (or none)
    const int half = (g.nx + 1) / 2, pairs = np > 0 ? np * g.ny * half : 0;
    const float cx = g.dxi * g.dxi, cy = g.dyi * g.dyi, cz = g.dzi * g.dzi;
    const DivRange w = div_range(g);
    const int q = (int)threadIdx.x < pairs ? threadIdx.x : 0;
    const int jk = quot(q, 1.0f / half), i = 1 + 2 * (q - jk * half), kk = quot(jk, 1.0f / g.ny);
    const int j = 1 + jk - kk * g.ny, k = ka + kk;
    const int at = (kk + 1) * slot + j * row + i + 1, id = gidx(g, i, j, k);
    const bool own = (int)threadIdx.x < pairs, both = i < g.nx;
    const bool down = own && kk == 0 && rank > 0, up = own && kk == np - 1 && k < g.nz;  // planes a neighbour reads
    const float b0 = own ? rhs[id] : 0.0f, b1 = own && both ? rhs[id + 1] : 0.0f;
    const float aw = i != 1 ? cx : 0.0f, ae0 = both ? cx : 0.0f, ae1 = i + 1 < g.nx ? cx : 0.0f;
    const float an = j != g.ny ? cy : 0.0f, as = j != 1 ? cy : 0.0f;
    const float af = k != g.nz ? cz : 0.0f, ab = k != 1 ? cz : 0.0f;
    const float d0 = -(ae0 + aw + an + as + af + ab), d1 = -(ae1 + cx + an + as + af + ab);
    const float rd0 = __frcp_rn(d0), rd1 = __frcp_rn(d1);
    // the own planes and one on either side, from both buffers; loads of several strides in flight
    const int have = np > 0 ? (np + 2) * slot : 0;
    const float rrow = 1.0f / row, rrows = 1.0f / (g.ny + 2);
    for (int q0 = threadIdx.x; q0 < have; q0 += JC_LOADS * blockDim.x) {
        float x[JC_LOADS], y[JC_LOADS];
#pragma unroll
        for (int e = 0; e < JC_LOADS; ++e) {
            const int q = q0 + e * blockDim.x;
            const int jk = quot(q, rrow), k = quot(jk, rrows), i = q - jk * row - 1;
            const bool in = q < have && i >= 0 && i <= g.nx + 1;
            const int c = gidx(g, i, jk - k * (g.ny + 2), ka - 1 + k);
            x[e] = in ? pin[c] : 0.0f;
            y[e] = in ? other[c] : 0.0f;
        }
#pragma unroll
        for (int e = 0; e < JC_LOADS; ++e) {
            const int q = q0 + e * blockDim.x;
            if (q < have) {
                sm[q] = x[e];
                sm[size + q] = y[e];
            }
        }
    }
    cluster_meet();
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    for (int it = 0; it < iters; ++it) {
        const int from = it & 1 ? size : 0, to = it & 1 ? 0 : size;
        const bool last = it == iters - 1;
        if (own) {
            const float* p = sm + from + at;
            auto word = [](const float* a) { return *reinterpret_cast<const float2*>(a); };
            const float2 c = word(p), n = word(p + row), s = word(p - row), u = word(p + slot), l = word(p - slot);
            const float x0 = b0 - ae0 * c.y - aw * p[-1] - an * n.x - as * s.x - af * u.x - ab * l.x;
            const float x1 = b1 - ae1 * p[2] - cx * c.x - an * n.y - as * s.y - af * u.y - ab * l.y;
            const float q0 = __fmul_rn(x0, rd0), q1 = __fmul_rn(x1, rd1);
            float2 v = {__fmaf_rn(__fmaf_rn(-q0, d0, x0), rd0, q0), __fmaf_rn(__fmaf_rn(-q1, d1, x1), rd1, q1)};
            const unsigned least = min(2u * __float_as_uint(x0) - 1u, 2u * __float_as_uint(x1) - 1u);
            if (!(least >= w.lo2 && fmaxf(fabsf(x0), fabsf(x1)) <= w.hi)) {
                v.x = div_rn_pre(x0, d0, rd0);
                v.y = div_rn_pre(x1, d1, rd1);
            }
            if (last) {
                out[id] = v.x;
                if (both) out[id + 1] = v.y;
            } else {
                if (!both) v.y = sm[to + at + 1];  // the ghost of this buffer
                *reinterpret_cast<float2*>(sm + to + at) = v;
                // the plane above the neighbour's last, the plane below its first
                if (down) store_remote(base + 4u * (unsigned)(to + at + pl * slot), rank - 1, v);
                if (up) store_remote(base + 4u * (unsigned)(to + at - np * slot), rank + 1, v);
            }
        }
        if (!last) cluster_meet();
    }
}

static int jc_blocks = 0;  // blocks of a cluster, set by jacobi_cluster_configure (0: none)

static int planes_of(const Geom& g) { return (g.nz + jc_blocks - 1) / jc_blocks; }
static size_t bytes_of(const Geom& g) { return 2 * sizeof(float) * (planes_of(g) + 2) * (size_t)jc_row(g) * (g.ny + 2); }
static long long pairs_of(const Geom& g) { return (long long)planes_of(g) * g.ny * ((g.nx + 1) / 2); }

// Up to one pair per thread, and sweeps enough to pay for the cluster's start
// and the loads (per sweep and at 0 sweeps, us, against one launch per sweep:
// 24 x 20 x 16 0.7 + 22 against 1.7 + 19, 32^3 1.1 + 24 against 1.8 + 20; with
// two pairs per thread 36^3 1.5 + 27 against 1.8 + 22).
bool jacobi_cluster_fits(const Geom& g, int iters) {
    return jc_blocks > 0 && pairs_of(g) <= JC_THREADS && bytes_of(g) <= JC_SMEM && iters >= (pairs_of(g) > 512 ? 7 : 3);
}

static void attributes(cudaLaunchAttribute* at, int blocks) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
}

cudaError_t jacobi_cluster_launch(const Geom& g, float* const p[2], int src, const float* rhs, int iters,
                                  cudaStream_t s) {
    cudaLaunchAttribute at[2];
    attributes(at, jc_blocks);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = jc_blocks;
    cfg.blockDim = ((int)pairs_of(g) + 31) / 32 * 32;
    cfg.dynamicSmemBytes = bytes_of(g);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    float* out = p[src ^ (iters & 1)];
    return cudaLaunchKernelEx(&cfg, k_jacobi_cluster, g, (const float*)p[src], (const float*)p[src ^ 1], rhs, out, iters,
                              planes_of(g));
}

cudaError_t jacobi_cluster_configure() {
    cudaError_t e = cudaFuncSetAttribute(k_jacobi_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, JC_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_jacobi_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    for (int n = 16; n >= 8; n >>= 1) {  // (a partition of the device may not hold 16)
        cudaLaunchAttribute at[2];
        attributes(at, n);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = n;
        cfg.blockDim = JC_THREADS;
        cfg.dynamicSmemBytes = JC_SMEM;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if ((e = cudaOccupancyMaxActiveClusters(&clusters, k_jacobi_cluster, &cfg)) != cudaSuccess) return e;
        if (clusters > 0) {
            jc_blocks = n;
            break;
        }
    }
    return cudaSuccess;
}

}  // namespace vof
