// jacobi.cu -- one Jacobi sweep of the pressure system per launch
// (solve_p_jacobi_kernel, voftrial1.cu:401-439): the odd sweep of an odd
// count, and counts up to two (jacobi_two.cu takes the others two at a time).
//
// Compiled with -fmad=false: each cell update keeps the reference's
//     pt = (rhs - ae*pE - aw*pW - an*pN - as*pS - af*pF - ab*pB) / ap
// with the same operand order.  The division uses div_rn_pre with the IEEE
// reciprocal of ap (a handful of values per launch), which equals the IEEE
// quotient.
#include <cuda_runtime.h>
#include <stdlib.h>

#include "jacobi.h"

#include "pdl.cuh"

namespace vof {

#if defined(__CUDA_ARCH__) && !defined(VOF_FMAD_FALSE)
#error "jacobi.cu must be compiled with -fmad=false -DVOF_FMAD_FALSE"
#endif

constexpr int JP_THREADS = 256;

// ---- one sweep, two cells per thread, streaming along z ---------------------
// Cells are paired by padded column (2m, 2m + 1): pair m of a row is one
// aligned 8-byte word (px is a multiple of 32).  The pairs of rows 1..ny are
// numbered flat, q = (j - 1) npair + m, and 32 consecutive pairs make a warp
// across row ends, so every lane has work at every width.  A thread marches
// kchunk planes with its pair's p(k - 1), p(k), p(k + 1) in registers; the y
// neighbours are loads (served by L1), the x neighbours come from the
// neighbouring lanes, or from memory at the ends of a warp and of a row; the
// next plane's operands are loaded a plane ahead; no shared memory, no
// barrier.  (The packed f32x2 instructions are not used here: in a
// chain of them the code generator fuses a product into the following
// subtraction, which changes the rounding; a probe on a B200 found a quarter
// of such two-term chains off by an ulp even with .rn on every instruction.)
// The ghost cell of a pair (column 0 or nx + 1) is never stored.
//
// The march is split: the first plane of the box (k = 1) and the last plane
// of the chunk run through the general plane step; the planes between load
// their successors unconditionally and take the inner diagonal, in a loop
// unrolled U times so that the plane registers are renamed instead of copied.
struct JPLine {
    const float2* P;
    const float2* R;
    float2* O;
    const float* pin;
    float* pout;
    int w, wp, wr, cw, ce, plane;
    float ae0, aw0, ae1, aw1, an, as, cz;
    float2 dm, rm;
    bool a0, a1, ldw, lde;
};

struct JPRegs {
    float2 pm, pc, pp, pS, pN, rc;
    float xw, xe;
};

// One plane k of the paired sweep.  MORE: load the next plane's operands (the
// caller guarantees k < k1 <= nz, so plane k + 2 <= nz + 1 exists).  EDGE: the
// plane may be the first or the last of the box.
template <bool MORE, bool EDGE>
__device__ __forceinline__ void jp_plane(const JPLine& L, const Geom& g, int k, JPRegs& s) {
    float2 pq, sn, nn, rn;
    float xwn = 0.0f, xen = 0.0f;
    if constexpr (MORE) {
        const int kn = k + 1, o1 = L.w + kn * L.wp;
        pq = L.P[o1 + L.wp];
        sn = L.P[o1 - L.wr];
        nn = L.P[o1 + L.wr];
        rn = L.R[o1];
        if (L.ldw) xwn = L.pin[L.cw + kn * L.plane];
        if (L.lde) xen = L.pin[L.ce + kn * L.plane];
    }
    float pw = __shfl_up_sync(0xffffffffu, s.pc.y, 1), pe = __shfl_down_sync(0xffffffffu, s.pc.x, 1);
    if (L.ldw) pw = s.xw;
    if (L.lde) pe = s.xe;
    float af = L.cz, ab = L.cz;
    float2 d = L.dm, rd = L.rm;
    if constexpr (EDGE) {
        const bool kb = k == 1, kt = k == g.nz;
        af = kt ? 0.0f : L.cz;
        ab = kb ? 0.0f : L.cz;
        if (kb || kt) {
            d = make_float2(-(L.ae0 + L.aw0 + L.an + L.as + af + ab), -(L.ae1 + L.aw1 + L.an + L.as + af + ab));
            rd = make_float2(__frcp_rn(d.x), __frcp_rn(d.y));
        }
    }
    const float v0 = div_rn_pre(s.rc.x - L.ae0 * s.pc.y - L.aw0 * pw - L.an * s.pN.x - L.as * s.pS.x -
                                    af * s.pp.x - ab * s.pm.x,
                                d.x, rd.x);
    const float v1 = div_rn_pre(s.rc.y - L.ae1 * pe - L.aw1 * s.pc.x - L.an * s.pN.y - L.as * s.pS.y -
                                    af * s.pp.y - ab * s.pm.y,
                                d.y, rd.y);
    const int o = L.w + k * L.wp;
    if (L.a0 && L.a1)
        L.O[o] = make_float2(v0, v1);
    else if (L.a0)
        L.pout[2 * o] = v0;
    else if (L.a1)
        L.pout[2 * o + 1] = v1;
    if constexpr (MORE) {
        s.pm = s.pc;
        s.pc = s.pp;
        s.pp = pq;
        s.pS = sn;
        s.pN = nn;
        s.rc = rn;
        s.xw = xwn;
        s.xe = xen;
    }
}

template <int U, int MINB>
__global__ void __launch_bounds__(JP_THREADS, MINB) k_jacobi_peel(Geom g, const float* __restrict__ pin,
                                                            const float* __restrict__ rhs,
                                                            float* __restrict__ pout, int kchunk) {
    pdl_enter(pin, rhs, pout);
    const int npair = g.nx / 2 + 1;  // pairs covering columns 0 .. nx
    const int nq = npair * g.ny;
    const int qt = blockIdx.x * JP_THREADS + threadIdx.x;
    const bool qa = qt < nq;
    const int q = qa ? qt : nq - 1;  // lanes past the end shadow the last pair
    const int jr = q / npair, m = q - jr * npair;
    const int j = jr + 1, i0 = 2 * m, i1 = i0 + 1;
    const int lane = threadIdx.x & 31;
    const int k0 = 1 + blockIdx.y * kchunk, k1 = min(g.nz, k0 + kchunk - 1);
    JPLine L;
    L.P = reinterpret_cast<const float2*>(pin);
    L.R = reinterpret_cast<const float2*>(rhs);
    L.O = reinterpret_cast<float2*>(pout);
    L.pin = pin;
    L.pout = pout;
    L.a0 = qa && i0 >= 1;
    L.a1 = qa && i1 <= g.nx;
    L.ldw = lane == 0 && m > 0;            // x- neighbour of cell i0 from memory
    L.lde = lane == 31 || m == npair - 1;  // x+ neighbour of cell i1 from memory
    L.plane = g.plane;
    const int c = gidx(g, i0, j, 0);  // even
    L.cw = c - 1;
    L.ce = c + min(2, g.px - 1 - i0);
    const float cx = g.dxi * g.dxi, cy = g.dyi * g.dyi;
    L.cz = g.dzi * g.dzi;
    L.ae0 = (i0 != g.nx) ? cx : 0.0f;
    L.aw0 = (i0 != 1) ? cx : 0.0f;
    L.ae1 = (i1 != g.nx) ? cx : 0.0f;
    L.aw1 = (i1 != 1) ? cx : 0.0f;
    L.an = (j != g.ny) ? cy : 0.0f;
    L.as = (j != 1) ? cy : 0.0f;
    L.dm = make_float2(-(L.ae0 + L.aw0 + L.an + L.as + L.cz + L.cz), -(L.ae1 + L.aw1 + L.an + L.as + L.cz + L.cz));
    L.rm = make_float2(__frcp_rn(L.dm.x), __frcp_rn(L.dm.y));
    L.w = c >> 1;
    L.wp = g.plane >> 1;
    L.wr = g.px >> 1;
    JPRegs s;
    s.pm = L.P[L.w + (k0 - 1) * L.wp];
    s.pc = L.P[L.w + k0 * L.wp];
    s.pp = L.P[L.w + (k0 + 1) * L.wp];
    s.pS = L.P[L.w + k0 * L.wp - L.wr];
    s.pN = L.P[L.w + k0 * L.wp + L.wr];
    s.rc = L.R[L.w + k0 * L.wp];
    s.xw = L.ldw ? pin[L.cw + k0 * L.plane] : 0.0f;
    s.xe = L.lde ? pin[L.ce + k0 * L.plane] : 0.0f;
    int k = k0;
    if (k == 1 && k < k1) {
        jp_plane<true, true>(L, g, k, s);
        ++k;
    }
    VOF_UNROLL(U)
    for (; k < k1; ++k) jp_plane<true, false>(L, g, k, s);
    jp_plane<false, true>(L, g, k1, s);
}

// z chunk of a launch of bx blocks per chunk whose resident blocks number
// `wave`: the longest chunk (fewest reloaded planes) whose launch fills its
// last wave of blocks to 85 % or more, else the one that fills it best
// (measured on a B200 at 200^3: 7 chunks of 29 planes in one wave, or 13 of
// 16 in 1.7 waves, 0.31 ms per 10 sweeps; 8 of 25 in 1.07 waves 0.39 ms).
// Down to one plane on small grids.
int wave_kchunk(int nz, int bx, int wave) {
    int best = nz;
    double best_fill = -1.0;
    for (int n = 1; n <= nz; ++n) {
        const int kc = (nz + n - 1) / n;  // n chunks of (nearly) equal length
        const long long blocks = (long long)bx * ((nz + kc - 1) / kc);
        const long long waves = (blocks + wave - 1) / wave;
        const double fill = (double)blocks / (double)(waves * wave);
        if (fill >= 0.85) return kc;
        if (fill > best_fill) {
            best_fill = fill;
            best = kc;
        }
    }
    return best;
}

// Blocks of k_jacobi_peel resident on the device at once, set by jacobi_configure.
static int jpe_wave = 4 * 148;

cudaError_t jacobi_peel_launch(const Geom& g, const float* pin, const float* rhs, float* pout, cudaStream_t s) {
    static int forced = -1;  // VOF_JACOBI_KCHUNK: planes per block
    if (forced < 0) {
        const char* v = getenv("VOF_JACOBI_KCHUNK");
        forced = v ? atoi(v) : 0;
    }
    const int nq = (g.nx / 2 + 1) * g.ny;
    const int bx = (nq + JP_THREADS - 1) / JP_THREADS;
    const int kchunk = forced > 0 ? (forced < g.nz ? forced : g.nz) : wave_kchunk(g.nz, bx, jpe_wave);
    const dim3 grid(bx, (g.nz + kchunk - 1) / kchunk);
    return pdl_launch(k_jacobi_peel<2, 4>, grid, JP_THREADS, 0, s, g, pin, rhs, pout, kchunk);
}

cudaError_t jacobi_configure() {
    cudaError_t e;
    int dev = 0, sms = 0, occ = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_jacobi_peel<2, 4>, JP_THREADS, 0)) != cudaSuccess)
        return e;
    jpe_wave = (sms > 0 ? sms : 148) * (occ > 0 ? occ : 1);
    return cudaSuccess;
}

}  // namespace vof
