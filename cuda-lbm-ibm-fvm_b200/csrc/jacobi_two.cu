// jacobi_two.cu -- two Jacobi sweeps of the pressure system per launch
// (solve_p_jacobi_kernel, voftrial1.cu:401-439, with the ping-pong of
// voftrial1.cu:1371-1375).
//
// Compiled with -fmad=false: each cell update keeps the reference's
//     pt = (rhs - ae*pE - aw*pW - an*pN - as*pS - af*pF - ab*pB) / ap
// with the same operand order and the IEEE quotient, so the bits are those of
// two separate sweeps.  A product that several updates use (cx*p of a cell is
// its west neighbour's ae*pE and its east neighbour's aw*pW; cz*p is used one
// plane below and one above) is formed once: the coefficients of a cell
// beside a wall that are 0 are those of products of ghost cells, so a product
// depends on its own cell alone.
//
// A block owns a tile of quads (four cells of a row, one float4) and marches z.
// At iteration k it forms the first sweep's plane k from the input planes
// k-1 .. k+1 and the second sweep's plane k-1 from the first sweep's planes
// k-2 .. k.  A thread keeps its quad's column in registers (as products), its
// x neighbours come from the lanes beside, its y neighbours from shared
// memory: the input plane's rows as a TMA load brought them, the first sweep's
// plane as the block wrote it an iteration before.  One barrier per plane.
// The TMA loads of a plane of p and of rhs run J2_STAGES - 2 iterations
// ahead, from one thread, and fill with zeros outside the field.  The first
// sweep's values on the tile's edge (one row, one quad) are computed twice.
//
// What bounds it: instruction issue and its barrier, at 33 thread instructions
// per cell and sweep on the tile and 41 with its halo (the one-sweep kernel
// k_jacobi_peel: 55), with half of the issue slots used while a block runs (15
// warps an SM; stalls on the barrier, shared memory, fixed latency and the
// scheduler's choice about alike; at 200^3 39 us a launch).  DRAM and L2
// see one read of p and rhs and one write of p per two sweeps.  Without any
// load it takes 5 % less, so the copies are hidden.  Measured on a B200, whole
// passes of steps against one sweep per launch: 400^3 in flow 16.6 -> 15.1 ms
// (4 steps), 128^3 with surface tension 2.13 -> 2.00 (8), 200^3 from rest
// 7.17 -> 6.93 (12), 201 x 157 x 93 3.07 -> 2.97 (12).  512 threads of up to
// 128 registers; 608 of 96 spill (200^3 7.05, 400^3 15.3), 384 leave too few
// warps (7.3, 16.3).  The second sweep a plane later, with both sweeps' chains
// side by side, and copies by cp.async from each thread were 10 to 15 %
// slower.
#include "jacobi_two.h"

#include <type_traits>

#include "tma.cuh"

namespace vof {

#if defined(__CUDA_ARCH__) && !defined(VOF_FMAD_FALSE)
#error "jacobi_two.cu must be compiled with -fmad=false -DVOF_FMAD_FALSE"
#endif

namespace {

struct Quad {
    float v[4];
};
__device__ __forceinline__ Quad quad(const float* a) {
    const float4 t = *reinterpret_cast<const float4*>(a);
    return {{t.x, t.y, t.z, t.w}};
}

// The greatest of three, NaN if one is.
__device__ __forceinline__ float max_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Quotients x / d of a quad by Markstein's correction (div_rn_pre).  Its range
// test on the numerators alone: with every |d| between the launch's least and
// greatest, lo <= |x| <= hi implies div_rn_pre's conditions on x and q0.  One
// test per quad; exact zeros pass it (their quotients are the signed zeros).
// Numerators below lo (ahead of a pressure front every block has some) take
// div_rn_tiny's scaled quotient, in line; what that leaves (a possible
// midpoint of the subnormal grid, huge or non-finite numerators) div_rn_pre.
// Every quotient that is not finite comes that way, and rest_of(q) sees it
// (a maximum that keeps NaN: a fmaxf would drop it).
template <typename Rest>
__device__ __forceinline__ Quad quotients(const Quad& x, const Quad& d, const Quad& rd, const DivRange& w,
                                          Rest&& rest_of) {
    Quad q;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float q0 = __fmul_rn(x.v[e], rd.v[e]);
        q.v[e] = __fmaf_rn(__fmaf_rn(-q0, d.v[e], x.v[e]), rd.v[e], q0);
    }
    // twice the magnitude's bits, less one: 0 becomes the greatest number
    unsigned m[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) m[e] = 2u * __float_as_uint(x.v[e]) - 1u;
    const unsigned least = min(min(m[0], m[1]), min(m[2], m[3]));
    const float most = max_nan(max_nan(fabsf(x.v[0]), fabsf(x.v[1]), fabsf(x.v[2])), fabsf(x.v[3]), 0.0f);
    if (!(least >= w.lo2 && most <= w.hi)) {
        bool rest = !(w.tiny && most <= w.hi);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float xs = __fmul_rn(x.v[e], 0x1p+64f), s0 = __fmul_rn(xs, rd.v[e]);
            const float qs = __fmaf_rn(__fmaf_rn(-s0, d.v[e], xs), rd.v[e], s0);
            const float y = __fmul_rn(qs, 0x1p-64f);
            if (m[e] < w.lo2) {
                q.v[e] = y;
                rest |= fabsf(__fsub_rn(qs, __fmul_rn(y, 0x1p+64f))) == 0x1p-86f;
            }
        }
        if (rest) {
#pragma unroll 1
            for (int e = 0; e < 4; ++e) {
                const float xe = e == 0 ? x.v[0] : e == 1 ? x.v[1] : e == 2 ? x.v[2] : x.v[3];
                const float de = e == 0 ? d.v[0] : e == 1 ? d.v[1] : e == 2 ? d.v[2] : d.v[3];
                const float re = e == 0 ? rd.v[0] : e == 1 ? rd.v[1] : e == 2 ? rd.v[2] : rd.v[3];
                const float y = div_rn_pre(xe, de, re);
                if (e == 0) q.v[0] = y;
                if (e == 1) q.v[1] = y;
                if (e == 2) q.v[2] = y;
                if (e == 3) q.v[3] = y;
            }
            rest_of(q);
        }
    }
    return q;
}

// The updates of a quad: right-hand sides, x products of the quad and of the
// cells beside it, y neighbours (north, south) with their coefficients, z
// products from above (up) and below (dn).
template <typename Rest>
__device__ __forceinline__ Quad update(const Quad& rhs, const Quad& X, float xw, float xe, float an, const Quad& n,
                                       float as, const Quad& s, const Quad& up, const Quad& dn, const Quad& d,
                                       const Quad& rd, const DivRange& w, Rest&& rest_of) {
    Quad t;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        t.v[e] = rhs.v[e] - (e < 3 ? X.v[e + 1] : xe) - (e > 0 ? X.v[e - 1] : xw) - an * n.v[e] - as * s.v[e] -
                 up.v[e] - dn.v[e];
    return quotients(t, d, rd, w, rest_of);
}

__device__ __forceinline__ Quad scaled(float c, const Quad& a) { return {{c * a.v[0], c * a.v[1], c * a.v[2], c * a.v[3]}}; }

}  // namespace

__global__ void __launch_bounds__(J2_THREADS, 1) k_jacobi_two(Geom g, J2Plan P, const float* __restrict__ pin,
                                                              const __grid_constant__ CUtensorMap map_p,
                                                              const __grid_constant__ CUtensorMap map_r,
                                                              float* __restrict__ pout, int* status) {
    extern __shared__ __align__(128) float smem[];
    const int nq = P.nq, rows = P.rows, pitch = 4 * nq;
    const int plane = (((rows + 2) * pitch * 4 + 127) & ~127) / 4;  // floats of one TMA box, 128-byte slots
    float* const sp = smem;                                        // [stage][plane]: p
    float* const sr = smem + J2_STAGES * plane;                    // [stage][plane]: rhs
    float* const s1 = smem + 2 * J2_STAGES * plane;                // [2][plane]: the first sweep
    uint64_t* const bar = reinterpret_cast<uint64_t*>(smem + (2 * J2_STAGES + 2) * plane);

    const int t = threadIdx.x, lane = t & 31;
    const int r = min(t / nq, rows - 1), q = t - (t / nq) * nq;  // threads past the tile shadow its last row
    const bool own = t < nq * rows;
    const int xq = (int)blockIdx.x * P.wq - P.hq;  // first quad of the tile
    const int i0 = 4 * (xq + q);
    const int jlo = (int)blockIdx.y * (rows - 2);  // row 0 of the tile (j of its first halo row)
    const int j = jlo + r;
    const int k0 = 1 + (int)blockIdx.z * P.kc, k1 = min(g.nz, k0 + P.kc - 1);
    const int ka = max(1, k0 - 1), kz = k1 + 1;  // iterations

    // stage of iteration k: rhs plane k and p plane k + 1
    const unsigned bytes = 2u * (unsigned)((rows + 2) * pitch) * 4u;
    auto issue = [&](int k, int s) {
        mbar_arrive_expect_tx(&bar[s], bytes);
        tma_load_3d(sp + s * plane, &map_p, 4 * xq, jlo - 1, k + 1, &bar[s]);
        tma_load_3d(sr + s * plane, &map_r, 4 * xq, jlo - 1, k, &bar[s]);
    };
    if (t == 0) {
        for (int s = 0; s < J2_STAGES; ++s) mbar_init(&bar[s], 1);
        fence_mbar_init();
        for (int s = 0; s < J2_STAGES && ka - 1 + s <= kz; ++s) issue(ka - 1 + s, s);
    }
    __syncthreads();

    const float cx = g.dxi * g.dxi, cy = g.dyi * g.dyi, cz = g.dzi * g.dzi;
    const float an = j < g.ny ? cy : 0.0f, as = j > 1 ? cy : 0.0f;
    // cx of a cell's product; 0 for the ghosts (it enters only the updates beside a wall)
    const float c0 = i0 == 0 || i0 == g.nx + 1 ? 0.0f : cx, c1 = i0 + 1 == g.nx + 1 ? 0.0f : cx;
    const float c2 = i0 + 2 == g.nx + 1 ? 0.0f : cx, c3 = i0 + 3 == g.nx + 1 ? 0.0f : cx;
    const float ce = i0 + 4 == g.nx + 1 ? 0.0f : cx;
    auto xprod = [&](const Quad& a) { return Quad{{c0 * a.v[0], c1 * a.v[1], c2 * a.v[2], c3 * a.v[3]}}; };
    auto diagonal = [&](float af, float ab, Quad& d, Quad& rd) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float ae = i0 + e != g.nx ? cx : 0.0f, aw = i0 + e != 1 ? cx : 0.0f;
            d.v[e] = -(ae + aw + an + as + af + ab);
            rd.v[e] = __frcp_rn(d.v[e]);
        }
    };
    const DivRange w = div_range(g);
    Quad d, rd;
    diagonal(cz, cz, d, rd);

    // quads of the first sweep (the others keep 0: they enter through zero
    // coefficients only) and of the second
    const bool first = own && j >= 1 && j <= g.ny && i0 >= 0 && i0 <= g.nx;
    const bool out = first && r >= 1 && r <= rows - 2 && q >= P.hq && q < nq - P.hq;
    const bool whole = i0 >= 1 && i0 + 3 <= g.nx;
    // The first sweep forms values for a row's ghosts as well, which enter the
    // second through a coefficient of 0 only: not where they overflow (huge
    // values in the ghosts of p, any in those of rhs).
    auto clear = [&](Quad& q) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (i0 + e < 1 || i0 + e > g.nx) q.v[e] = 0.0f;
    };
    auto leave = [](Quad&) {};
    const int so = (r + 1) * pitch + 4 * q;  // own quad in a plane slot (row 0: the row before the tile)

    Quad zm, zc, pc;  // A: cz * p(k-1), cz * p(k), p(k)
    Quad wm = {{0, 0, 0, 0}}, wc = wm, ic = wm, rp = wm;  // B: cz * p1(k-2), cz * p1(k-1), p1(k-1), rhs(k-1)
    {
        const bool in = i0 >= 0 && i0 + 3 < g.px && j < g.py;
        const Quad pm = in ? quad(pin + gidx(g, i0, j, ka - 1)) : wm;
        zm = scaled(ka > 1 ? cz : 0.0f, pm);
    }
    bool ok = mbar_wait(&bar[0], 0);
    pc = quad(sp + so);
    zc = scaled(cz, pc);
    // stages of iterations k - 1 and k (offsets of their slots), the parity of
    // the wait for k; buffers of the first sweep's planes k and k - 1
    int cur = 0, nxt = 1, phase = 0;
    const float* pk = sp + so;              // own quad in p's plane k
    float* sa = s1 + (ka & 1) * plane + so;
    float* sb = s1 + (~ka & 1) * plane + so;
    float* o = pout + gidx(g, i0, j, ka - 1);
    // Iteration k.  EDGE: k or k - 1 may be the first or last plane of the box,
    // or k may be before the second sweep's first iteration or past the box.
    auto step = [&](int k, auto edge) {
        constexpr bool EDGE = decltype(edge)::value;
        ok &= mbar_wait(&bar[nxt], phase);
        const float* pkn = sp + nxt * plane + so;
        const Quad rk = quad(pkn + J2_STAGES * plane);
        Quad in = {{0, 0, 0, 0}};
        if (!EDGE || k <= g.nz) {  // first sweep, plane k
            const Quad pn = quad(pkn);
            const Quad up = scaled(!EDGE || k < g.nz ? cz : 0.0f, pn);
            const Quad X = xprod(pc);
            float xw = __shfl_up_sync(0xffffffffu, X.v[3], 1), xe = __shfl_down_sync(0xffffffffu, X.v[0], 1);
            if (first) {
                if (lane == 0) xw = cx * pk[-1];
                if (lane == 31) xe = ce * pk[4];
                if (EDGE) {
                    Quad dk, rdk;
                    diagonal(k < g.nz ? cz : 0.0f, k > 1 ? cz : 0.0f, dk, rdk);
                    in = update(rk, X, xw, xe, an, quad(pk + pitch), as, quad(pk - pitch), up, zm, dk, rdk, w, clear);
                } else {
                    in = update(rk, X, xw, xe, an, quad(pk + pitch), as, quad(pk - pitch), up, zm, d, rd, w, clear);
                }
            }
            zm = zc;
            zc = up;
            pc = pn;
        }
        const Quad wn = scaled(cz, in);
        if (!EDGE || k > k0) {  // second sweep, plane k - 1
            const Quad X = xprod(ic);
            float xw = __shfl_up_sync(0xffffffffu, X.v[3], 1), xe = __shfl_down_sync(0xffffffffu, X.v[0], 1);
            if (out) {
                if (lane == 0) xw = cx * sb[-1];
                if (lane == 31) xe = ce * sb[4];
                Quad v;
                if (EDGE) {
                    Quad dk, rdk;
                    diagonal(k <= g.nz ? cz : 0.0f, k > 2 ? cz : 0.0f, dk, rdk);
                    v = update(rp, X, xw, xe, an, quad(sb + pitch), as, quad(sb - pitch), wn, wm, dk, rdk, w, leave);
                } else {
                    v = update(rp, X, xw, xe, an, quad(sb + pitch), as, quad(sb - pitch), wn, wm, d, rd, w, leave);
                }
                if (whole) {
                    *reinterpret_cast<float4*>(o) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (i0 + e >= 1 && i0 + e <= g.nx) o[e] = v.v[e];
                }
            }
        }
        if (own) *reinterpret_cast<float4*>(sa) = make_float4(in.v[0], in.v[1], in.v[2], in.v[3]);
        wm = wc;
        wc = wn;
        ic = in;
        rp = rk;
        __syncthreads();
        // the stage of iteration k - 1 is no longer read: refill it
        if (t == 0 && k - 1 + J2_STAGES <= kz) {
            fence_proxy_async_smem();
            issue(k - 1 + J2_STAGES, cur);
        }
        cur = nxt;
        if (++nxt == J2_STAGES) {
            nxt = 0;
            phase ^= 1;
        }
        pk = pkn;
        float* x = sa;
        sa = sb;
        sb = x;
        o += g.plane;
    };
    using Inner = std::integral_constant<bool, false>;
    using Edge = std::integral_constant<bool, true>;
    const int m0 = max(3, k0 + 1), m1 = min(kz, g.nz - 1);  // inner iterations, two at a time (registers renamed)
    int k = ka;
    for (; k < m0 && k <= kz; ++k) step(k, Edge{});
#pragma unroll 1
    for (; k < m1; k += 2) {
        step(k, Inner{});
        step(k + 1, Inner{});
    }
    for (; k <= kz; ++k) step(k, Edge{});
    if (!ok) {
        // a copy that did not land in time may still be in flight: wait (bounded) for the stages before leaving
        for (int s = 0; s < J2_STAGES; ++s) mbar_wait(&bar[s], s >= nxt ? phase : phase ^ 1, 1u << 16);
        atomicOr(status, DEV_TMA_TIMEOUT);
    }
}

// Columns [from, px) of every row set to 1 (a warp per row; px - from <= 31).
__global__ void __launch_bounds__(256) k_fill_padding(float* a, int px, int from, int rows) {
    const int i = from + (threadIdx.x & 31);
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8)
        if (i < px) a[(size_t)r * px + i] = 1.0f;
}

cudaError_t jacobi_two_prepare(const Geom& g, float* const field[4], J2Tables* t, cudaStream_t s) {
    t->plan = j2_plan(g.nx, g.ny, g.nz);
    const J2Plan& p = t->plan;
    for (int q = 0; q < 4; ++q) {
        const cudaError_t e =
            make_tensor_map_3d(&t->map[q], field[q], g.px, g.py, g.nz + 2, 4 * p.nq, p.rows + 2, 1);
        if (e != cudaSuccess) return e;
    }
    const int rows = g.py * (g.nz + 2);
    k_fill_padding<<<rows < 4736 ? (rows + 7) / 8 : 592, 256, 0, s>>>(field[3], g.px, g.nx + 2, rows);
    return cudaGetLastError();
}

cudaError_t jacobi_two_launch(const Geom& g, const J2Tables& t, int in, const float* pin, float* pout, int* status,
                              cudaStream_t s) {
    const J2Plan& p = t.plan;
    const dim3 grid(p.tx, p.ty, (g.nz + p.kc - 1) / p.kc);
    k_jacobi_two<<<grid, p.threads, p.smem, s>>>(g, p, pin, t.map[in], t.map[3], pout, status);
    return cudaGetLastError();
}

cudaError_t jacobi_two_configure() {
    return cudaFuncSetAttribute(k_jacobi_two, cudaFuncAttributeMaxDynamicSharedMemorySize, J2_SMEM);
}

}  // namespace vof
