// plain_step.cu -- the FP32 drop-in step (voftrial1.cu:1364-1401) as fused
// sm_100a kernels over the padded layout of vof_device.cuh.
//
// Arithmetic contract: every per-point expression keeps the reference's
// operand order, and this translation unit is compiled with -fmad=false, so
// no multiply-add is contracted into an FMA.  The results are therefore
// bit-identical to the reference's kernels compiled with -fmad=false and to
// the FP32 CPU restatement in oracle/ (built with -ffp-contract=off); the
// reference built with nvcc's default -fmad=true differs from both in the
// last bits of contracted expressions.
//
// Kernel map (reference kernels each one replaces):
//   k_predict2     advect_{u,v,w}_kernel + cal_nu_rho_kernel   voftrial1.cu:95-104, 230-399
//                  two cells per thread (k_predict: one; VOF_PREDICT=1)
//   k_rhs4         the rhs expression of solve_p_jacobi_kernel voftrial1.cu:418-422
//                  four cells per thread (k_rhs: one, marching z; VOF_RHS=1)
//   k_jacobi_two   (jacobi_two.cu) two solve_p_jacobi_kernel sweeps per launch,  voftrial1.cu:401-439
//                  four cells per thread (an odd one: k_jacobi_peel, jacobi.cu);
//                  all of them in one cluster on small grids: k_jacobi_cluster
//   k_correct4     update_{u,v,w}_kernel + apply_bc_velocity   voftrial1.cu:441-493, 959-1051, 1107-1120
//                  four cells per thread (k_correct: one; VOF_CORRECT=1)
//   k_fct_tile     (fct_sweep.cu; k_fct_lines on small grids) fct_{x,y,z}_sweep_stage1..4, and on
//                  the last sweep post_process_f_kernel + apply_bc_F   voftrial1.cu:502-905, 1053-1135
#include "plain_step.h"

#include "fct_sweep.h"
#include "jacobi.h"
#include "jacobi_cluster.h"
#include "jacobi_two.h"
#include "pdl.cuh"

#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

namespace vof {

#ifndef VOF_PLAIN_NO_FMAD_CHECK
// Compile-time guard: the build must pass -fmad=false for this file.
#if defined(__CUDA_ARCH__) && !defined(VOF_FMAD_FALSE)
#error "plain_step.cu must be compiled with -fmad=false -DVOF_FMAD_FALSE"
#endif
#endif

// All kernels below march along z: a thread owns one (i, j) column of a
// 32 x 8 tile and walks a chunk of k, computing its index once and carrying
// the column's k-1 / k / k+1 values in registers; in-plane neighbours come
// from L1.  The per-point arithmetic is the reference's, unchanged.
constexpr int TX = 32, TY = 8;

struct Column {
    int i, j, k0, k1;
    __device__ Column(const Geom& g, int lo_i, int lo_j, int kchunk) {
        i = blockIdx.x * TX + threadIdx.x + lo_i;
        j = blockIdx.y * TY + threadIdx.y + lo_j;
        k0 = 1 + blockIdx.z * kchunk;
        k1 = min(g.nz, k0 + kchunk - 1);
    }
};

// Indices whose clamped value is x on an axis of n interior cells: x itself,
// plus the ghost 0 when x == 1 and the ghost n+1 when x == n.
__device__ __forceinline__ int mirrors(int x, int n, int* out) {
    // fixed positions (no runtime index: the list stays in registers)
    out[0] = x;
    out[1] = (x == 1) ? 0 : n + 1;
    out[2] = n + 1;
    return 1 + (x == 1) + (x == n);
}

// ---------------------------------------------------------------------------
// Momentum predictor: u*, v*, w* on the interior faces the reference updates
// (u: i in [imin+1, imax], j,k interior; v, w likewise), nu from F on the fly.
// advect_u/v/w_kernel + cal_nu_rho_kernel, voftrial1.cu:95-104, 230-399.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_predict(Geom g,
                                                 const float* __restrict__ F,
                                                 const float* __restrict__ u,
                                                 const float* __restrict__ v,
                                                 const float* __restrict__ w,
                                                 float* __restrict__ us,
                                                 float* __restrict__ vs,
                                                 float* __restrict__ ws, int kchunk) {
    const Column col(g, 1, 1, kchunk);
    const int i = col.i, j = col.j;
    if (i > g.nx || j > g.ny || col.k0 > g.nz) return;
    const int sy = g.px, sz = g.plane;
    int id = gidx(g, i, j, col.k0);
    // column windows along k
    float u_km = __ldg(u + id - sz), u_c = __ldg(u + id);
    float v_km = __ldg(v + id - sz), v_c = __ldg(v + id);
    float w_km = __ldg(w + id - sz), w_c = __ldg(w + id);
    float wim_c = __ldg(w + id - 1), wjm_c = __ldg(w + id - sy);
    float uip_km = __ldg(u + id + 1 - sz), vjp_km = __ldg(v + id + sy - sz);
    for (int k = col.k0; k <= col.k1; ++k, id += sz) {
        const float u_kp = __ldg(u + id + sz), v_kp = __ldg(v + id + sz), w_kp = __ldg(w + id + sz);
        const float wim_kp = __ldg(w + id - 1 + sz), wjm_kp = __ldg(w + id - sy + sz);
        const float uip_c = __ldg(u + id + 1), vjp_c = __ldg(v + id + sy);
        const float nu = nu_of(g, __ldg(F + id));

        if (i >= 2) {  // advect_u_kernel, voftrial1.cu:230-285
            const float v_here = 0.25f * (__ldg(v + id - 1) + __ldg(v + id - 1 + sy) + v_c + vjp_c);
            const float w_here = 0.25f * (wim_c + wim_kp + w_c + w_kp);
            const float uim = __ldg(u + id - 1);
            const float ujm = __ldg(u + id - sy), ujp = __ldg(u + id + sy);
            const float dudx = (u_c > 0.0f) ? (u_c - uim) * g.dxi : (uip_c - u_c) * g.dxi;
            const float dudy = (v_here > 0.0f) ? (u_c - ujm) * g.dyi : (ujp - u_c) * g.dyi;
            const float dudz = (w_here > 0.0f) ? (u_c - u_km) * g.dzi : (u_kp - u_c) * g.dzi;
            const float visc = nu * (uim - 2.0f * u_c + uip_c) * g.dxi * g.dxi +
                               nu * (ujm - 2.0f * u_c + ujp) * g.dyi * g.dyi +
                               nu * (u_km - 2.0f * u_c + u_kp) * g.dzi * g.dzi;
            const float adv = -u_c * dudx - v_here * dudy - w_here * dudz;
            us[id] = u_c + g.dt * (visc + adv + g.gx);
        }
        if (j >= 2) {  // advect_v_kernel, voftrial1.cu:287-342
            const float u_here = 0.25f * (__ldg(u + id - sy) + u_c + __ldg(u + id + 1 - sy) + uip_c);
            const float w_here = 0.25f * (wjm_kp + wjm_c + w_c + w_kp);
            const float vim = __ldg(v + id - 1), vip = __ldg(v + id + 1);
            const float vjm = __ldg(v + id - sy);
            const float dvdx = (u_here > 0.0f) ? (v_c - vim) * g.dxi : (vip - v_c) * g.dxi;
            const float dvdy = (v_c > 0.0f) ? (v_c - vjm) * g.dyi : (vjp_c - v_c) * g.dyi;
            const float dvdz = (w_here > 0.0f) ? (v_c - v_km) * g.dzi : (v_kp - v_c) * g.dzi;
            const float visc = nu * (vim - 2.0f * v_c + vip) * g.dxi * g.dxi +
                               nu * (vjm - 2.0f * v_c + vjp_c) * g.dyi * g.dyi +
                               nu * (v_km - 2.0f * v_c + v_kp) * g.dzi * g.dzi;
            const float adv = -u_here * dvdx - v_c * dvdy - w_here * dvdz;
            vs[id] = v_c + g.dt * (visc + adv + g.gy);
        }
        if (k >= 2) {  // advect_w_kernel, voftrial1.cu:344-399
            const float u_here = 0.25f * (uip_km + u_km + uip_c + u_c);
            const float v_here = 0.25f * (vjp_km + v_km + v_c + vjp_c);
            const float wip = __ldg(w + id + 1), wjp = __ldg(w + id + sy);
            const float dwdx = (u_here > 0.0f) ? (w_c - wim_c) * g.dxi : (wip - w_c) * g.dxi;
            const float dwdy = (v_here > 0.0f) ? (w_c - wjm_c) * g.dyi : (wjp - w_c) * g.dyi;
            const float dwdz = (w_c > 0.0f) ? (w_c - w_km) * g.dzi : (w_kp - w_c) * g.dzi;
            const float visc = nu * (wim_c - 2.0f * w_c + wip) * g.dxi * g.dxi +
                               nu * (wjm_c - 2.0f * w_c + wjp) * g.dyi * g.dyi +
                               nu * (w_km - 2.0f * w_c + w_kp) * g.dzi * g.dzi;
            const float adv = -u_here * dwdx - v_here * dwdy - w_c * dwdz;
            ws[id] = w_c + g.dt * (visc + adv + g.gz);
        }
        u_km = u_c; u_c = u_kp;
        v_km = v_c; v_c = v_kp;
        w_km = w_c; w_c = w_kp;
        wim_c = wim_kp; wjm_c = wjm_kp;
        uip_km = uip_c; vjp_km = vjp_c;
    }
}

// ---------------------------------------------------------------------------
// Continuum surface force (extension; no counterpart in the reference, whose
// sigma no kernel reads).  J. U. Brackbill, D. B. Kothe, C. Zemach, "A
// continuum method for modeling surface tension", J. Comput. Phys. 100 (1992):
// the body force sigma kappa grad(F) with the interface normal n = grad F /
// |grad F| and kappa = -div n, both by central differences at cell centres;
// F's ghosts are the zero-gradient copies, and a normal beyond a wall is the
// mirror image of the one inside (its wall-normal component negated: a 90
// degree contact angle).  On a face, kappa is the mean of its two cells,
// grad F their difference, and the acceleration is divided by the face
// density of the correction, 0.5 (rho_a + rho_b); the predictor adds it to u*,
// v*, w* on the faces it updates.  FP32, operations in a fixed order.
// ---------------------------------------------------------------------------
// The normal at a cell from the differences of its neighbours; zero where the
// gradient is no larger than eps (or NaN), as it is at most cells: away from
// the interface the differences are zeros and no root or quotient is formed.
struct Normal {
    float x, y, z;
};
__device__ __forceinline__ Normal csf_normal(float dx, float dy, float dz, float hx, float hy, float hz, float eps) {
    Normal n = {0.0f, 0.0f, 0.0f};
    if (dx == 0.0f && dy == 0.0f && dz == 0.0f) return n;
    const float gxv = dx * hx, gyv = dy * hy, gzv = dz * hz;
    const float mag = sqrtf(gxv * gxv + gyv * gyv + gzv * gzv);
    if (!(mag > eps)) return n;
    if (mag >= 0x1p-100f && mag < 0x1p+126f) {  // div_rn_pre's divisors
        const float r = __frcp_rn(mag);
        n.x = div_rn_pre(gxv, mag, r);
        n.y = div_rn_pre(gyv, mag, r);
        n.z = div_rn_pre(gzv, mag, r);
    } else {
        n.x = gxv / mag;
        n.y = gyv / mag;
        n.z = gzv / mag;
    }
    return n;
}

// kappa from F.  A block covers 32 x 16 columns, the outermost of them a halo
// for the differences of the normals, and marches a chunk of planes: at plane k
// a thread forms its normal, takes the x neighbours' from the lanes beside, the
// y neighbours' from shared memory, and keeps the in-plane part of the
// divergence until the next plane's normal completes it.  18 us at 128^3, where
// a pass that stored the normals and one that read them took 17.4 + 12.1, and
// the normals of the six neighbours formed per cell 23.6.  Bound by the warps
// with interface cells, which the block waits for (chunks of 4 to 16 planes,
// loads a plane ahead, 8 rows: 17.3 to 19.6).
constexpr int CSF_X = 32, CSF_Y = 16;
__global__ void __launch_bounds__(CSF_X* CSF_Y, 3) k_csf_curv(Geom g, const float* __restrict__ F,
                                                              float* __restrict__ kap, int kchunk) {
    __shared__ float rows[2][CSF_Y][CSF_X];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i = blockIdx.x * (CSF_X - 2) + tx, j = blockIdx.y * (CSF_Y - 2) + ty;
    const int k0 = 1 + blockIdx.z * kchunk, k1 = min(g.nz, k0 + kchunk - 1);
    const int ka = max(1, k0 - 1), kb = min(g.nz, k1 + 1);
    const bool in = i >= 1 && i <= g.nx && j >= 1 && j <= g.ny;
    const bool out = in && tx >= 1 && tx < CSF_X - 1 && ty >= 1 && ty < CSF_Y - 1;
    const int sy = g.px, sz = g.plane;
    const float hx = 0.5f * g.dxi, hy = 0.5f * g.dyi, hz = 0.5f * g.dzi;
    const float eps = 1e-6f * g.dxi;
    int id = gidx(g, i, j, ka);
    float fm = in ? __ldg(F + id - sz) : 0.0f, fc = in ? __ldg(F + id) : 0.0f;
    float zm = 0.0f, zc = 0.0f, plane = 0.0f;  // the z components at k - 2 and k - 1, the in-plane part at k - 1
    for (int k = ka; k <= kb; ++k, id += sz) {
        Normal n = {0.0f, 0.0f, 0.0f};
        float fp = 0.0f;
        if (in) {
            fp = __ldg(F + id + sz);
            n = csf_normal(__ldg(F + id + 1) - __ldg(F + id - 1), __ldg(F + id + sy) - __ldg(F + id - sy), fp - fm, hx,
                           hy, hz, eps);
        }
        rows[k & 1][ty][tx] = n.y;
        if (out && k > k0) kap[id - sz] = -(plane + (n.z - (k > 2 ? zm : -zc)) * hz);
        const float e = __shfl_down_sync(0xffffffffu, n.x, 1), w = __shfl_up_sync(0xffffffffu, n.x, 1);
        __syncthreads();
        if (out) {
            // neighbours beyond a wall: the mirror image of the cell at the wall
            const float xe = i < g.nx ? e : -n.x, xw = i > 1 ? w : -n.x;
            const float yn = j < g.ny ? rows[k & 1][ty + 1][tx] : -n.y, ys = j > 1 ? rows[k & 1][ty - 1][tx] : -n.y;
            plane = (xe - xw) * hx + (yn - ys) * hy;
        }
        zm = zc;
        zc = n.z;
        fm = fc;
        fc = fp;
    }
    if (out && k1 == g.nz) kap[id - sz] = -(plane + (-zc - (g.nz > 1 ? zm : -zc)) * hz);
}

// A face's acceleration: the force (csf_force) over its density.  A force of
// +-0, as away from the interface, is its own quotient when the densities are
// positive (r lies between the two).
__device__ __forceinline__ float csf_force(const Geom& g, float Fa, float Fb, float ka, float kb, float hinv) {
    return g.sigma * (0.5f * (ka + kb)) * ((Fb - Fa) * hinv);
}
__device__ __forceinline__ float csf_accel(const Geom& g, float f, float Fa, float Fb) {
    if (f == 0.0f && fminf(g.rpair[0], g.rpair[1]) > 1e-30f) return f;
    const float r = 0.5f * (rho_of(g, Fa) + rho_of(g, Fb));
    return f / r;
}

// The predictor with two cells per thread.  Cells are paired by padded column
// (2m, 2m + 1: one aligned 8-byte word), the pairs of all rows of a plane
// numbered flat so that 32 consecutive pairs make a warp across row ends, and
// a thread marches a chunk of planes, carrying its pair's k-1 / k values in
// registers as k_predict does.  Every operand is a float2 load (10 per pair
// and plane: u, v, w of the next plane, the rows j-1 and j+1 of u, v, w,
// w of the next plane's row j-1, v of row j+1, and F); the x-1 and x+1
// neighbours come from the lanes beside (a pair's left neighbour is the left
// lane's second cell, its right neighbour the right lane's first), or from
// memory at the ends of a warp and of a row.  Each cell's three updates keep
// k_predict's expressions and operand order (same bits).  Bound by instruction
// issue (209 thread instructions per cell, 70 % of the slots used): 77 -> 70
// us at 200^3 and 507 -> 476 at 400^3 by march_kchunk's shorter chunks, of
// which blocks of 128 threads rather than 256 are 1 to 3 %.  Packed FP32 pairs
// (f32x2) took 99 us at 200^3, one viscosity for two equal cells 76.6.
// The pair's left (x-1 of the first cell) and right (x+1 of the second cell)
// neighbours of a value held as a pair by every lane.
__device__ __forceinline__ float left_of(float2 a, bool ldw, const float* __restrict__ p, int idl) {
    const float s = __shfl_up_sync(0xffffffffu, a.y, 1);
    return ldw ? __ldg(p + idl) : s;
}
__device__ __forceinline__ float right_of(float2 a, bool lde, const float* __restrict__ p, int idr) {
    const float s = __shfl_down_sync(0xffffffffu, a.x, 1);
    return lde ? __ldg(p + idr) : s;
}

// PDL: launched ahead of the end of the kernel before (pdl.cuh; small grids).
// CSF: the surface tension's acceleration added to each face: 31.4 us at 128^3
// (21.6 without), a pass over u*, v*, w* of its own 17.4 to 24.8 more.
template <bool CSF, bool PDL>
__global__ void __launch_bounds__(128, CSF ? 6 : 8) k_predict2(Geom g, const float* __restrict__ F,
                                                               const float* __restrict__ u,
                                                               const float* __restrict__ v,
                                                               const float* __restrict__ w, float* __restrict__ us,
                                                               float* __restrict__ vs, float* __restrict__ ws,
                                                               int kchunk, const float* __restrict__ kap) {
    if constexpr (PDL) pdl_enter(F, u, v, w, us, vs, ws);
    const int npair = g.nx / 2 + 1;  // pairs covering columns 0 .. nx
    const int nq = npair * g.ny;
    const int qt = blockIdx.x * blockDim.x + threadIdx.x;
    const bool qa = qt < nq;
    const int q = qa ? qt : nq - 1;  // lanes past the end shadow the last pair
    const int jr = q / npair, m = q - jr * npair;
    const int j = jr + 1, i0 = 2 * m;
    const int lane = threadIdx.x & 31;
    const bool ldw = lane == 0 && m > 0;            // x-1 neighbours from memory
    const bool lde = lane == 31 || m == npair - 1;  // x+1 neighbours from memory
    const int k0 = 1 + blockIdx.y * kchunk, k1 = min(g.nz, k0 + kchunk - 1);
    const int sy = g.px, sz = g.plane;
    // which cells of the pair are updated (u from i = 2, v and w from i = 1)
    const bool a0 = qa && i0 >= 1 && i0 <= g.nx, a1 = qa && i0 + 1 <= g.nx;
    const bool u0 = qa && i0 >= 2 && i0 <= g.nx, u1 = qa && i0 + 1 >= 2 && i0 + 1 <= g.nx;
    auto L2 = [](const float* __restrict__ p, int id) { return __ldg(reinterpret_cast<const float2*>(p + id)); };
    int id = gidx(g, i0, j, k0);  // even
    // column windows along k (values of the pair's two cells)
    float2 u_km = L2(u, id - sz), u_c = L2(u, id);
    float2 v_km = L2(v, id - sz), v_c = L2(v, id);
    float2 w_km = L2(w, id - sz), w_c = L2(w, id);
    float2 wjm_c = L2(w, id - sy), vjp_km = L2(v, id + sy - sz);
    // x neighbours carried from the previous plane
    float wim_c = left_of(w_c, ldw, w, id - 1);
    float uip_km = right_of(u_km, lde, u, id + 2 - sz);
    float2 f_km, kap_km;
    if (CSF) {
        f_km = L2(F, id - sz);
        kap_km = L2(kap, id - sz);
    }
    for (int k = k0; k <= k1; ++k, id += sz) {
        const float2 u_kp = L2(u, id + sz), v_kp = L2(v, id + sz), w_kp = L2(w, id + sz);
        const float2 wjm_kp = L2(w, id - sy + sz), vjp_c = L2(v, id + sy);
        const float2 ujm = L2(u, id - sy), ujp = L2(u, id + sy), vjm = L2(v, id - sy), wjp = L2(w, id + sy);
        const float2 f2 = L2(F, id);
        const float wim_kp = left_of(w_kp, ldw, w, id - 1 + sz);
        const float uim0 = left_of(u_c, ldw, u, id - 1), uip1 = right_of(u_c, lde, u, id + 2);
        const float vim0 = left_of(v_c, ldw, v, id - 1), vip1 = right_of(v_c, lde, v, id + 2);
        const float vjp_im0 = left_of(vjp_c, ldw, v, id - 1 + sy);
        const float ujm_ip1 = right_of(ujm, lde, u, id + 2 - sy);
        const float wip1 = right_of(w_c, lde, w, id + 2);
        float out_u[2], out_v[2], out_w[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            // this cell's values and its x neighbours
            const float uc = e ? u_c.y : u_c.x, ukm = e ? u_km.y : u_km.x, ukp = e ? u_kp.y : u_kp.x;
            const float vc = e ? v_c.y : v_c.x, vkm = e ? v_km.y : v_km.x, vkp = e ? v_kp.y : v_kp.x;
            const float wc = e ? w_c.y : w_c.x, wkm = e ? w_km.y : w_km.x, wkp = e ? w_kp.y : w_kp.x;
            const float uim = e ? u_c.x : uim0, uip_c = e ? uip1 : u_c.y;
            const float vim = e ? v_c.x : vim0, vip = e ? vip1 : v_c.y;
            const float wim_cc = e ? w_c.x : wim_c, wim_kpp = e ? w_kp.x : wim_kp;
            const float wip = e ? wip1 : w_c.y;
            const float vjpc = e ? vjp_c.y : vjp_c.x, vjp_im = e ? vjp_c.x : vjp_im0;
            const float vjpkm = e ? vjp_km.y : vjp_km.x;
            const float ujmc = e ? ujm.y : ujm.x, ujpc = e ? ujp.y : ujp.x, ujm_ip = e ? ujm_ip1 : ujm.y;
            const float vjmc = e ? vjm.y : vjm.x;
            const float wjmc = e ? wjm_c.y : wjm_c.x, wjmkp = e ? wjm_kp.y : wjm_kp.x;
            const float wjpc = e ? wjp.y : wjp.x;
            const float uipkm = e ? uip_km : u_km.y;
            const float nu = nu_of(g, e ? f2.y : f2.x);
            {  // advect_u_kernel, voftrial1.cu:230-285
                const float v_here = 0.25f * (vim + vjp_im + vc + vjpc);
                const float w_here = 0.25f * (wim_cc + wim_kpp + wc + wkp);
                const float dudx = (uc > 0.0f) ? (uc - uim) * g.dxi : (uip_c - uc) * g.dxi;
                const float dudy = (v_here > 0.0f) ? (uc - ujmc) * g.dyi : (ujpc - uc) * g.dyi;
                const float dudz = (w_here > 0.0f) ? (uc - ukm) * g.dzi : (ukp - uc) * g.dzi;
                const float visc = nu * (uim - 2.0f * uc + uip_c) * g.dxi * g.dxi +
                                   nu * (ujmc - 2.0f * uc + ujpc) * g.dyi * g.dyi +
                                   nu * (ukm - 2.0f * uc + ukp) * g.dzi * g.dzi;
                const float adv = -uc * dudx - v_here * dudy - w_here * dudz;
                out_u[e] = uc + g.dt * (visc + adv + g.gx);
            }
            {  // advect_v_kernel, voftrial1.cu:287-342
                const float u_here = 0.25f * (ujmc + uc + ujm_ip + uip_c);
                const float w_here = 0.25f * (wjmkp + wjmc + wc + wkp);
                const float dvdx = (u_here > 0.0f) ? (vc - vim) * g.dxi : (vip - vc) * g.dxi;
                const float dvdy = (vc > 0.0f) ? (vc - vjmc) * g.dyi : (vjpc - vc) * g.dyi;
                const float dvdz = (w_here > 0.0f) ? (vc - vkm) * g.dzi : (vkp - vc) * g.dzi;
                const float visc = nu * (vim - 2.0f * vc + vip) * g.dxi * g.dxi +
                                   nu * (vjmc - 2.0f * vc + vjpc) * g.dyi * g.dyi +
                                   nu * (vkm - 2.0f * vc + vkp) * g.dzi * g.dzi;
                const float adv = -u_here * dvdx - vc * dvdy - w_here * dvdz;
                out_v[e] = vc + g.dt * (visc + adv + g.gy);
            }
            {  // advect_w_kernel, voftrial1.cu:344-399
                const float u_here = 0.25f * (uipkm + ukm + uip_c + uc);
                const float v_here = 0.25f * (vjpkm + vkm + vc + vjpc);
                const float dwdx = (u_here > 0.0f) ? (wc - wim_cc) * g.dxi : (wip - wc) * g.dxi;
                const float dwdy = (v_here > 0.0f) ? (wc - wjmc) * g.dyi : (wjpc - wc) * g.dyi;
                const float dwdz = (wc > 0.0f) ? (wc - wkm) * g.dzi : (wkp - wc) * g.dzi;
                const float visc = nu * (wim_cc - 2.0f * wc + wip) * g.dxi * g.dxi +
                                   nu * (wjmc - 2.0f * wc + wjpc) * g.dyi * g.dyi +
                                   nu * (wkm - 2.0f * wc + wkp) * g.dzi * g.dzi;
                const float adv = -u_here * dwdx - v_here * dwdy - wc * dwdz;
                out_w[e] = wc + g.dt * (visc + adv + g.gz);
            }
        }
        if (CSF) {
            const float2 kc = L2(kap, id), fj = L2(F, id - sy), kj = L2(kap, id - sy);
            const float fi = left_of(f2, ldw, F, id - 1), ki = left_of(kc, ldw, kap, id - 1);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float Fc = e ? f2.y : f2.x, kk = e ? kc.y : kc.x;
                const float Fx = e ? f2.x : fi, Fy = e ? fj.y : fj.x, Fz = e ? f_km.y : f_km.x;
                const float ax = csf_force(g, Fx, Fc, e ? kc.x : ki, kk, g.dxi);
                const float ay = csf_force(g, Fy, Fc, e ? kj.y : kj.x, kk, g.dyi);
                const float az = csf_force(g, Fz, Fc, e ? kap_km.y : kap_km.x, kk, g.dzi);
                out_u[e] = out_u[e] + g.dt * csf_accel(g, ax, Fx, Fc);
                out_v[e] = out_v[e] + g.dt * csf_accel(g, ay, Fy, Fc);
                out_w[e] = out_w[e] + g.dt * csf_accel(g, az, Fz, Fc);
            }
            f_km = f2;
            kap_km = kc;
        }
        float2* US = reinterpret_cast<float2*>(us + id);
        if (u0 && u1)
            *US = make_float2(out_u[0], out_u[1]);
        else if (u0)
            us[id] = out_u[0];
        else if (u1)
            us[id + 1] = out_u[1];
        if (j >= 2) {
            if (a0 && a1)
                *reinterpret_cast<float2*>(vs + id) = make_float2(out_v[0], out_v[1]);
            else if (a0)
                vs[id] = out_v[0];
            else if (a1)
                vs[id + 1] = out_v[1];
        }
        if (k >= 2) {
            if (a0 && a1)
                *reinterpret_cast<float2*>(ws + id) = make_float2(out_w[0], out_w[1]);
            else if (a0)
                ws[id] = out_w[0];
            else if (a1)
                ws[id + 1] = out_w[1];
        }
        u_km = u_c;
        u_c = u_kp;
        v_km = v_c;
        v_c = v_kp;
        w_km = w_c;
        w_c = w_kp;
        wim_c = wim_kp;
        wjm_c = wjm_kp;
        uip_km = uip1;
        vjp_km = vjp_c;
    }
}

// ---------------------------------------------------------------------------
// Pressure right-hand side rho/dt * div(u*) (voftrial1.cu:418-422).  Without
// FMA contraction the stored value is exactly the one the reference forms
// inside every Jacobi sweep, so computing it once per step changes nothing.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_rhs(Geom g,
                                             const float* __restrict__ F,
                                             const float* __restrict__ us,
                                             const float* __restrict__ vs,
                                             const float* __restrict__ ws,
                                             float* __restrict__ rhs, int kchunk) {
    pdl_enter(F, us, vs, ws, rhs);
    const Column col(g, 1, 1, kchunk);
    if (col.i > g.nx || col.j > g.ny || col.k0 > g.nz) return;
    int id = gidx(g, col.i, col.j, col.k0);
    float wsc = __ldg(ws + id);
    const float rdt = __frcp_rn(g.dt);
    // (unrolled so that the loads of several planes are in flight together)
#pragma unroll 4
    for (int k = col.k0; k <= col.k1; ++k, id += g.plane) {
        const float wsp = __ldg(ws + id + g.plane);
        const float rho = rho_of(g, __ldg(F + id));
        rhs[id] = div_rn_pre(rho, g.dt, rdt) *
                  ((__ldg(us + id + 1) - __ldg(us + id)) * g.dxi +
                   (__ldg(vs + id + g.px) - __ldg(vs + id)) * g.dyi +
                   (wsp - wsc) * g.dzi);
        wsc = wsp;
    }
}

// The same with four cells per thread: quads of a row as in k_correct4 (one
// aligned float4 word; quads of a plane numbered flat, one plane per
// blockIdx.y), every operand an aligned float4 load -- F, u*, v* of the row
// and of the row above, w* of the plane and of the plane above -- and the
// u* east of the quad's last cell from the next lane, or from memory at the
// end of a warp or of a row.  k_rhs's expression and operand order per cell.
// One rho / dt for a quad of equal F.  Bound by DRAM and its latency: 34.5 us
// at 200^3 (4.6 TB/s), 223 at 400^3 (5.7).
__device__ __forceinline__ float4 ld4g(const float* __restrict__ a) {
    return __ldg(reinterpret_cast<const float4*>(a));
}
__device__ __forceinline__ float el4(const float4& v, int e) {
    return e == 0 ? v.x : (e == 1 ? v.y : (e == 2 ? v.z : v.w));
}

__global__ void __launch_bounds__(256) k_rhs4(Geom g, const float* __restrict__ F, const float* __restrict__ us,
                                              const float* __restrict__ vs, const float* __restrict__ ws,
                                              float* __restrict__ rhs) {
    const int nquad = g.nx / 4 + 1;  // quads covering columns 0 .. nx
    const int total = nquad * g.ny;
    const int qt = blockIdx.x * blockDim.x + threadIdx.x;
    const bool qa = qt < total;
    const int q = qa ? qt : total - 1;  // lanes past the end shadow the last quad
    const int jr = q / nquad, m = q - jr * nquad;
    const int j = jr + 1, k = blockIdx.y + 1, i0 = 4 * m;
    const int lane = threadIdx.x & 31;
    const bool lde = lane == 31 || m == nquad - 1;  // u* east of the quad from memory
    const int id = gidx(g, i0, j, k);  // a multiple of 4
    const float4 f4 = ld4g(F + id), u4 = ld4g(us + id), v4 = ld4g(vs + id), vn4 = ld4g(vs + id + g.px);
    const float4 w4 = ld4g(ws + id), wn4 = ld4g(ws + id + g.plane);
    const float ue_m = lde ? __ldg(us + id + 4) : 0.0f;
    float ue = __shfl_down_sync(0xffffffffu, u4.x, 1);
    if (lde) ue = ue_m;
    if (!qa) return;
    const float rdt = __frcp_rn(g.dt);
    float c[4], r[4];  // rho / dt
    c[0] = div_rn_pre(rho_of(g, f4.x), g.dt, rdt);
    const unsigned f0 = __float_as_uint(f4.x);
    if (((__float_as_uint(f4.y) ^ f0) | (__float_as_uint(f4.z) ^ f0) | (__float_as_uint(f4.w) ^ f0)) == 0) {
        c[1] = c[2] = c[3] = c[0];
    } else {
#pragma unroll
        for (int e = 1; e < 4; ++e) c[e] = div_rn_pre(rho_of(g, el4(f4, e)), g.dt, rdt);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float uip = e == 3 ? ue : el4(u4, e + 1);
        r[e] = c[e] * ((uip - el4(u4, e)) * g.dxi + (el4(vn4, e) - el4(v4, e)) * g.dyi +
                       (el4(wn4, e) - el4(w4, e)) * g.dzi);
    }
    if (i0 >= 1 && i0 + 3 <= g.nx) {
        *reinterpret_cast<float4*>(rhs + id) = make_float4(r[0], r[1], r[2], r[3]);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
        if (i0 + e >= 1 && i0 + e <= g.nx) rhs[id + e] = r[e];
}

// ---------------------------------------------------------------------------
// Velocity correction fused with the free-slip boundary conditions.
// update_{u,v,w}_kernel (voftrial1.cu:441-493) followed by apply_bc_velocity
// (voftrial1.cu:1107-1120, kernels :959-1051).  The three BC launches (j,
// then i, then k) compose to a closed form over the (nx+2)(ny+2)(nz+2) box,
// with c* an index clamped to the interior range and u_new the corrected
// face velocity:
//   u(i,j,k) = 0 for i == 1 or i == nx+1,  u_new(i, cj, ck) for 2 <= i <= nx,
//              u(0, cj, ck) (never updated) for i == 0
//   v(i,j,k) = 0 for j == 1 or j == ny+1,  v_new(ci, j, ck) for 2 <= j <= ny,
//              v(ci, 0, ck) for j == 0
//   w(i,j,k) = 0 for k == 1 or k == nz+1,  w_new(ci, cj, k) for 2 <= k <= nz,
//              w(ci, cj, 0) for k == 0
// The thread of interior cell (i,j,k) writes every box entry whose clamped
// source is its own, so each entry is written once and no thread reads an
// entry another thread writes.
//
// dt / r: faces between two pure cells have r in {rho_g, rho_l, (rho_g +
// rho_l)/2} (Geom::rpair); their IEEE quotients are formed once per context
// (Geom::qpair) and reused when r matches bit for bit.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float dt_over(const Geom& g, float r) {
    if (r == g.rpair[0]) return g.qpair[0];
    if (r == g.rpair[1]) return g.qpair[1];
    if (r == g.rpair[2]) return g.qpair[2];
    return g.dt / r;
}

__global__ void k_density_pairs(Geom g, float* out) {
    const float rg = rho_of(g, 0.0f), rl = rho_of(g, 1.0f);
    const float r0 = 0.5f * (rg + rg), r1 = 0.5f * (rl + rl), r2 = 0.5f * (rg + rl);
    out[0] = r0;
    out[1] = r1;
    out[2] = r2;
    out[3] = g.dt / r0;
    out[4] = g.dt / r1;
    out[5] = g.dt / r2;
}

struct EdgeDims {
    int nx, ny, nz, px, plane;
    __device__ int at(int i, int j, int k) const { return k * plane + j * px + i; }
};

// The boundary copies of a cell on the domain's edge.
__device__ __forceinline__ void store_edge_body(EdgeDims g, float* __restrict__ u, float* __restrict__ v,
                                                float* __restrict__ w, int i, int j, int k, float un, float vn,
                                                float wn) {
    int mi[3], mj[3], mk[3];
    const int nmi = mirrors(i, g.nx, mi), nmj = mirrors(j, g.ny, mj), nmk = mirrors(k, g.nz, mk);
    for (int b = 0; b < nmk; ++b)
        for (int a = 0; a < nmj; ++a) u[g.at(i, mj[a], mk[b])] = un;
    for (int b = 0; b < nmk; ++b)
        for (int a = 0; a < nmi; ++a) v[g.at(mi[a], j, mk[b])] = vn;
    for (int b = 0; b < nmj; ++b)
        for (int a = 0; a < nmi; ++a) w[g.at(mi[a], mj[b], k)] = wn;
    // far walls and the never-updated first planes
    if (i == g.nx)
        for (int b = 0; b < nmk; ++b)
            for (int a = 0; a < nmj; ++a) u[g.at(g.nx + 1, mj[a], mk[b])] = 0.0f;
    if (j == g.ny)
        for (int b = 0; b < nmk; ++b)
            for (int a = 0; a < nmi; ++a) v[g.at(mi[a], g.ny + 1, mk[b])] = 0.0f;
    if (k == g.nz)
        for (int b = 0; b < nmj; ++b)
            for (int a = 0; a < nmi; ++a) w[g.at(mi[a], mj[b], g.nz + 1)] = 0.0f;
    if (i == 1 && (nmj > 1 || nmk > 1)) {
        const float s0 = u[g.at(0, j, k)];
        for (int b = 0; b < nmk; ++b)
            for (int a = 0; a < nmj; ++a)
                if (a || b) u[g.at(0, mj[a], mk[b])] = s0;
    }
    if (j == 1 && (nmi > 1 || nmk > 1)) {
        const float s0 = v[g.at(i, 0, k)];
        for (int b = 0; b < nmk; ++b)
            for (int a = 0; a < nmi; ++a)
                if (a || b) v[g.at(mi[a], 0, mk[b])] = s0;
    }
    if (k == 1 && (nmi > 1 || nmj > 1)) {
        const float s0 = w[g.at(i, j, 0)];
        for (int b = 0; b < nmj; ++b)
            for (int a = 0; a < nmi; ++a)
                if (a || b) w[g.at(mi[a], mj[b], 0)] = s0;
    }
}

// The same out of line, for kernels that must not hold its registers.
static __device__ __noinline__ void store_edge(EdgeDims g, float* __restrict__ u, float* __restrict__ v,
                                               float* __restrict__ w, int i, int j, int k, float un, float vn,
                                               float wn) {
    store_edge_body(g, u, v, w, i, j, k, un, vn, wn);
}

// Writes the corrected face velocities of cell (i, j, k) and, on the domain
// edges, the boundary copies of apply_bc_velocity (voftrial1.cu:959-1051,
// 1107-1120) in closed form.  OUTLINE: the edge copies through a call.
template <bool OUTLINE>
__device__ __forceinline__ void store_corrected(const Geom& g, float* __restrict__ u, float* __restrict__ v,
                                                float* __restrict__ w, int i, int j, int k, int id, float un,
                                                float vn, float wn) {
    const bool edge_i = (i == 1 || i == g.nx), edge_j = (j == 1 || j == g.ny), edge_k = (k == 1 || k == g.nz);
    if (!(edge_i || edge_j || edge_k)) {  // bulk: one write per component
        u[id] = un;
        v[id] = vn;
        w[id] = wn;
        return;
    }
    const EdgeDims d{g.nx, g.ny, g.nz, g.px, g.plane};
    if (OUTLINE)
        store_edge(d, u, v, w, i, j, k, un, vn, wn);
    else
        store_edge_body(d, u, v, w, i, j, k, un, vn, wn);
}

__global__ void __launch_bounds__(256) k_correct(Geom g,
                                                 const float* __restrict__ F,
                                                 const float* __restrict__ us,
                                                 const float* __restrict__ vs,
                                                 const float* __restrict__ ws,
                                                 const float* __restrict__ p,
                                                 float* __restrict__ u, float* __restrict__ v,
                                                 float* __restrict__ w) {
    pdl_enter(F, us, vs, ws, p, u, v, w);
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z * blockDim.z + threadIdx.z + 1;
    if (i > g.nx || j > g.ny || k > g.nz) return;
    const int sy = g.px, sz = g.plane;
    const int id = gidx(g, i, j, k);
    const float rho_c = rho_of(g, __ldg(F + id));
    const float p_c = __ldg(p + id);
    float un = 0.0f, vn = 0.0f, wn = 0.0f;  // wall faces (i, j or k == 1) are 0
    if (i >= 2) {
        const float r = 0.5f * (rho_c + rho_of(g, __ldg(F + id - 1)));
        un = __ldg(us + id) - dt_over(g, r) * (p_c - __ldg(p + id - 1)) * g.dxi;
    }
    if (j >= 2) {
        const float r = 0.5f * (rho_c + rho_of(g, __ldg(F + id - sy)));
        vn = __ldg(vs + id) - dt_over(g, r) * (p_c - __ldg(p + id - sy)) * g.dyi;
    }
    if (k >= 2) {
        const float r = 0.5f * (rho_c + rho_of(g, __ldg(F + id - sz)));
        wn = __ldg(ws + id) - dt_over(g, r) * (p_c - __ldg(p + id - sz)) * g.dzi;
    }
    store_corrected<false>(g, u, v, w, i, j, k, id, un, vn, wn);
}

// The correction with four cells per thread: a quad i = 4m .. 4m+3 of a row
// (one aligned float4 word of the padded layout; px is a multiple of 32), the
// quads of all rows of a plane numbered flat so that 32 consecutive quads
// make a warp across row ends, one plane per blockIdx.y.  Every operand is an
// aligned float4 load (the cell, its y-1 and its z-1 neighbours of F and p;
// u*, v*, w*); the x-1 neighbour of the quad's first cell comes from the
// lane before (its last cell's density and pressure), or from memory at the
// start of a warp.  Each face keeps k_correct's expression and operand order
// (same bits).  Quads without an edge cell store float4 words; the others go
// through store_corrected cell by cell.
//
// Most quads lie in one phase: where the 13 values of F that enter are equal,
// one density and one quotient serve the 12 faces (47 M warp instructions at
// 200^3 without this, issue and latency together the bound; DRAM now: 69.7 ->
// 59.5 us at 200^3, 4.3 TB/s; 460 -> 385 at 400^3, 5.3 TB/s).
__global__ void __launch_bounds__(256, 4) k_correct4(Geom g, const float* __restrict__ F,
                                                  const float* __restrict__ us, const float* __restrict__ vs,
                                                  const float* __restrict__ ws, const float* __restrict__ p,
                                                  float* __restrict__ u, float* __restrict__ v,
                                                  float* __restrict__ w) {
    const int nquad = g.nx / 4 + 1;  // quads covering columns 0 .. nx
    const int total = nquad * g.ny;
    const int qt = blockIdx.x * blockDim.x + threadIdx.x;
    const bool qa = qt < total;
    const int q = qa ? qt : total - 1;  // lanes past the end shadow the last quad
    const int jr = q / nquad, m = q - jr * nquad;
    const int j = jr + 1, k = blockIdx.y + 1, i0 = 4 * m;
    const int lane = threadIdx.x & 31;
    const bool ldw = lane == 0 && m > 0;  // the x-1 neighbour from memory
    const int sy = g.px, sz = g.plane;
    const int id = gidx(g, i0, j, k);  // a multiple of 4
    const float4 fc = ld4g(F + id), fs = ld4g(F + id - sy), fb = ld4g(F + id - sz);
    const float4 pc = ld4g(p + id), ps = ld4g(p + id - sy), pb = ld4g(p + id - sz);
    const float4 u4 = ld4g(us + id), v4 = ld4g(vs + id), w4 = ld4g(ws + id);
    const float fl = ldw ? __ldg(F + id - 1) : 0.0f, pl = ldw ? __ldg(p + id - 1) : 0.0f;
    float fw = __shfl_up_sync(0xffffffffu, fc.w, 1), pw = __shfl_up_sync(0xffffffffu, pc.w, 1);
    if (ldw) {
        fw = fl;
        pw = pl;
    }
    if (m == 0) fw = fc.x;  // (enters no face)
    float qu[4], qv[4], qw[4];  // dt over the face densities
    const unsigned f0 = __float_as_uint(fc.x);
    unsigned differ = __float_as_uint(fw) ^ f0;
#pragma unroll
    for (int e = 0; e < 4; ++e)
        differ |= (__float_as_uint(el4(fc, e)) ^ f0) | (__float_as_uint(el4(fs, e)) ^ f0) |
                  (__float_as_uint(el4(fb, e)) ^ f0);
    if (differ == 0) {
        const float rho = rho_of(g, fc.x);
        const float q0 = dt_over(g, 0.5f * (rho + rho));
#pragma unroll
        for (int e = 0; e < 4; ++e) qu[e] = qv[e] = qw[e] = q0;
    } else {
        float rw = rho_of(g, fw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float rho_c = rho_of(g, el4(fc, e));
            qu[e] = dt_over(g, 0.5f * (rho_c + rw));
            qv[e] = dt_over(g, 0.5f * (rho_c + rho_of(g, el4(fs, e))));
            qw[e] = dt_over(g, 0.5f * (rho_c + rho_of(g, el4(fb, e))));
            rw = rho_c;
        }
    }
    float un[4], vn[4], wn[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float p_c = el4(pc, e);
        // wall faces (i, j or k == 1) are 0
        un[e] = i0 + e >= 2 ? el4(u4, e) - qu[e] * (p_c - (e == 0 ? pw : el4(pc, e - 1))) * g.dxi : 0.0f;
        vn[e] = j >= 2 ? el4(v4, e) - qv[e] * (p_c - el4(ps, e)) * g.dyi : 0.0f;
        wn[e] = k >= 2 ? el4(w4, e) - qw[e] * (p_c - el4(pb, e)) * g.dzi : 0.0f;
    }
    if (!qa) return;
    const bool bulk = i0 >= 2 && i0 + 3 <= g.nx - 1 && j != 1 && j != g.ny && k != 1 && k != g.nz;
    if (bulk) {
        *reinterpret_cast<float4*>(u + id) = make_float4(un[0], un[1], un[2], un[3]);
        *reinterpret_cast<float4*>(v + id) = make_float4(vn[0], vn[1], vn[2], vn[3]);
        *reinterpret_cast<float4*>(w + id) = make_float4(wn[0], wn[1], wn[2], wn[3]);
        return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int i = i0 + e;
        if (i >= 1 && i <= g.nx) store_corrected<true>(g, u, v, w, i, j, k, id + e, un[e], vn[e], wn[e]);
    }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
cudaError_t plain_configure() {
    cudaError_t e = jacobi_configure();
    if (e == cudaSuccess) e = jacobi_two_configure();
    return e == cudaSuccess ? jacobi_cluster_configure() : e;
}

cudaError_t plain_density_pairs(Geom* g) {
    float* d = nullptr;
    float h[6];
    cudaError_t e = cudaMalloc(&d, sizeof(h));
    if (e != cudaSuccess) return e;
    k_density_pairs<<<1, 1>>>(*g, d);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return e;
    for (int q = 0; q < 3; ++q) {
        g->rpair[q] = h[q];
        g->qpair[q] = h[3 + q];
    }
    return cudaSuccess;
}

cudaError_t plain_density_pairs_on(Geom* g, float* dev6, cudaStream_t s) {
    float h[6];
    k_density_pairs<<<1, 1, 0, s>>>(*g, dev6);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, dev6, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    for (int q = 0; q < 3; ++q) {
        g->rpair[q] = h[q];
        g->qpair[q] = h[3 + q];
    }
    return cudaSuccess;
}

bool plain_supported(const Geom& g) {
    return fct_supported(g.nx) && fct_supported(g.ny) && fct_supported(g.nz);
}

// How the sweeps are launched.  All in one (k_jacobi_cluster) on grids of some
// ten thousand cells; two per launch (k_jacobi_two), an odd count starting
// with one single sweep (k_jacobi_peel), on large ones (j2_chosen); between,
// one per launch.  VOF_JACOBI=peel / two force either (same bits).
enum class Sweeps { ONE, TWO, ALL };
static int jacobi_forced() {
    static int forced = -1;
    if (forced < 0) {
        const char* v = getenv("VOF_JACOBI");
        forced = !v ? 0 : !strcmp(v, "peel") ? 1 : !strcmp(v, "two") ? 2 : 0;
    }
    return forced;
}
static Sweeps jacobi_kind(const Geom& g, int iters) {
    const int forced = jacobi_forced();
    if (iters <= 2 || forced == 1) return Sweeps::ONE;
    if (forced != 2 && jacobi_cluster_fits(g, iters)) return Sweeps::ALL;
    return j2_chosen(g.nx, g.ny, g.nz, iters, forced) ? Sweeps::TWO : Sweeps::ONE;
}

cudaError_t plain_prepare(const Geom& g, int jacobi_iters, PlainBuffers* b, J2Tables* t, cudaStream_t s) {
    b->j2 = nullptr;
    if (!j2_chosen(g.nx, g.ny, g.nz, jacobi_iters, jacobi_forced())) return cudaSuccess;
    float* const field[4] = {b->p0, b->p1, b->p2, b->rhs};
    b->j2 = t;
    return jacobi_two_prepare(g, field, t, s);
}

static int jacobi_launches(const Geom& g, int iters) {
    const Sweeps q = jacobi_kind(g, iters);
    return q == Sweeps::ALL ? 1 : q == Sweeps::TWO ? (iters + 1) / 2 : iters;
}

int plain_kernels_per_step(const Geom& g, int jacobi_iters) {
    return 1 + (g.csf ? 1 : 0) + 1 + jacobi_launches(g, jacobi_iters) + 1 + 3;
}

// Column-marching launch shape: 32 x 8 columns per block, z split into
// chunks of about 16 planes (long enough to reuse the k-window, short enough
// for a few waves of blocks per SM).  On small grids the chunks shrink (down
// to one plane) until the launch has about 600 blocks: a launch of a few
// blocks marching 16 planes each is bound by the latency of its march.
static void column_launch(const Geom& g, dim3& grid, int& kchunk) {
    const int bx = (g.nx + TX - 1) / TX, by = (g.ny + TY - 1) / TY;
    const int target = (int)(((long long)g.nz * bx * by) / 600);
    const int len = target < 1 ? 1 : (target > 16 ? 16 : target);
    const int nch = (g.nz + len - 1) / len;
    kchunk = (g.nz + nch - 1) / nch;
    grid = dim3(bx, by, (g.nz + kchunk - 1) / kchunk);
}

// ev (optional, PLAIN_PHASES+1 events): ev[0] before the step, ev[q+1]
// after phase q (predict, rhs, pressure, correct, sweep 1, sweep 2, sweep 3).
static inline cudaError_t mark(cudaEvent_t* ev, int q, cudaStream_t s) {
    return ev ? cudaEventRecord(ev[q], s) : cudaSuccess;
}

// Four-cell kernels (k_rhs4, k_correct4) when their launch has at least
// about 7 blocks per SM of a B200 (measured: faster from 128^3 up, slower at
// 32^3 and 64^3, where the one-cell kernels' four times as many threads
// fill the GPU better).  VOF_RHS / VOF_CORRECT = 1 or 4 force either.
static bool quads_fill(const Geom& g) {
    const long long blocks = (long long)(((g.nx / 4 + 1) * g.ny + 255) / 256) * g.nz;
    return blocks >= 1024;
}
// SMs of the current device (queried once).
static int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) !=
                                                      cudaSuccess)
            n = 148;
    }
    return n;
}

// Planes per block of k_predict2 (and k_csf_curv): the least estimate of its
// time in planes of one resident block, waves of (kc + extra) planes each (extra
// for the first window) and part of a block for the uneven end.  Chunks as long as
// one wave allows left the SMs with fewer blocks than others idle at the end:
// (blocks of 256) 200^3 29 planes a block 76.8 us, 20 79.3, 16 73.0, 10 71.3,
// 8 (chosen) 71.7, 7 69.3, 4 72.5; 400^3 50 planes 507, 20 (chosen) 480, 16
// 482, 10 484, 7 495, 4 528; 128^3 8 planes 23.0, 4 (chosen) 22.2, 2 22.6.
static int march_kchunk(int nz, int bx, int wave, int extra) {
    int best = 1;
    double least = 1e30;
    for (int kc = 1; kc <= nz; ++kc) {
        const double waves = (double)bx * ((nz + kc - 1) / kc) / wave;
        const double cost = ((waves > 1.0 ? waves : 1.0) + 0.6) * (kc + extra);
        if (cost < least) {
            least = cost;
            best = kc;
        }
        if (waves < 0.5) break;
    }
    return best;
}

// 1: the one-cell kernel, 4: the four-cell kernel, else by size.
static int env_kernel(const char* name) {
    const char* v = getenv(name);
    return v ? atoi(v) : 0;
}

cudaError_t plain_front(const Geom& g, const PlainBuffers& b, cudaStream_t s, cudaEvent_t* ev) {
    const dim3 blk(TX, TY, 1);
    dim3 grid;
    int kchunk = 1;
    column_launch(g, grid, kchunk);
    cudaError_t e;
    if ((e = mark(ev, 0, s)) != cudaSuccess) return e;
    static int pforced = -1;  // VOF_PREDICT=1: k_predict (one cell per thread); else k_predict2
    if (pforced < 0) pforced = env_kernel("VOF_PREDICT");
    const int bx = ((g.nx / 2 + 1) * g.ny + 127) / 128;
    if (g.csf && b.csf[3]) {  // surface tension (extension): curvature, then face accelerations in the predictor
        const dim3 cg((g.nx + CSF_X - 3) / (CSF_X - 2), (g.ny + CSF_Y - 3) / (CSF_Y - 2));
        const int cc = march_kchunk(g.nz, cg.x * cg.y, 3 * sm_count(), 3);
        k_csf_curv<<<dim3(cg.x, cg.y, (g.nz + cc - 1) / cc), CSF_X * CSF_Y, 0, s>>>(g, b.F, b.csf[3], cc);
        const int kc = march_kchunk(g.nz, bx, 6 * sm_count(), 1);
        k_predict2<true, false><<<dim3(bx, (g.nz + kc - 1) / kc), 128, 0, s>>>(g, b.F, b.u, b.v, b.w, b.us, b.vs, b.ws, kc,
                                                                        b.csf[3]);
    } else if (pforced == 1) {
        k_predict<<<grid, blk, 0, s>>>(g, b.F, b.u, b.v, b.w, b.us, b.vs, b.ws, kchunk);
    } else {
        const int kc = march_kchunk(g.nz, bx, 8 * sm_count(), 1);
        const dim3 pg(bx, (g.nz + kc - 1) / kc);
        if (quads_fill(g))
            k_predict2<false, false><<<pg, 128, 0, s>>>(g, b.F, b.u, b.v, b.w, b.us, b.vs, b.ws, kc, nullptr);
        else
            pdl_launch(k_predict2<false, true>, pg, 128, 0, s, g, b.F, b.u, b.v, b.w, b.us, b.vs, b.ws, kc, nullptr);
    }
    if ((e = cudaGetLastError()) != cudaSuccess || (e = mark(ev, 1, s)) != cudaSuccess) return e;
    static int forced = -1;  // VOF_RHS=1: k_rhs (one cell per thread, z march), 4: k_rhs4
    if (forced < 0) forced = env_kernel("VOF_RHS");
    if (forced == 1 || (forced != 4 && !quads_fill(g))) {
        pdl_launch(k_rhs, grid, blk, 0, s, g, b.F, b.us, b.vs, b.ws, b.rhs, kchunk);
    } else {
        const int total = (g.nx / 4 + 1) * g.ny;
        k_rhs4<<<dim3((total + 255) / 256, g.nz), 256, 0, s>>>(g, b.F, b.us, b.vs, b.ws, b.rhs);
    }
    if ((e = cudaGetLastError()) != cudaSuccess || (e = mark(ev, 2, s)) != cudaSuccess) return e;
    return cudaSuccess;
}

// The correction: k_correct4 (four cells per thread) on large grids, else
// k_correct (one cell per thread).  Both give the same bits.
cudaError_t plain_correct(const Geom& g, const PlainBuffers& b, const float* p, cudaStream_t s) {
    static int forced = -1;
    if (forced < 0) forced = env_kernel("VOF_CORRECT");
    if (forced == 1 || (forced != 4 && !quads_fill(g))) {
        const dim3 cb(32, 4, 2);
        const dim3 cg((g.nx + 31) / 32, (g.ny + 3) / 4, (g.nz + 1) / 2);
        pdl_launch(k_correct, cg, cb, 0, s, g, b.F, b.us, b.vs, b.ws, p, b.u, b.v, b.w);
    } else {
        const int total = (g.nx / 4 + 1) * g.ny;
        k_correct4<<<dim3((total + 255) / 256, g.nz), 256, 0, s>>>(g, b.F, b.us, b.vs, b.ws, p, b.u, b.v, b.w);
    }
    return cudaGetLastError();
}

cudaError_t plain_back(const Geom& g, const PlainBuffers& b, int istep, const float* p, cudaStream_t s,
                       cudaEvent_t* ev) {
    cudaError_t e;
    if ((e = mark(ev, 3, s)) != cudaSuccess) return e;
    if ((e = plain_correct(g, b, p, s)) != cudaSuccess || (e = mark(ev, 4, s)) != cudaSuccess) return e;

    // Sweep order by istep % 3 (voftrial1.cu:1384-1396).  The sweeps run out
    // of place, F -> s1 -> s2 -> F, through the two pressure buffers that do
    // not hold the pressure: the next step's solve writes their interiors
    // before it reads them, and their ghost cells (never written by a sweep or
    // a Jacobi launch) hold finite values, which a sweep reads only through
    // the zero velocity of a wall face.
    const int r = ((istep % 3) + 3) % 3;
    static const int order[3][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}};
    float* s1 = (p == b.p0) ? b.p1 : b.p0;
    float* s2 = b.p2;
    const float* src[3] = {b.F, s1, s2};
    float* dst[3] = {s1, s2, b.F};
    for (int q = 0; q < 3; ++q) {
        const int axis = order[r][q];
        const float* vel = axis == 0 ? b.u : (axis == 1 ? b.v : b.w);
        if ((e = fct_launch_to(g, axis, q == 2, src[q], dst[q], vel, s)) != cudaSuccess || (e = mark(ev, 5 + q, s)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t plain_pressure(const Geom& g, const PlainBuffers& b, int jacobi_iters, int* p_parity, cudaStream_t s) {
    cudaError_t e;

    // Jacobi (voftrial1.cu:1371-1375).  The reference ping-pongs p <-> pt once
    // per sweep, so after N sweeps its pressure sits in the buffer it started
    // in when N is even and in the other one when N is odd; the launches end in
    // that same buffer (which keeps the reference's ghost entries in a
    // download), through the scratch buffer first when their number is of the
    // other parity.
    float* pbuf[3] = {b.p0, b.p1, b.p2};
    const int src = *p_parity, dst = src ^ (jacobi_iters & 1);
    int cur = src;
    const Sweeps kind = jacobi_kind(g, jacobi_iters);
    if (kind == Sweeps::ALL) {
        if ((e = jacobi_cluster_launch(g, pbuf, src, b.rhs, jacobi_iters, s)) != cudaSuccess) return e;
    } else if (kind == Sweeps::TWO) {
        if (!b.j2) return cudaErrorInvalidValue;
        const int L = jacobi_launches(g, jacobi_iters);
        const bool detour = (L & 1) != (src != dst);
        for (int q = 0; q < L; ++q) {
            const int left = L - 1 - q;  // launches after this one, each between the two buffers
            const int to = detour && q == 0 ? 2 : dst ^ (left & 1);
            if (q == 0 && (jacobi_iters & 1))
                e = jacobi_peel_launch(g, pbuf[cur], b.rhs, pbuf[to], s);
            else
                e = jacobi_two_launch(g, *b.j2, cur, pbuf[cur], pbuf[to], b.status, s);
            if (e != cudaSuccess) return e;
            cur = to;
        }
    } else {
        for (int it = 0; it < jacobi_iters; ++it, cur ^= 1)
            if ((e = jacobi_peel_launch(g, pbuf[cur], b.rhs, pbuf[cur ^ 1], s)) != cudaSuccess) return e;
    }
    *p_parity = dst;
    return cudaSuccess;
}

cudaError_t plain_step(const Geom& g, const PlainBuffers& b, int istep, int jacobi_iters,
                       int* p_parity, cudaStream_t s, cudaEvent_t* ev) {
    cudaError_t e = plain_front(g, b, s, ev);
    if (e != cudaSuccess) return e;
    if ((e = plain_pressure(g, b, jacobi_iters, p_parity, s)) != cudaSuccess) return e;
    float* pbuf[3] = {b.p0, b.p1, b.p2};
    return plain_back(g, b, istep, pbuf[*p_parity], s, ev);
}

int plain_phase_launches(const Geom& g, int phase, int jacobi_iters) {
    if (phase == PHASE_JACOBI) return jacobi_launches(g, jacobi_iters);
    return (phase == PHASE_PREDICT && g.csf) ? 2 : 1;
}

}  // namespace vof
