// fct_sweep.cu -- one directionally split FCT sweep of the volume fraction
// (fct_{x,y,z}_sweep_stage1..4, voftrial1.cu:509-905) as a single kernel.
//
// Compiled with -fmad=false like plain_step.cu: every expression below keeps
// the reference's operand order and no multiply-add is contracted.
//
// Why the four reference stages collapse into one pass over a grid line.
// Stage 2 of a sweep zeroes the other direction's antidiffusive fluxes
// (voftrial1.cu:573-574, 712-713), so the terms they contribute to pp, pm and
// the stage-4 update vanish (exactly, up to the sign of a zero, which the
// final clamp01f removes).  What is left couples only cells of the same line
// along the sweep axis, with a reach of three cells.  The zero-filled buffers
// the reference never writes (voftrial1.cu:1200-1203) fix the line ends:
//   Ftd at the two ghost cells is 0, rp and rm at the ghost cells are 0, and
//   the limiter c of the first face (c[1]) is 0; the wall-face velocities
//   are 0 after apply_bc_velocity, so the ghost F values enter only as 0*F.
//
// The per-cell expressions (and the reference's length factors per sweep)
// are in fct_line.cuh, shared with the sweep adjoint.
//
// The sweeps run out of place: a block reads F beyond what it writes.
#include "fct_sweep.h"

#include "fct_line.cuh"
#include "pdl.cuh"

namespace vof {

#if defined(__CUDA_ARCH__) && !defined(VOF_FMAD_FALSE)
#error "fct_sweep.cu must be compiled with -fmad=false -DVOF_FMAD_FALSE"
#endif

namespace {

using fct::Sweep;
using fct::face_limit;
using fct::ftd_from;
using fct::limiter;

// Indices whose clamped value is x on an axis of n interior cells: x itself,
// plus the ghost 0 when x == 1 and the ghost n+1 when x == n.
__device__ __forceinline__ int mirrors(int x, int n, int* out) {
    out[0] = x;  // fixed positions (no runtime index)
    out[1] = (x == 1) ? 0 : n + 1;
    out[2] = n + 1;
    return 1 + (x == 1) + (x == n);
}

// apply_bc_F (voftrial1.cu:1122-1135) for one cell of the final sweep: the
// cell (i, j, k) and every ghost whose clamped interior index is (i, j, k)
// take f.  Out of line: only cells on the domain's edge come here, and inlined
// it would hold registers in every thread of the marching kernels.
__device__ __noinline__ void store_mirrored(float* __restrict__ F, int px, int plane, int nx, int ny, int nz, int i,
                                            int j, int k, float f) {
    int iv[3], jv[3], kv[3];
    const int ni = mirrors(i, nx, iv), nj = mirrors(j, ny, jv), nk = mirrors(k, nz, kv);
    for (int c = 0; c < nk; ++c)
        for (int b = 0; b < nj; ++b)
            for (int a = 0; a < ni; ++a) F[kv[c] * plane + jv[b] * px + iv[a]] = f;
}

// The ghost copies of the cell at index o whose value is f, in line: dx, dy, dz
// lead to the copy beyond the wall that the cell is at along each axis (0: at
// none).  For boxes of more than one cell along every axis.
__device__ __forceinline__ void store_ghosts(float* __restrict__ F, int o, int dx, int dy, int dz, float f) {
    if (dx) F[o + dx] = f;
    if (dy) {
        F[o + dy] = f;
        if (dx) F[o + dy + dx] = f;
    }
    if (dz) {
        F[o + dz] = f;
        if (dx) F[o + dz + dx] = f;
        if (dy) {
            F[o + dz + dy] = f;
            if (dx) F[o + dz + dy + dx] = f;
        }
    }
}
// Offset to the copy beyond the wall of cell c of n, cells `stride` apart.
__device__ __forceinline__ int beyond(int c, int n, int stride) { return c == 1 ? -stride : (c == n ? stride : 0); }
__device__ __forceinline__ bool thin(const Geom& g) { return g.nx == 1 || g.ny == 1 || g.nz == 1; }

}  // namespace

// ---- one thread per position: small grids ------------------------------------
// A block owns LPB lines over their full length, a thread one position of one
// line (the cell q and the face below it); the stages run one after another
// with a barrier between, a neighbour's stage values coming from shared
// memory.  What bounds it is latency: two loads, four barriers and two chains
// of divisions, 3 us at 32^3 and 4.2 us at 64^3 with the launch (a march along
// each line, the earlier shape, 7.9 and 11.8: some ten dependent cells and a
// warm-up of eight evaluations per warp).
template <int AXIS, bool FINAL>
__global__ void __launch_bounds__(1024) k_fct_lines(Geom g, const float* __restrict__ Fsrc,
                                                    float* __restrict__ F, const float* __restrict__ vel, int lpb) {
    pdl_enter(Fsrc, F, vel);
    extern __shared__ float smem[];
    const Sweep<AXIS> S(g);
    const int n = S.n, npos = n + 2;
    const int na = AXIS == 0 ? g.ny : g.nx, nb = AXIS == 2 ? g.ny : g.nz;
    // x lines: positions across lanes; y and z lines: lines across lanes
    const int t = threadIdx.x;
    const int l = AXIS == 0 ? t / npos : t % lpb, q = AXIS == 0 ? t - l * npos : t / lpb;
    const int line = blockIdx.x * lpb + l;
    const int a = 1 + line % na, b = 1 + line / na;
    const bool live = l < lpb && q < npos && b <= nb;
    const int qs = AXIS == 0 ? 1 : lpb;  // neighbouring positions in shared memory
    const int tile = npos * lpb, at = AXIS == 0 ? l * npos + q : q * lpb + l;
    float* sF = smem + at;
    float* sV = sF + tile;
    float* sL = sV + tile;  // low-order flux of the face below, later rp
    float* sA = sL + tile;  // antidiffusive flux of the face below
    float* sT = sA + tile;
    float* sM = sT + tile;  // rm
    const int id = AXIS == 0 ? gidx(g, q, a, b) : (AXIS == 1 ? gidx(g, a, q, b) : gidx(g, a, b, q));
    float Fq = 0.0f, Vq = 0.0f;
    if (live) {
        Fq = __ldg(Fsrc + id);
        Vq = __ldg(vel + id);
        sF[0] = Fq;
        sV[0] = Vq;
    }
    // Where F is 0 at c-3 .. c+3 and every |face velocity| < vq (which keeps
    // every dv above 0.01 vol), every stage value is zero up to its sign, which
    // no comparison sees and the final clamp01f removes: a block of zeros ends here.
    const float vq = 0.49f * S.vol / S.dvfac;
    const bool quiet = __syncthreads_and(!live || (Fq == 0.0f && fabsf(Vq) < vq));
    const bool cell = live && q >= 1 && q <= n;
    float fnew = 0.0f;
    if (!quiet) {
        float lo = 0.0f, af = 0.0f, dv = 1.0f, rdv = 1.0f;
        if (live && q >= 1) fct::flux(Vq, sF[-qs], Fq, S.dt, lo, af);
        if (cell) {
            dv = S.dv(Vq, sV[qs]);
            rdv = __frcp_rn(dv);
        }
        if (live) {
            sL[0] = lo;
            sA[0] = af;
        }
        __syncthreads();
        float T = 0.0f;
        if (cell) T = ftd_from(S, Fq, lo, sL[qs], dv, rdv);
        if (live) sT[0] = T;
        __syncthreads();
        float rp = 0.0f, rm = 0.0f, an = 0.0f;
        if (cell) {
            an = sA[qs];
            limiter(S, sT[-qs], T, sT[qs], af, an, rp, rm);
        }
        if (live) {
            sL[0] = rp;
            sM[0] = rm;
        }
        __syncthreads();
        if (cell) {
            const float cl = q == 1 ? 0.0f : face_limit(af, sL[-qs], sM[-qs], rp, rm);  // (c[1] is never written)
            const float ch = face_limit(an, rp, rm, sL[qs], sM[qs]);
            fnew = clamp01f(fct::stage4(S, T, af, cl, an, ch, dv, rdv));
        }
    }
    if (!cell) return;
    if (!FINAL) {
        F[id] = fnew;
        return;
    }
    fnew = clamp01f(fnew);  // post_process_f_kernel, voftrial1.cu:502-507
    const int i = AXIS == 0 ? q : a, j = AXIS == 0 ? a : (AXIS == 1 ? q : b), k = AXIS == 2 ? q : b;
    if (i > 1 && i < g.nx && j > 1 && j < g.ny && k > 1 && k < g.nz)
        F[id] = fnew;
    else  // apply_bc_F (voftrial1.cu:1122-1135)
        store_mirrored(F, g.px, g.plane, g.nx, g.ny, g.nz, i, j, k, fnew);
}

// ---- several positions per thread: large grids ---------------------------------
// The stages of k_fct_lines on a tile of 256 M positions, M per thread, so
// that a thread has 2 M loads in flight.  Lines along y or z: 32 lines (lanes)
// by 8 M positions; a value is exact wherever its three-cell reach stays
// inside the tile, so a tile writes all but its three outermost positions, and
// consecutive tiles of a line overlap by six.  Lines along x: as many whole
// rows as fit, their positions numbered flat.  A tile of zeros (most of a dam
// break is gas) ends after its loads.  Fin and Fout must be different buffers.
// Measured on a B200 (per sweep, y / z / x lines, with the earlier kernels, a
// march of one thread per line segment and a warp per window of a row):
// 200^3 from rest 32 / 36 / 34 us (44 / 45 / 39), 201 x 157 x 93 in flow 14 /
// 16 / 15 (29 / 33 / 17), 128^3 10 / 12 / 15 (22 / 23 / 18), 400^3 243 / 269 /
// 298 (293 / 299 / 306).  Where there is liquid it is bound by instruction
// issue (six quotients a cell), in gas by its loads.
constexpr int FT_THREADS = 256;

template <int AXIS, bool FINAL, int M>
__global__ void __launch_bounds__(FT_THREADS) k_fct_tile(Geom g, const float* __restrict__ Fin, float* __restrict__ F,
                                                         const float* __restrict__ vel, int seg) {
    constexpr int TILE = M * FT_THREADS, NS = AXIS == 0 ? 1 : 32;  // neighbouring positions in shared memory
    __shared__ float sF[TILE], sV[TILE], sL[TILE], sA[TILE];
    const Sweep<AXIS> S(g);
    const int n = S.n, tid = threadIdx.x;
    // position q[m] of a line and its index in the field; cells c0 .. c1 are written
    int q[M], id[M];
    bool in[M];
    int c0 = 1, c1 = n;
    int da[M], db[M];  // final sweep: offsets across the line to its ghost copies
    if (AXIS == 0) {  // seg: rows per tile
        const int npos = n + 2, step = FT_THREADS / npos, rest = FT_THREADS - step * npos;
        int r = tid / npos, p = tid - r * npos;
        const int line = blockIdx.x * seg + r;
        int k = line / g.ny, j = line - k * g.ny;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            q[m] = p;
            in[m] = r < seg && k < g.nz;
            id[m] = gidx(g, p, j + 1, k + 1);
            da[m] = beyond(j + 1, g.ny, g.px);
            db[m] = beyond(k + 1, g.nz, g.plane);
            p += rest;
            const int more = step + (p >= npos);
            p -= p >= npos ? npos : 0;
            r += more;
            j += more;
            while (j >= g.ny) {
                j -= g.ny;
                ++k;
            }
        }
    } else {  // seg: cells written per tile and line
        const int nb = AXIS == 1 ? g.nz : g.ny, line = blockIdx.x * 32 + (tid & 31);
        const int a = 1 + line % g.nx, b = 1 + line / g.nx;
        const int qs = AXIS == 1 ? g.px : g.plane, base = AXIS == 1 ? gidx(g, a, 0, b) : gidx(g, a, b, 0);
        c0 = 1 + blockIdx.y * seg;
        c1 = min(n, c0 + seg - 1);
#pragma unroll
        for (int m = 0; m < M; ++m) {
            q[m] = c0 - 3 + (tid >> 5) + m * (FT_THREADS / 32);
            in[m] = b <= nb && q[m] >= 0 && q[m] <= n + 1 && q[m] <= c1 + 3;
            id[m] = base + q[m] * qs;
            da[m] = beyond(a, g.nx, 1);
            db[m] = beyond(b, nb, AXIS == 1 ? g.plane : g.px);
        }
    }
    float Fq[M], Vq[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
        Fq[m] = in[m] ? __ldg(Fin + id[m]) : 0.0f;
        Vq[m] = in[m] ? __ldg(vel + id[m]) : 0.0f;
    }
    const float vq = 0.49f * S.vol / S.dvfac;
    bool zero = true;
#pragma unroll
    for (int m = 0; m < M; ++m) zero = zero && Fq[m] == 0.0f && fabsf(Vq[m]) < vq;
    const bool quiet = __syncthreads_and(zero);
    float out[M];
#pragma unroll
    for (int m = 0; m < M; ++m) out[m] = 0.0f;
    if (!quiet) {
        // (a cell's upper neighbour, a face's lower one: inside the tile)
        auto face = [&](int m) { return in[m] && q[m] >= 1 && (AXIS == 0 || tid + m * FT_THREADS >= NS); };
        auto cell = [&](int m) {
            return in[m] && q[m] >= 1 && q[m] <= n && (AXIS == 0 || tid + m * FT_THREADS < TILE - NS);
        };
#pragma unroll
        for (int m = 0; m < M; ++m) {
            sF[tid + m * FT_THREADS] = Fq[m];
            sV[tid + m * FT_THREADS] = Vq[m];
        }
        __syncthreads();
        float lo[M], af[M], dv[M], T[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int x = tid + m * FT_THREADS;
            lo[m] = af[m] = 0.0f;
            dv[m] = 1.0f;
            if (face(m)) fct::flux(Vq[m], sF[x - NS], Fq[m], S.dt, lo[m], af[m]);
            if (cell(m)) dv[m] = S.dv(Vq[m], sV[x + NS]);
            sL[x] = lo[m];
            sA[x] = af[m];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int x = tid + m * FT_THREADS;
            T[m] = 0.0f;
            if (cell(m)) T[m] = ftd_from(S, Fq[m], lo[m], sL[x + NS], dv[m], __frcp_rn(dv[m]));
            sF[x] = T[m];
        }
        __syncthreads();
        float rp[M], rm[M];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int x = tid + m * FT_THREADS;
            rp[m] = rm[m] = 0.0f;
            if (face(m) && cell(m)) limiter(S, sF[x - NS], T[m], sF[x + NS], af[m], sA[x + NS], rp[m], rm[m]);
            sL[x] = rp[m];
            sV[x] = rm[m];
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int x = tid + m * FT_THREADS;
            if (!in[m] || q[m] < c0 || q[m] > c1) continue;
            const float an = sA[x + NS];
            const float cl = q[m] == 1 ? 0.0f : face_limit(af[m], sL[x - NS], sV[x - NS], rp[m], rm[m]);
            const float ch = face_limit(an, rp[m], rm[m], sL[x + NS], sV[x + NS]);
            out[m] = clamp01f(fct::stage4(S, T[m], af[m], cl, an, ch, dv[m], __frcp_rn(dv[m])));
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
        if (FINAL) out[m] = clamp01f(out[m]);  // post_process_f_kernel, voftrial1.cu:502-507
        in[m] = in[m] && q[m] >= c0 && q[m] <= c1;
        if (in[m]) F[id[m]] = out[m];
    }
    if (!FINAL) return;
    // apply_bc_F (voftrial1.cu:1122-1135): the ghost copies of the box's outer cells
    const int qs = AXIS == 0 ? 1 : (AXIS == 1 ? g.px : g.plane);
    if (thin(g)) {
#pragma unroll 1
        for (int m = 0; m < M; ++m) {
            // (no runtime index: the arrays stay in registers)
            int o = 0;
            bool w = false;
            float f = 0.0f;
#pragma unroll
            for (int u = 0; u < M; ++u)
                if (u == m) {
                    o = id[u];
                    w = in[u];
                    f = out[u];
                }
            const int k = o / g.plane, r = o - k * g.plane, j = r / g.px;
            if (w) store_mirrored(F, g.px, g.plane, g.nx, g.ny, g.nz, r - j * g.px, j, k, f);
        }
        return;
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (in[m]) store_ghosts(F, id[m], beyond(q[m], n, qs), da[m], db[m], out[m]);
}

// Lines per block of k_fct_lines (0: the line is too long for it): up to 32,
// fewer while the launch has under four blocks per SM.
static int lines_per_block(int n, long long lines) {
    int lpb = 32;
    while (lpb > 4 && (lpb * (n + 2) > 1024 || lines < 592LL * lpb)) lpb >>= 1;
    return lpb * (n + 2) <= 1024 ? lpb : 0;
}

// The extents a sweep takes: a line of n cells of 32 lines, twice, in the
// shared memory of a block (the limit vof_create has always checked; the
// kernels above take rows of up to 1534 cells).
bool fct_supported(int n) { return 2u * 32u * sizeof(float) * (size_t)((n + 2) | 1) <= 227u * 1024u; }

template <int AXIS, bool FINAL, int M>
static void launch_tile(const Geom& g, long long lines, const float* Fin, float* F, const float* vel, cudaStream_t s) {
    const int n = AXIS == 0 ? g.nx : (AXIS == 1 ? g.ny : g.nz);
    if (AXIS == 0) {
        const int rows = M * FT_THREADS / (n + 2);
        k_fct_tile<AXIS, FINAL, M><<<(unsigned)((lines + rows - 1) / rows), FT_THREADS, 0, s>>>(g, Fin, F, vel, rows);
    } else {
        const int most = M * FT_THREADS / 32 - 6, nseg = (n + most - 1) / most;
        const dim3 grid((unsigned)((lines + 31) / 32), nseg);
        k_fct_tile<AXIS, FINAL, M><<<grid, FT_THREADS, 0, s>>>(g, Fin, F, vel, (n + nseg - 1) / nseg);
    }
}

template <int AXIS, bool FINAL>
static cudaError_t launch_axis(const Geom& g, const float* Fin, float* F, const float* vel, cudaStream_t s) {
    const int n = AXIS == 0 ? g.nx : (AXIS == 1 ? g.ny : g.nz);
    const long long cells = (long long)g.nx * g.ny * g.nz, lines = cells / n;
    // one position per thread up to 2^19 cells (64^3: 4.4 us a y sweep, the
    // tiles 5.8; 100 x 80 x 126: 10.2 and 6.9)
    const int lpb = lines_per_block(n, lines);
    if (lpb && cells <= 1 << 19) {
        return pdl_launch(k_fct_lines<AXIS, FINAL>, (unsigned)((lines + lpb - 1) / lpb),
                          (lpb * (n + 2) + 31) / 32 * 32, 6 * lpb * (n + 2) * (int)sizeof(float), s, g, Fin, F, vel,
                          lpb);
    }
    if (AXIS != 0) {
        // positions per thread: 4, from 2^25 cells 6 (less overlap: 400^3, z
        // lines, 269 us against 278; 128^3 13.3 against 11.8)
        if (cells >= 1 << 25)
            launch_tile<AXIS, FINAL, 6>(g, lines, Fin, F, vel, s);
        else
            launch_tile<AXIS, FINAL, 4>(g, lines, Fin, F, vel, s);
        return cudaGetLastError();
    }
    // x lines: 4 positions per thread, or the count that whole rows fill 8 % better
    int best = 4;
    for (int m = 5; m <= 6; ++m)
        if (100 * best * (m * FT_THREADS / (n + 2)) > 108 * m * (best * FT_THREADS / (n + 2))) best = m;
    if (best == 4)
        launch_tile<AXIS, FINAL, 4>(g, lines, Fin, F, vel, s);
    else if (best == 5)
        launch_tile<AXIS, FINAL, 5>(g, lines, Fin, F, vel, s);
    else
        launch_tile<AXIS, FINAL, 6>(g, lines, Fin, F, vel, s);
    return cudaGetLastError();
}

cudaError_t fct_launch_to(const Geom& g, int axis, bool final_sweep, const float* Fin, float* Fout, const float* vel,
                          cudaStream_t s) {
    if (axis == 0)
        return final_sweep ? launch_axis<0, true>(g, Fin, Fout, vel, s) : launch_axis<0, false>(g, Fin, Fout, vel, s);
    if (axis == 1)
        return final_sweep ? launch_axis<1, true>(g, Fin, Fout, vel, s) : launch_axis<1, false>(g, Fin, Fout, vel, s);
    return final_sweep ? launch_axis<2, true>(g, Fin, Fout, vel, s) : launch_axis<2, false>(g, Fin, Fout, vel, s);
}

}  // namespace vof
