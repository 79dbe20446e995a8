// bs_mg.cu -- aggregation multigrid preconditioner for the PPE BiCGStab.
//
// The reference solves the Jacobi-scaled PPE with unpreconditioned FGMRES /
// BiCGStab (solver.f90:129-350); the iteration count then grows with the
// number of particles across the domain.  This multigrid cycle is applied as
// a right preconditioner; the Krylov recurrence, dots and the stopping test
// stay FP64, so the converged pressure is the solution of the same FP64
// system.
//
// Level 0: particle rows (the sliced-ELL PPE).  Level 1: one aggregate per
// half-cell -- the four 2h x 2h quadrants of a search cell (~7 rows each).
// The rows of a cell are contiguous, so the Galerkin product P^T A P
// (P = half-cell indicator) is a warp reduction per cell, and because every
// neighbour lies within 2h the coarse operator is a 9-point stencil on the
// half-cell grid.  Level 2: the cells; level l+1: 2x2 boxes of level l,
// again 9-point Galerkin stencils.  Smoother: damped Jacobi, one pre-sweep
// from zero and one post-sweep; coarse corrections scaled by cscale (over-
// correction for the piecewise-constant prolongation); levels 1..wlev visit
// the next level twice (the second time on the updated residual), so the
// cycle is a W-cycle at the top and a V-cycle below; coarsest level: Jacobi
// sweeps by one block per scene.  Every scene coarsens on its own, so its
// cycle is the same alone and inside a batch.  The particle-level kernels
// skip converged scenes.  T = double (FP64 mode) or float (mixed mode, FP32
// cycle).
#include <cstring>

#include "bs_internal.cuh"

using namespace bs;

namespace {

// A scene whose cycle output nobody reads: converged, or (fg: inside FGMRES)
// its restart cycle has ended and waits for the other scenes'
__device__ __forceinline__ bool mg_skip(const Dev& D, int s, int fg) {
    return D.dyn[s].converged != 0 || (fg && D.dyn[s].fg_state != 0);
}

// ------------------------------------------------------------ setup
// level 0: 1/adiag per row, and the row's half-cell (quadrant of its cell,
// split at the cell's mid-lines as the quadrant search does, search.f90:328)
template <typename T>
__global__ void k_mg_dinv0(Dev D) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const ScenePar& P = D.par[s];
    if (r >= P.row0 + D.dyn[s].n) return;
    const double d = D.adiag[r];
    ((T*)D.mg.dinv0)[r] = (d != 0.0 && isfinite(d)) ? (T)(1.0 / d) : (T)0;
    ((T*)D.mg.adiagT)[r] = (T)d;
    const int lc = D.cell[r] - P.cell0;
    const int i0 = lc % P.celly, j0 = lc / P.celly;
    const double xl = cell_xleft(P, j0 + 1), xr = cell_xright(P, j0 + 1);
    const double yb = cell_ybot(P, i0 + 1), yt = cell_ytop(P, i0 + 1);
    const int lower = D.y[r] <= yb + fabs((yt - yb) / 2.0);
    const int right = D.x[r] > xl + fabs((xl - xr) / 2.0);
    D.mg.sub[r] = (uint8_t)(lower | (right << 1));
    D.mg.agg1[r] = D.mg.off[1][s] + (2 * j0 + right) * (2 * P.celly) + 2 * i0 + lower;
}

// level 1 = P^T A0 P over the half-cells: one warp per cell, a lane per row
// accumulating the row's 9 stencil entries, then one masked warp reduction
// per (half-cell, entry); lane m keeps entry m and m+32 of the 36 results.
// An offset beyond one half-cell (a pair split by rounding at a mid-line)
// is clamped into the stencil.  Sums in the level's type T (FP32 in the
// mixed form, from the FP32 copy of the matrix); the neighbour's cell column
// offset (-1, 0, 1) from two comparisons instead of an integer division.
// Bound by the latency of a neighbour's chain (index, then its cell): four at once,
// with k_mg_dinv0 30 and 23 us at 15 k rows, 216 and 153 at 712 k, before and now.
template <typename T>
__global__ void k_mg_gal0(Dev D) {
    BS_PDL_ENTRY();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (c >= D.ncell_total) return;
    const int s = D.cell_scene[c];
    const ScenePar& P = D.par[s];
    if (c - P.cell0 >= P.ncell) return;   // reserved cells beyond the scene's current grid
    const int celly = P.celly;
    const int r0 = D.cell_start[c], r1 = D.cell_end[c];
    const T* A = (const T*)(sizeof(T) == 8 ? D.aval : (void*)D.aval32);
    const uint8_t* sub = D.mg.sub;
    constexpr int B = 4;   // neighbours loaded at once
    T mine0 = 0, mine1 = 0;
    for (int base = r0; base < r1; base += 32) {
        const int r = base + lane;
        T acc[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k] = 0;
        int sb = -1;
        if (r < r1) {
            sb = sub[r];
            const int si = sb & 1, sj = sb >> 1;
            acc[4] += (T)D.adiag[r];
            const int n = D.ncount[r];
            for (int k0 = 0; k0 < n; k0 += B) {
                int cols[B], cells[B], subs[B];
                T vs[B];
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    const long e = ell(r, min(k0 + m, n - 1), D.kmax);
                    cols[m] = D.nidx[e];
                    vs[m] = A[e];
                }
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    cells[m] = D.cell[cols[m]];
                    subs[m] = sub[cols[m]];
                }
#pragma unroll
                for (int m = 0; m < B; ++m) {
                    const int d = cells[m] - c;
                    const int u = d + celly + 1;   // in [0, 2 celly + 2] for the 3x3 neighbour cells
                    const int dj = (u >= 2 * celly) ? 1 : ((u >= celly) ? 0 : -1);
                    const int di = d - dj * celly;
                    const int s2 = subs[m];
                    const int dI = min(max(2 * di + (s2 & 1) - si, -1), 1);
                    const int dJ = min(max(2 * dj + (s2 >> 1) - sj, -1), 1);
                    const int q = (dJ + 1) * 3 + (dI + 1);
#pragma unroll
                    for (int t = 0; t < 9; ++t)
                        if (t == q && k0 + m < n) acc[t] += vs[m];
                }
            }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                T v = (sb == t) ? acc[k] : (T)0;
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                const int m = t * 9 + k;
                if (m < 32) { if (lane == m) mine0 += v; }
                else if (lane == m - 32) mine1 += v;
            }
    }
    T* Al = (T*)D.mg.A[1];
    T* dl = (T*)D.mg.dinv[1];
    const int n1 = D.mg.n[1];
    const int lc = c - P.cell0;
    const int i0 = lc % celly, j0 = lc / celly;
    const int o1 = D.mg.off[1][s], ny1 = 2 * celly;
    auto put = [&](int m, T v) {
        const int t = m / 9, k = m - 9 * (m / 9);
        const int Q = o1 + (2 * j0 + (t >> 1)) * ny1 + 2 * i0 + (t & 1);
        Al[(long)k * n1 + Q] = v;
        if (k == 4) dl[Q] = (v != (T)0 && isfinite(v)) ? (T)1 / v : (T)0;
    };
    put(lane, mine0);
    if (lane < 4) put(lane + 32, mine1);
}

// level l+1 from level l: one thread per coarse cell
template <typename T>
__global__ void k_mg_galc(Dev D, int l) {
    BS_PDL_ENTRY();
    const int Q = blockIdx.x * blockDim.x + threadIdx.x;
    const MgDev& M = D.mg;
    if (Q >= M.n[l + 1]) return;
    const int s = M.scene_of[l + 1][Q];
    const int q = Q - M.off[l + 1][s];
    const int nyc = M.ny[l + 1][s];
    if (q >= nyc * M.nx[l + 1][s]) return;   // reserved beyond the scene's current grid
    const int I = q % nyc, J = q / nyc;
    const int nyf = M.ny[l][s], nxf = M.nx[l][s], fo = M.off[l][s];
    const T* Af = (const T*)M.A[l];
    const int nf = M.n[l];
    // the four children's stencils, all loads before the sums; entry k of child
    // (a, b) falls on one entry of the coarse stencil
    T v[4][9];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        const int fi = 2 * I + (ch & 1), fj = 2 * J + (ch >> 1);
        const bool in = fi < nyf && fj < nxf;
        const int c = fo + fj * nyf + fi;
#pragma unroll
        for (int k = 0; k < 9; ++k) v[ch][k] = in ? Af[(long)k * nf + c] : (T)0;
    }
    double acc[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) acc[k] = 0.0;
#pragma unroll
    for (int ch = 0; ch < 4; ++ch)
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int ci = ((ch & 1) + k % 3 + 1) / 2 - 1, cj = ((ch >> 1) + k / 3 + 1) / 2 - 1;   // -1, 0 or 1
            if (v[ch][k] != (T)0) acc[(cj + 1) * 3 + ci + 1] += (double)v[ch][k];
        }
    T* Ac = (T*)M.A[l + 1];
    const int nc = M.n[l + 1];
#pragma unroll
    for (int k = 0; k < 9; ++k) Ac[(long)k * nc + Q] = (T)acc[k];
    ((T*)M.dinv[l + 1])[Q] = (acc[4] != 0.0 && isfinite(acc[4])) ? (T)(1.0 / acc[4]) : (T)0;
}

// ------------------------------------------------------------ cycle
// Level 0 pre-smooth from zero (z0 = w D^-1 in), residual, restriction to
// the half-cells: r1[h] = sum_{i in h} (in_i - (A0 z0)_i).  One warp per
// cell, four sums (one per quadrant); every half-cell is written, empty
// ones with 0.
// sum over the row's off-diagonal nonzeros of A * u (sliced ELL), four
// independent index/value loads in flight before the gathers
template <typename T>
__device__ __forceinline__ T ell_dot(const T* __restrict__ A, const int* __restrict__ idx,
                                     const T* __restrict__ u, int r, int n, int kmax, T acc) {
    long e = ell(r, 0, kmax);
    int k = 0;
    for (; k + 4 <= n; k += 4, e += 128) {
        const int j0 = __ldg(idx + e), j1 = __ldg(idx + e + 32), j2 = __ldg(idx + e + 64), j3 = __ldg(idx + e + 96);
        const T a0 = __ldg(A + e), a1 = __ldg(A + e + 32), a2 = __ldg(A + e + 64), a3 = __ldg(A + e + 96);
        const T u0 = u[j0], u1 = u[j1], u2 = u[j2], u3 = u[j3];
        acc += a0 * u0;
        acc += a1 * u1;
        acc += a2 * u2;
        acc += a3 * u3;
    }
    for (; k < n; ++k, e += 32) acc += __ldg(A + e) * u[__ldg(idx + e)];
    return acc;
}

// Level 0, pass 1: the residual after the pre-sweep from zero, v = xin - A u
// (u = omega xin / adiag, written with the input), one thread per row on the
// aligned row blocks (coalesced slices of the ELL), into zz (free until the
// prolongation)
template <typename T>
__global__ void k_mg_l0_resid(Dev D, int fg) {
    BS_PDL_ENTRY();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = D.blk_scene[r / BS_ALIGN];
    if (mg_skip(D, s, fg)) return;
    if (r >= D.par[s].row0 + D.dyn[s].n) return;
    const T* __restrict__ u = (const T*)D.mg.u;
    const T* __restrict__ A = (const T*)(sizeof(T) == 8 ? D.aval : (void*)D.aval32);
    T v = ((const T*)D.mg.xin)[r];
    if (D.mg.pre0) v -= ell_dot<T>(A, D.nidx, u, r, D.ncount[r], D.kmax, ((const T*)D.mg.adiagT)[r] * u[r]);
    ((T*)D.mg.zz)[r] = v;
}

// Level 0, pass 2: restriction of that residual to the half-cells, a thread
// per half-cell summing the rows of its quadrant in row order (the four
// threads of a cell read the cell's rows together; one wave of threads)
template <typename T>
__global__ void k_mg_l0_down(Dev D, int fg) {
    BS_PDL_ENTRY();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = t >> 2, quad = t & 3;   // quad = lower | right << 1, as mg.sub
    if (c >= D.ncell_total) return;
    const int s = D.cell_scene[c];
    if (mg_skip(D, s, fg) || c - D.par[s].cell0 >= D.par[s].ncell) return;
    const T* __restrict__ zz = (const T*)D.mg.zz;
    const uint8_t* __restrict__ sub = D.mg.sub;
    const int r0 = D.cell_start[c], r1 = D.cell_end[c];
    T q = 0;
    int r = r0;
    for (; r + 4 <= r1; r += 4) {   // four rows' loads in flight
        const T v0 = zz[r], v1 = zz[r + 1], v2 = zz[r + 2], v3 = zz[r + 3];
        const int t0 = sub[r], t1 = sub[r + 1], t2 = sub[r + 2], t3 = sub[r + 3];
        q += (t0 == quad) ? v0 : (T)0;
        q += (t1 == quad) ? v1 : (T)0;
        q += (t2 == quad) ? v2 : (T)0;
        q += (t3 == quad) ? v3 : (T)0;
    }
    for (; r < r1; ++r) q += (sub[r] == quad) ? zz[r] : (T)0;
    const ScenePar& P = D.par[s];
    const int lc = c - P.cell0;
    const int i0 = lc % P.celly, j0 = lc / P.celly;
    const int Q = D.mg.off[1][s] + (2 * j0 + (quad >> 1)) * (2 * P.celly) + 2 * i0 + (quad & 1);
    ((T*)D.mg.r[1])[Q] = q;
}

// zz = u + cscale * e1[half-cell]: the level-0 value after the coarse correction
template <typename T>
__global__ void k_mg_l0_prolong(Dev D, int fg) {
    BS_PDL_ENTRY();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = D.blk_scene[r / BS_ALIGN];
    if (mg_skip(D, s, fg)) return;
    if (r >= D.par[s].row0 + D.dyn[s].n) return;
    const T pre = D.mg.pre0 ? ((const T*)D.mg.u)[r] : (T)0;
    ((T*)D.mg.zz)[r] = pre + (T)D.mg.cscale * ((const T*)D.mg.z[1])[D.mg.agg1[r]];
}

// ---- level operations on the cell levels (l >= 1), one cell per call.
// A scene's view of a level: its grid, its first cell in the level's arrays
// and the level's total size (the stride of the stencil arrays).  The
// per-level kernels build views from the MgLevel tables (kernel arguments,
// in the constant bank: no memory round trip for a cell's scene, offsets and
// grid).  On these
// small levels the kernels are bound by the latency of their dependent
// loads, not by bandwidth.  Converged scenes are not skipped here (their
// cells are few and the result is unused).
struct LevelS {
    int l, n, off, nx, ny;
};

// largest scene index k with G.off[k] <= c (scenes absent from the level
// have empty ranges)
__device__ __forceinline__ int scene_at(const MgLevel& G, int c) {
    int lo = 0, hi = G.ns - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (G.off[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ LevelS view_of(const MgLevel& G, int k) {
    LevelS v;
    v.l = G.l; v.n = G.n; v.off = G.off[k]; v.nx = G.nx[k]; v.ny = G.ny[k];
    return v;
}

// Levels l -> l+1 for coarse cell q of the scene: pre-smooth from zero,
// residual, restriction (2x2 sum).  The smoothed values w r D^-1 of the 4x4
// fine cells around the box are loaded once and all loads are issued before
// the sums (one round of memory latency instead of one per child: these
// levels are bound by their chains of dependent loads); the sums run in the
// same order as child by child.
template <typename T>
__device__ __forceinline__ void op_down(const MgDev& M, const LevelS& F, const LevelS& C, int q) {
    const int I = q % C.ny, J = q / C.ny;
    const T* __restrict__ A = (const T*)M.A[F.l];
    const T* __restrict__ dinv = (const T*)M.dinv[F.l];
    const T* __restrict__ r = (const T*)M.r[F.l];
    const T w = (T)M.omega;
    T sum = 0;
    if (!M.prec) {
        for (int b = 0; b < 2; ++b)
            for (int a = 0; a < 2; ++a) {
                const int fi = 2 * I + a, fj = 2 * J + b;
                if (fi < F.ny && fj < F.nx) sum += r[F.off + fj * F.ny + fi];
            }
        ((T*)M.r[C.l])[C.off + q] = sum;
        return;
    }
    const int fi0 = 2 * I - 1, fj0 = 2 * J - 1;   // the 4x4 neighbourhood's corner
    T y[4][4], rc[2][2];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int ni = fi0 + a, nj = fj0 + b;
            const bool in = ni >= 0 && nj >= 0 && ni < F.ny && nj < F.nx;
            const int nb = F.off + nj * F.ny + ni;
            y[b][a] = in ? w * r[nb] * __ldg(dinv + nb) : (T)0;
            if (a >= 1 && a <= 2 && b >= 1 && b <= 2) rc[b - 1][a - 1] = in ? r[nb] : (T)0;
        }
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const int fi = 2 * I + a, fj = 2 * J + b;
            if (fi >= F.ny || fj >= F.nx) continue;
            const int c = F.off + fj * F.ny + fi;
            T ax = 0;
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                const int ni = fi + (t % 3) - 1, nj = fj + (t / 3) - 1;
                if (ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx) continue;
                ax += __ldg(A + (long)t * F.n + c) * y[b + t / 3][a + t % 3];
            }
            sum += rc[b][a] - ax;
        }
    ((T*)M.r[C.l])[C.off + q] = sum;
}

// One child (a, b) of coarse cell q's 2x2 box: r_c - (A (w D^-1 r))_c, the
// value op_down adds for it (0 for a child beyond the fine grid); the
// neighbourhood's loads issued before the sum.
template <typename T>
__device__ __forceinline__ T down_child(const MgDev& M, const LevelS& F, const LevelS& C, int q, int a, int b) {
    const int I = q % C.ny, J = q / C.ny;
    const int fi = 2 * I + a, fj = 2 * J + b;
    if (fi >= F.ny || fj >= F.nx) return (T)0;
    const T* __restrict__ A = (const T*)M.A[F.l];
    const T* __restrict__ dinv = (const T*)M.dinv[F.l];
    const T* __restrict__ r = (const T*)M.r[F.l];
    const T w = (T)M.omega;
    const int c = F.off + fj * F.ny + fi;
    const T rc = r[c];
    if (!M.prec) return rc;
    T yv[9], av[9];
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int ni = fi + (t % 3) - 1, nj = fj + (t / 3) - 1;
        const bool in = !(ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx);
        const int nb = F.off + nj * F.ny + ni;
        yv[t] = in ? w * r[nb] * __ldg(dinv + nb) : (T)0;
        av[t] = in ? __ldg(A + (long)t * F.n + c) : (T)0;
    }
    T ax = 0;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int ni = fi + (t % 3) - 1, nj = fj + (t / 3) - 1;
        if (ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx) continue;
        ax += av[t] * yv[t];
    }
    return rc - ax;
}

// In-place residual on level l, cell q of the scene: r = r - A z (between
// the two visits of a W-cycle level; reads its own r and the stencil's z).
template <typename T>
__device__ __forceinline__ void op_resid(const MgDev& M, const LevelS& F, int q) {
    const int i = q % F.ny, j = q / F.ny;
    const int c = F.off + q;
    const T* __restrict__ A = (const T*)M.A[F.l];
    const T* z = (const T*)M.z[F.l];
    T* r = (T*)M.r[F.l];
    T zv[9], av[9];   // loads first (one round of latency), then the sum in stencil order
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
        const bool in = !(ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx);
        zv[t] = in ? z[F.off + nj * F.ny + ni] : (T)0;
        av[t] = in ? __ldg(A + (long)t * F.n + c) : (T)0;
    }
    const T rc = r[c];
    T ax = 0;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
        if (ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx) continue;
        ax += av[t] * zv[t];
    }
    r[c] = rc - ax;
}

// Levels l+1 -> l for cell q of the scene: prolongation (constant per box,
// scaled) + one post-sweep; with acc the result is added to z.
template <typename T>
__device__ __forceinline__ void op_up(const MgDev& M, const LevelS& F, const LevelS& C, int acc, int q) {
    const int i = q % F.ny, j = q / F.ny;
    const int c = F.off + q;
    const T* __restrict__ A = (const T*)M.A[F.l];
    const T* __restrict__ dinv = (const T*)M.dinv[F.l];
    const T* __restrict__ r = (const T*)M.r[F.l];
    const T* __restrict__ e = (const T*)M.z[C.l];
    const T w = (T)M.omega, cs = (T)M.cscale;
    const T wp = M.prec ? w : (T)0;
    // every load of the 3x3 neighbourhood issued before the sum (one round
    // of latency), the sum in stencil order
    T zv[9], av[9];
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
        const bool in = !(ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx);
        const int nb = F.off + nj * F.ny + ni;
        zv[t] = in ? wp * r[nb] * __ldg(dinv + nb) + cs * e[C.off + (nj / 2) * C.ny + (ni / 2)] : (T)0;
        av[t] = in ? __ldg(A + (long)t * F.n + c) : (T)0;
    }
    const T zc = zv[4];
    T ax = 0;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
        const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
        if (ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx) continue;
        ax += av[t] * zv[t];
    }
    const T v = zc + w * __ldg(dinv + c) * (r[c] - ax);
    T* zo = (T*)M.z[F.l];
    zo[c] = acc ? zo[c] + v : v;
}

// Coarsest level of one scene: damped Jacobi sweeps from zero by the whole
// block in shared memory (z, z2: coarse_max values each); with acc the
// result is added to z.  Every thread of the block calls it.
template <typename T>
__device__ __forceinline__ void op_coarse(const MgDev& M, const LevelS& F, int acc, T* z) {
    T* z2 = z + M.coarse_max;
    const int m = F.nx * F.ny;
    const T* __restrict__ A = (const T*)M.A[F.l];
    const T* __restrict__ dinv = (const T*)M.dinv[F.l];
    const T* __restrict__ r = (const T*)M.r[F.l];
    const T w = (T)M.omega;
    for (int q = threadIdx.x; q < m; q += blockDim.x) z[q] = 0;
    __syncthreads();
    if (m <= (int)blockDim.x) {
        // one cell per thread: its stencil, D^-1 and r held in registers
        // across the sweeps, which then touch shared memory only
        const int q = threadIdx.x;
        const bool act = q < m;
        const int i = q % F.ny, j = q / F.ny;
        const int c = F.off + q;
        T a9[9], dc = 0, rcv = 0;
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
            a9[t] = (act && !(ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx)) ? __ldg(A + (long)t * F.n + c) : (T)0;
        }
        if (act) {
            dc = __ldg(dinv + c);
            rcv = r[c];
        }
        for (int it = 0; it < M.coarse_sweeps; ++it) {
            if (act) {
                T ax = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
                    if (ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx) continue;
                    ax += a9[t] * z[nj * F.ny + ni];
                }
                z2[q] = z[q] + w * dc * (rcv - ax);
            }
            __syncthreads();
            if (act) z[q] = z2[q];
            __syncthreads();
        }
    } else {
        for (int it = 0; it < M.coarse_sweeps; ++it) {
            for (int q = threadIdx.x; q < m; q += blockDim.x) {
                const int i = q % F.ny, j = q / F.ny;
                const int c = F.off + q;
                T ax = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
                    if (ni < 0 || nj < 0 || ni >= F.ny || nj >= F.nx) continue;
                    ax += __ldg(A + (long)t * F.n + c) * z[nj * F.ny + ni];
                }
                z2[q] = z[q] + w * __ldg(dinv + c) * (r[c] - ax);
            }
            __syncthreads();
            for (int q = threadIdx.x; q < m; q += blockDim.x) z[q] = z2[q];
            __syncthreads();
        }
    }
    T* out = (T*)M.z[F.l];
    for (int q = threadIdx.x; q < m; q += blockDim.x) out[F.off + q] = acc ? out[F.off + q] + z[q] : z[q];
}

// ---- the lower levels of a visit on chip (option mg_tail)
// From the chosen level l0 down, a scene's visit (or the two visits of a
// W-cycle level with the residual between them) runs as one launch: a
// thread-block cluster per scene keeps every level's stencils and vectors in
// its shared memory, so a level operation costs a barrier instead of a launch
// and a round of L2 loads.  Each launch moves kilobytes: the per-level
// launches were bound by launch latency and dependent loads.
//  * A level of more than BS_CHIP_SOLO cells is split over the cluster's
//    blocks by columns (the boundaries are those of the first level below
//    that limit, doubled per level, so a 2x2 box never straddles two blocks).
//    A block stores its columns and one column to each side; whoever writes a
//    boundary column also stores it into the neighbour's copy (distributed
//    shared memory), then the cluster's barrier makes it visible.
//  * Smaller levels run in the cluster's first block (a block barrier costs
//    less than a cluster barrier there); the result of the largest of them
//    goes to slabs of the blocks that prolong from it.
//  * A thread holds one 2x2 box (quad): the 4x4 values around it are eight
//    two-value loads, a quarter of what a thread per cell reads from shared
//    memory, whose bandwidth bounds these operations.
//  * Columns carry a zero cell above and below and beyond the grid's sides,
//    and the stencil is 0 where it leaves the grid, so there are no range
//    tests (adding 0 changes no sum).
//  * The stencils, D^-1 and index tables of a block do not change during a
//    solve: k_mg_chip_pack writes them once, as they lie in shared memory, and
//    each visit fetches them by one bulk copy before it waits for the
//    preceding kernel.
// Every value is formed by the same operations in the same order as by the
// separate launches (bit-identical).
// What bounds it: chains of short dependent operations.  Two visits of a
// 22,800-cell level and the four below it (22 operations) take 27 us on 16
// blocks, against 17 launches of ~2.6 us; a block barrier costs 40 cycles, a
// cluster barrier with remote stores before it 650, an operation on a small
// level 1,200.  Per FGMRES column 37 -> 9 launches at 0.71 M particles, 17 ->
// 3 at 0.18 M, 9 -> 1 at 13 k; mixed step 15.99 -> 14.55, 5.00 -> 4.49 and
// 2.07 -> 1.92 ms.
#define BS_CHIP_THREADS 512
// cells of the largest level that the first block holds alone: beyond it a
// split operation is the shorter one (with 1536 the second largest level of
// the scenes above would be whole, and no longer fit beside the largest:
// 1.056x instead of 1.10x of the per-level launches at 0.18 M)
#define BS_CHIP_SOLO 1024
// One level of one block; offsets and strides in bytes of shared memory.
// Arrays R, Z, Y lie `area` apart from R; A: 9 x Q quads of T; tab: Q x uint2
// (chip_quad).
struct __align__(16) ChipLev {
    int R, area, sy, DV;              // sy: bytes per stored column (an even number of values)
    int A, tab, Q, ny;                // quads; rows
    int ncsy, left, nx, nc;           // nc sy; (j0 - the left neighbour's j0) sy; grid columns; this block's columns
    int j0, esh, cols, pad;           // first column; (j0 / 2) columns of the next level; columns reserved
};
struct __align__(16) ChipGeo {
    int d;                            // levels [0, d) are split, the first block holds the rest
    int zs;                           // the blocks' slab of level d's z
    int zero, zero0;                  // end of the zero-filled arrays, and of those of a block without solo levels
    int img, img0;                    // end of the constants, likewise; they begin at `zero`
    int pad0, pad1;
};
#define BS_CHIP_HDR ((int)(sizeof(ChipLev) * BS_MG_SUBL + sizeof(ChipGeo)))
// Tables of the levels of one block of the cluster (cs a power of two, width
// = sizeof(T)).  Shared memory: the tables, the zero-filled arrays (the split
// levels' first), the constants (likewise).
__host__ __device__ inline void chip_layout(ChipLev* V, ChipGeo* G, int nl, int nx0, int ny0, int cs, int rank,
                                            int width) {
    int d = 0;
    for (int u = 0; u < nl; ++u) {
        ChipLev& L = V[u];
        L.nx = (nx0 + (1 << u) - 1) >> u;   // halved (rounded up) u times
        L.ny = (ny0 + (1 << u) - 1) >> u;
        L.sy = ((L.ny + 3) & ~1) * width;
        if (cs > 1 && L.nx * L.ny > BS_CHIP_SOLO && d == u && u + 1 < nl) ++d;
    }
    int lg = 0;
    while ((1 << lg) < cs) ++lg;
    const int nxd = V[d].nx;
    const int c0 = (rank * nxd) >> lg, c1 = ((rank + 1) * nxd) >> lg, cl = ((rank - 1) * nxd) >> lg;
    const int cm = (nxd + cs - 1) >> lg;
    int at = BS_CHIP_HDR;
    for (int u = 0; u < nl; ++u) {
        ChipLev& L = V[u];
        if (u >= d) {
            L.j0 = 0;
            L.nc = L.cols = L.nx;
            L.left = 0;
        } else {
            const int j1 = c1 << (d - u);
            L.j0 = c0 << (d - u);
            L.nc = (j1 < L.nx ? j1 : L.nx) - L.j0;
            L.cols = cm << (d - u);
            L.left = ((c0 - cl) << (d - u)) * L.sy;
        }
        L.ncsy = L.nc * L.sy;
        L.esh = u + 1 < nl ? (L.j0 / 2) * V[u + 1].sy : 0;
        L.pad = 0;
        if (u == d) {
            G->zs = at;
            if (d > 0) at += (cm + 2) * L.sy;
            at = (at + 15) & ~15;
            G->zero0 = at;
        }
        L.area = ((L.cols + 3) * L.sy + 15) & ~15;   // a quad's window may reach one column beyond
        L.R = at;
        at += 3 * L.area;
        L.Q = ((L.cols + 1) / 2) * ((L.ny + 1) / 2);
    }
    G->zero = at;
    for (int u = 0; u < nl; ++u) {
        ChipLev& L = V[u];
        if (u == d) G->img0 = at;
        L.DV = at;
        L.A = at + L.area;
        L.tab = L.A + 9 * 4 * L.Q * width;
        at = (L.tab + 8 * L.Q + 15) & ~15;
    }
    G->img = at;
    G->d = d;
    G->pad0 = G->pad1 = 0;
}
// e / n for 0 <= e < 2^20 from inv = 1.0f / n (the half keeps the product off
// the integers, beyond its rounding error)
__device__ __forceinline__ int chip_div(int e, float inv) { return __float2int_rz(((float)e + 0.5f) * inv); }

// Quad q of level L (values of `width` bytes): x = offset of the corner of its
// 4x4 window | offset of its coarse cell << 16, both in values; y = children in
// the grid (bits 0..3, a + 2b) | its column is the block's first (16) | last (32)
__device__ __forceinline__ uint2 chip_quad(const ChipLev& L, int width, int q, int* I, int* J) {
    const int nyc = (L.ny + 1) / 2, syc = (nyc + 3) & ~1;
    *J = chip_div(q, 1.0f / (float)nyc);
    *I = q - *J * nyc;
    unsigned f = 0;
    for (int ch = 0; ch < 4; ++ch)
        if (2 * *I + (ch & 1) < L.ny && 2 * *J + (ch >> 1) < L.nc) f |= 1u << ch;
    if (f && *J == 0) f |= 16;
    if (f && *J == (L.nc + 1) / 2 - 1) f |= 32;
    return make_uint2((unsigned)(2 * *J * (L.sy / width) + 2 * *I) | (unsigned)((*J + 1) * syc + *I + 1) << 16, f);
}

// The constants of every block of every scene's cluster, once per solve
template <typename T>
__global__ void __launch_bounds__(BS_CHIP_THREADS) k_mg_chip_pack(Dev D, __grid_constant__ const MgChip S) {
    __shared__ ChipLev V[BS_MG_SUBL];
    __shared__ ChipGeo G;
    const MgDev& M = D.mg;
    const int cs = S.cs, k = blockIdx.x / cs, rank = blockIdx.x % cs, t = threadIdx.x;
    const int nl = S.lev[k] - S.l0 + 1;
    if (t == 0 && nl > 0) chip_layout(V, &G, nl, S.nx[k], S.ny[k], cs, rank, sizeof(T));
    __syncthreads();
    BS_PDL_ENTRY();
    if (nl < 1 || (rank > 0 && G.d == 0)) return;
    unsigned char* const img = (unsigned char*)M.chip_img + (long)blockIdx.x * S.stride;
    for (int e = t; e < BS_CHIP_HDR / 4; e += BS_CHIP_THREADS)
        ((int*)img)[e] = e < (int)sizeof(V) / 4 ? ((const int*)V)[e] : ((const int*)&G)[e - (int)sizeof(V) / 4];
    unsigned char* const cst = img + BS_CHIP_HDR - G.zero;   // constants at their shared-memory offsets
    for (int u = 0; u < (rank == 0 ? nl : G.d); ++u) {
        const ChipLev L = V[u];
        const int n = M.n[S.l0 + u], off = S.off[u][k];
        const T* __restrict__ A = (const T*)M.A[S.l0 + u] + off;
        const T* __restrict__ dv = (const T*)M.dinv[S.l0 + u] + off;
        T* const DV = (T*)(cst + L.DV);
        const int sy = L.sy / (int)sizeof(T);
        const float invy = 1.0f / (float)sy;
        for (int e = t; e < (L.cols + 3) * sy; e += BS_CHIP_THREADS) {
            const int jl = chip_div(e, invy), i = e - jl * sy - 1, j = L.j0 - 1 + jl;
            DV[e] = (i >= 0 && i < L.ny && j >= 0 && j < L.nx && jl <= L.nc + 1) ? dv[j * L.ny + i] : (T)0;
        }
        for (int e = t; e < 4 * L.Q; e += BS_CHIP_THREADS) {   // a thread per child
            const int q = e >> 2, ch = e & 3;
            int I, J;
            const uint2 w = chip_quad(L, sizeof(T), q, &I, &J);
            if (ch == 0) ((uint2*)(cst + L.tab))[q] = w;
            const int i = 2 * I + (ch & 1), j = L.j0 + 2 * J + (ch >> 1);
            T v[9];
#pragma unroll
            for (int s = 0; s < 9; ++s) {
                const int ni = i + (s % 3) - 1, nj = j + (s / 3) - 1;
                const bool in = (w.y >> ch & 1) && !(ni < 0 || nj < 0 || ni >= L.ny || nj >= L.nx);
                v[s] = in ? A[s * n + j * L.ny + i] : (T)0;
            }
#pragma unroll
            for (int s = 0; s < 9; ++s) ((T*)(cst + L.A))[(s * L.Q + q) * 4 + ch] = v[s];
        }
    }
}

// Shared memory by 32-bit address (these chains of short dependent operations
// are bound by their instruction count).  The order of the accesses of a thread
// is that of the source.
__device__ __forceinline__ void sld(unsigned a, float& x) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(a)); }
__device__ __forceinline__ void sld(unsigned a, double& x) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(a)); }
__device__ __forceinline__ void sld2(unsigned a, float& x, float& y) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x), "=f"(y) : "r"(a));
}
__device__ __forceinline__ void sld2(unsigned a, double& x, double& y) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a));
}
__device__ __forceinline__ void sld4(unsigned a, float (&v)[4]) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a));
}
__device__ __forceinline__ void sld4(unsigned a, double (&v)[4]) {
    sld2(a, v[0], v[1]);
    sld2(a + 16, v[2], v[3]);
}
__device__ __forceinline__ int4 sld_i4(unsigned a) {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 sld_u2(unsigned a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned sld_u(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sst(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sst(unsigned a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
// the 4x4 window at p (an even value: two-value loads), W[column][row]
template <typename T>
__device__ __forceinline__ void chip_window(unsigned p, int sy, T (&W)[4][4]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        sld2(p + c * sy, W[c][0], W[c][1]);
        sld2(p + c * sy + 2 * (int)sizeof(T), W[c][2], W[c][3]);
    }
}
// (A W) of the quad's four children
template <typename T>
__device__ __forceinline__ void chip_dots(const T (&a)[9][4], const T (&W)[4][4], T (&ax)[4]) {
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) ax[ch] = 0;
#pragma unroll
    for (int s = 0; s < 9; ++s)
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) ax[ch] += a[s][ch] * W[(ch >> 1) + s / 3][(ch & 1) + s % 3];
}

// Has the block's constants' copy landed?  (bounded: a copy that never ended
// would hang the GPU)
__device__ __forceinline__ bool chip_landed(unsigned bar, int tries) {
    unsigned ok = 0;
    for (int it = 0; it < tries && !ok; ++it)
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared.b64 p, [%1], 0; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok)
                     : "r"(bar)
                     : "memory");
    return ok != 0;
}
constexpr int CHIP_TRIES = 1 << 20;

template <int N>
struct ChipInt {
    static constexpr int value = N;
};

template <typename T>
__global__ void __launch_bounds__(BS_CHIP_THREADS) k_mg_chip(Dev D, __grid_constant__ const MgChip S, int fg) {
    constexpr int NT = BS_CHIP_THREADS, SZ = (int)sizeof(T);
    constexpr bool KEEP = SZ == 4;                 // the first level's stencil stays in registers
    extern __shared__ __align__(16) unsigned char chip_smem[];
    __shared__ unsigned ops[BS_MG_MAXOPS + 1];
    __shared__ int nlist;
    __shared__ unsigned lost;                      // a block of the cluster gave up
    __shared__ __align__(8) unsigned long long bar;
    const MgDev& M = D.mg;
    const int cs = S.cs, lg = 31 - __clz(cs);
    const int k = blockIdx.x >> lg, rank = cs > 1 ? (int)cluster_rank() : 0;
    const int t = threadIdx.x;
    const int nl = S.lev[k] - S.l0 + 1;            // the scene's levels l0 .. lev
    const int d = S.d[k];                          // levels [0, d) are split
    if (nl < 1 || (rank > 0 && d == 0)) {          // no such level, or the first block does it all
        BS_PDL_ENTRY();
        return;
    }
    // constants of the solve
    const unsigned sbar = (unsigned)__cvta_generic_to_shared(&bar), sb = (unsigned)__cvta_generic_to_shared(chip_smem);
    const unsigned sops = (unsigned)__cvta_generic_to_shared(ops), slost = (unsigned)__cvta_generic_to_shared(&lost);
    if (t == 0) {
        const unsigned char* img = (const unsigned char*)M.chip_img + (long)blockIdx.x * S.stride;
        const unsigned bytes = (unsigned)((rank == 0 ? S.img[k] : S.img0[k]) - S.zero[k]);
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(sbar));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(sbar), "r"(bytes + BS_CHIP_HDR) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sb),
                     "l"(img), "r"(BS_CHIP_HDR), "r"(sbar)
                     : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         sb + S.zero[k]),
                     "l"(img + BS_CHIP_HDR), "r"(bytes), "r"(sbar)
                     : "memory");
    }
    if (t >= NT - 32) {   // the ops that this block takes part in: op | level << 8 | add << 16 | last << 17
        const int lane = t & 31, nops = S.nops;
        int n = 0;
        for (int base = 0; base < nops; base += 32) {
            const int o = base + lane;
            const int op = o < nops ? S.op[o] : 0, u = o < nops ? S.lv[o] - S.l0 : nl;
            const bool on = u < nl && (u < d || rank == 0) && (op == 3 ? u == nl - 1 : op == 1 || u < nl - 1);
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on)
                ops[n + __popc(m & ((1u << lane) - 1))] =
                    op | u << 8 | (S.acc[o] ? 1 << 16 : 0) | (o == nops - 1 ? 1 << 17 : 0);
            n += __popc(m);
        }
        if (lane == 0) {
            ops[n] = 0;
            nlist = n;
        }
    }
    {
        const int e1 = (rank == 0 ? S.zero[k] : S.zero0[k]) >> 4;
        for (int e = BS_CHIP_HDR / 16 + t; e < e1; e += NT)
            reinterpret_cast<float4*>(chip_smem)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (t == 0) lost = 0;
    if (d > 0) cluster_arrive();                   // every block of the cluster runs before remote stores
    __syncthreads();
    if (__syncthreads_or(!chip_landed(sbar, rank == S.lose ? 0 : CHIP_TRIES))) {
        // Gives up, together with its cluster: the others store into this block's
        // shared memory until the barrier behind their first operation, and leave
        // there when they find `lost`.  Its own copy ends first.
        chip_landed(sbar, CHIP_TRIES);
        BS_PDL_ENTRY();
        const bool live = !mg_skip(D, k, fg);      // (else the others leave without an operation)
        if (d > 0) cluster_wait();
        if (live && d > 0) {
            if (t < cs) st_rank(slost, t, 1u);
            cluster_arrive();
            cluster_wait();
        }
        if (live && t == 0) set_err(D, k, BS_ERR_SOLVER_BREAK);
        return;
    }
    // level tables: x y z w = (R, area, sy, DV), (A, tab, Q, ny), (ncsy, left, nx, nc), (j0, esh, cols, -)
    auto lev = [&](int u, int part) { return sld_i4(sb + u * (int)sizeof(ChipLev) + part * 16); };
    const unsigned zs = sb + (d > 0 ? sld_u(sb + BS_MG_SUBL * (int)sizeof(ChipLev) + 4) : 0);
    const T w = (T)M.omega, cscale = (T)M.cscale;
    const bool prec = M.prec != 0;
    const T wp = prec ? w : (T)0;
    const int sweeps = M.coarse_sweeps;
    const int4 F0 = lev(0, 0), F1 = lev(0, 1), F2 = lev(0, 2), F3 = lev(0, 3);
    const int j00 = F3.x, ny0 = F1.w;
    T a0[9][4];
#pragma unroll
    for (int s = 0; s < 9; ++s) {
        a0[s][0] = a0[s][1] = a0[s][2] = a0[s][3] = 0;
        if (KEEP && t < F1.z) sld4(sb + F1.x + (s * F1.z + t) * 4 * SZ, a0[s]);
    }
    BS_PDL_ENTRY();
    const bool sdone = mg_skip(D, k, fg);
    if (!sdone) {   // the visit's right-hand side (with the side columns) and its pre-sweep from zero
        const T* __restrict__ rg = (const T*)M.r[S.l0] + S.off[0][k];
        const int nc = F2.w, nx = F2.z;
        constexpr int NW = NT / 32, CC = 2, RR = 3;   // columns and rows of a lane in flight
        for (int j0 = t >> 5; j0 < nc + 2; j0 += CC * NW)
            for (int i0 = t & 31; i0 < ny0; i0 += 32 * RR) {
                T r[CC][RR], dv[CC][RR];
#pragma unroll
                for (int c = 0; c < CC; ++c)
#pragma unroll
                    for (int q = 0; q < RR; ++q) {
                        const int jl = j0 + c * NW, j = j00 - 1 + jl, i = i0 + 32 * q;
                        const bool in = jl < nc + 2 && j >= 0 && j < nx && i < ny0;
                        r[c][q] = in ? __ldcg(rg + (j * ny0 + i)) : (T)0;
                    }
#pragma unroll
                for (int c = 0; c < CC; ++c)
#pragma unroll
                    for (int q = 0; q < RR; ++q) {
                        const int jl = j0 + c * NW, j = j00 - 1 + jl, i = i0 + 32 * q;
                        if (!(jl < nc + 2 && j >= 0 && j < nx && i < ny0)) continue;
                        const int e = jl * F0.z + (i + 1) * SZ;
                        sld(sb + F0.w + e, dv[c][q]);
                        sst(sb + F0.x + e, r[c][q]);
                        sst(sb + F0.x + 2 * F0.y + e, w * r[c][q] * dv[c][q]);
                    }
            }
    }
    if (d > 0) cluster_wait();
    __syncthreads();
    if (sdone) return;   // a finished scene (the same for every block of its cluster)

    T* const zg = (T*)M.z[S.l0] + S.off[0][k];
    const int nxd = d > 0 ? lev(d, 2).z : 1;
    const float inv_nxd = 1.0f / (float)nxd;
    const int nops = nlist;
    unsigned word = sld_u(sops);
    int4 L0 = lev((word >> 8) & 255, 0), L1 = lev((word >> 8) & 255, 1);
    uint2 qd = t < L1.z ? sld_u2(sb + L1.y + 8 * t) : make_uint2(0, 0);
    for (int o = 0; o < nops; ++o) {
        const int op = word & 255, u = (word >> 8) & 255;
        const bool acc = word & (1 << 16), last = word & (1 << 17);
        const bool solo = u >= d;
        const int sy = L0.z;
        const unsigned R = sb + L0.x, Z = R + L0.y, Y = Z + L0.y, DV = sb + L0.w;
        const unsigned A = sb + L1.x + t * 4 * SZ;
        const int strideA = L1.z * 4 * SZ;
        const int at = (qd.x & 0xffff) * SZ, an = (qd.x >> 16) * SZ;   // window corner, coarse cell
        const int ac = at + sy + SZ;                                    // the first child
        const unsigned flags = qd.y;
        const bool lpush = !solo && (flags & 16) && rank > 0, rpush = !solo && (flags & 32) && rank < cs - 1;
        const int ny = L1.w;
        const int4 N0 = lev(u + 1 < nl ? u + 1 : u, 0);
        auto dots = [&](const T(&W)[4][4], T(&ax)[4]) {
            if (KEEP && u == 0) {
                chip_dots(a0, W, ax);
            } else {
                T a[9][4];
#pragma unroll
                for (int s = 0; s < 9; ++s) sld4(A + s * strideA, a[s]);
                chip_dots(a, W, ax);
            }
        };
        // the first solo level's z (column J) goes to the slabs of the blocks that prolong from it
        auto publish = [&](int cell, int J, T v) {
            const int dst = chip_div((J + 1) * cs - 1, inv_nxd);   // the block that owns the column
            const int b0 = (dst * nxd) >> lg, b1 = ((dst + 1) * nxd) >> lg;
            st_rank(zs + cell - b0 * sy, dst, v);
            if (J == b0 && dst > 0) st_rank(zs + cell - (((dst - 1) * nxd) >> lg) * sy, dst - 1, v);
            if (J == b1 - 1 && dst < cs - 1) st_rank(zs + cell - b1 * sy, dst + 1, v);
        };
        auto barrier = [&]() {
            if (solo) {
                __syncthreads();
            } else {
                cluster_arrive();
                cluster_wait();
            }
        };
        if (op == 0) {   // residual after the pre-sweep, restriction; the next level's pre-sweep
            const bool away = !solo && u + 1 >= d; // the next level lies in the first block
            if (flags) {
                T ax[4] = {0, 0, 0, 0}, r[4];
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) sld(R + ac + (ch >> 1) * sy + (ch & 1) * SZ, r[ch]);
                if (prec) {
                    T W[4][4];
                    chip_window(Y + at, sy, W);
                    dots(W, ax);
                }
                T sum = 0;
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) sum += prec ? r[ch] - ax[ch] : r[ch];
                const unsigned n = sb + N0.x + an;
                if (away) {
                    st_rank(n + lev(u, 3).y, 0, sum);
                } else {
                    T dv;
                    sld(sb + N0.w + an, dv);
                    const T y = w * sum * dv;
                    sst(n, sum);
                    sst(n + 2 * N0.y, y);
                    if (u + 1 < d && (lpush || rpush)) {
                        const int4 N2 = lev(u + 1, 2);
                        if (lpush) {
                            st_rank(n + N2.y, rank - 1, sum);
                            st_rank(n + 2 * N0.y + N2.y, rank - 1, y);
                        }
                        if (rpush) {
                            st_rank(n - N2.x, rank + 1, sum);
                            st_rank(n + 2 * N0.y - N2.x, rank + 1, y);
                        }
                    }
                }
            }
        } else if (op == 1) {   // r -= A z, and the pre-sweep of the visit that follows
            if (flags) {
                T W[4][4], ax[4];
                chip_window(Z + at, sy, W);
                dots(W, ax);
                const int4 L2 = lev(u, 2);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    if (!(flags >> ch & 1)) continue;
                    const int c = ac + (ch >> 1) * sy + (ch & 1) * SZ;
                    T r, dv;
                    sld(R + c, r);
                    sld(DV + c, dv);
                    const T v = r - ax[ch];
                    const T y = w * v * dv;
                    sst(R + c, v);
                    sst(Y + c, y);
                    if (lpush && ch < 2) {
                        st_rank(R + c + L2.y, rank - 1, v);
                        st_rank(Y + c + L2.y, rank - 1, y);
                    }
                    if (rpush && ch >= 2) {
                        st_rank(R + c - L2.x, rank + 1, v);
                        st_rank(Y + c - L2.x, rank + 1, y);
                    }
                }
            }
        } else if (op == 2) {   // prolongation and post-sweep
            const bool slab = !solo && u + 1 >= d;
            if (slab) barrier();   // the first block's z has arrived
            if (flags) {
                const unsigned E = (slab ? zs : sb + N0.x + N0.y) + an;
                const int se = N0.z;
                T W[4][4], DW[4][4], EW[3][3], ax[4], rc[4], dc[4];
                chip_window(R + at, sy, W);
                chip_window(DV + at, sy, DW);
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int r = 0; r < 3; ++r) sld(E + (c - 1) * se + (r - 1) * SZ, EW[c][r]);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    rc[ch] = W[1 + (ch >> 1)][1 + (ch & 1)];
                    dc[ch] = DW[1 + (ch >> 1)][1 + (ch & 1)];
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        W[c][r] = wp * W[c][r] * DW[c][r] + cscale * EW[(c + 1) / 2][(r + 1) / 2];
                dots(W, ax);
                const int4 L2 = lev(u, 2);
                const bool pub = u == d && d > 0;
                // the quad's first column and row
                const int cj = last || pub ? 2 * (chip_div(an / SZ, 1.0f / (float)(se / SZ)) - 1) : 0;
                const int g = last ? (j00 + cj) * ny + 2 * (an / SZ - (cj / 2 + 1) * (se / SZ) - 1) : 0;
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    if (!(flags >> ch & 1)) continue;
                    const int c = ac + (ch >> 1) * sy + (ch & 1) * SZ;
                    T v = W[1 + (ch >> 1)][1 + (ch & 1)] + w * dc[ch] * (rc[ch] - ax[ch]);
                    if (acc) {
                        T z;
                        sld(Z + c, z);
                        v = z + v;
                    }
                    if (last) {   // the visit's result (u == 0)
                        zg[g + (ch >> 1) * ny + (ch & 1)] = v;
                        continue;
                    }
                    sst(Z + c, v);
                    if (lpush && ch < 2) st_rank(Z + c + L2.y, rank - 1, v);
                    if (rpush && ch >= 2) st_rank(Z + c - L2.x, rank + 1, v);
                    if (pub) publish(c, cj + (ch >> 1), v);
                }
            }
        } else {   // coarsest level: damped Jacobi from zero, a cell per thread of the first warps
            const int m = lev(u, 2).z * ny;
            const bool on = t < m;
            const int j = on ? chip_div(t, 1.0f / (float)ny) : 0, i = on ? t - j * ny : 0;
            const int c = (j + 1) * sy + (i + 1) * SZ;
            T z = 0, old = 0;
            auto sweep = [&](auto threads) {   // the warps that hold cells (t < threads)
                constexpr int NTHR = decltype(threads)::value;
                // the cell's stencil: child (i & 1) + 2 (j & 1) of its quad
                const unsigned ach = sb + L1.x + (((j >> 1) * ((ny + 1) / 2) + (i >> 1)) * 4 + (i & 1) + 2 * (j & 1)) * SZ;
                T a[9], rhs, dc;
#pragma unroll
                for (int s = 0; s < 9; ++s) sld(ach + s * strideA, a[s]);
                sld(R + c, rhs);
                sld(DV + c, dc);
                if (acc) sld(Z + c, old);
                if (on) sst(Y + c, (T)0);
                const T wd = w * dc;
                asm volatile("bar.sync 1, %0;" ::"n"(NTHR) : "memory");
                // z and its next value alternate between two arrays
                unsigned x = Y + c - sy, y = Z + c;
                int flip = (int)(Z - Y);
                for (int it = 0; it < sweeps; ++it) {
                    T v[9], ax = 0;
#pragma unroll
                    for (int s = 0; s < 9; ++s) sld(x + (s / 3) * sy + (s % 3 - 1) * SZ, v[s]);
#pragma unroll
                    for (int s = 0; s < 9; ++s) ax += a[s] * v[s];
                    z = z + wd * (rhs - ax);
                    if (on) sst(y, z);
                    asm volatile("bar.sync 1, %0;" ::"n"(NTHR) : "memory");
                    x += flip;
                    y -= flip;
                    flip = -flip;
                }
            };
            if (m <= 128) {
                if (t < 128) sweep(ChipInt<128>());
            } else if (m <= 256) {
                if (t < 256) sweep(ChipInt<256>());
            } else {
                sweep(ChipInt<NT>());
            }
            if (on) {
                const T v = acc ? old + z : z;
                sst(Z + c, v);
                if (u == 0) zg[t] = v;   // a scene without levels below
                else if (u == d && d > 0) publish(c, j, v);
            }
        }
        word = sld_u(sops + 4 * (o + 1));
        if (last) break;
        L0 = lev((word >> 8) & 255, 0);
        L1 = lev((word >> 8) & 255, 1);
        qd = t < L1.z ? sld_u2(sb + L1.y + 8 * t) : make_uint2(0, 0);
        barrier();
        if (o == 0 && d > 0 && sld_u(slost)) return;   // (the first operation of a split visit is one of a split level)
        if (op == 0 && !solo && u + 1 >= d && rank == 0) {   // the pre-sweep of the level the others restricted to
            const int4 N3 = lev(u + 1, 2);
            for (int e = t * SZ; e < N3.x + 2 * N0.z; e += NT * SZ) {
                T r, dv;
                sld(sb + N0.x + e, r);
                sld(sb + N0.w + e, dv);
                sst(sb + N0.x + 2 * N0.y + e, w * r * dv);
            }
            __syncthreads();
        }
    }
}

// ---- one launch per level operation
// A quad of lanes per coarse cell: lane (a, b) smooths child (a, b), the
// first lane adds the four values in op_down's order (b outer, a inner), so
// the result is bit-identical to op_down with a quarter of its loads per
// thread in flight at once.
template <typename T>
__global__ void k_mg_down(Dev D, __grid_constant__ const MgLevel F, __grid_constant__ const MgLevel C) {
    BS_PDL_ENTRY();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int Q = g >> 2, child = g & 3;
    bool ok = false;
    int q = 0, k = 0;
    T val = 0;
    if (Q < C.n) {
        k = scene_at(C, Q);
        q = Q - C.off[k];
        ok = q < C.nx[k] * C.ny[k];   // not reserved beyond the scene's current grid
        if (ok) val = down_child<T>(D.mg, view_of(F, k), view_of(C, k), q, child & 1, child >> 1);
    }
    const int base = (threadIdx.x & 31) & ~3;
    const T v0 = __shfl_sync(0xffffffffu, val, base), v1 = __shfl_sync(0xffffffffu, val, base + 1);
    const T v2 = __shfl_sync(0xffffffffu, val, base + 2), v3 = __shfl_sync(0xffffffffu, val, base + 3);
    if (ok && child == 0) {
        T sum = 0;
        sum += v0;
        sum += v1;
        sum += v2;
        sum += v3;
        ((T*)D.mg.r[C.l])[C.off[k] + q] = sum;
    }
}

template <typename T>
__global__ void k_mg_resid(Dev D, __grid_constant__ const MgLevel F) {
    BS_PDL_ENTRY();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= F.n) return;
    const int k = scene_at(F, c);
    const LevelS f = view_of(F, k);
    const int q = c - f.off;
    if (q >= f.nx * f.ny) return;
    op_resid<T>(D.mg, f, q);
}

template <typename T>
__global__ void k_mg_up(Dev D, __grid_constant__ const MgLevel F, __grid_constant__ const MgLevel C, int acc) {
    BS_PDL_ENTRY();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= F.n) return;
    const int k = scene_at(F, c);
    if (F.l >= F.lev[k]) return;   // the coarse solve wrote this level
    const LevelS f = view_of(F, k);
    const int q = c - f.off;
    if (q >= f.nx * f.ny) return;
    op_up<T>(D.mg, f, view_of(C, k), acc, q);
}

template <typename T>
__global__ void k_mg_coarse(Dev D, __grid_constant__ const MgLevel F, int acc) {
    BS_PDL_ENTRY();
    const int k = blockIdx.x;
    if (F.lev[k] != F.l) return;
    extern __shared__ unsigned char smem[];
    op_coarse<T>(D.mg, view_of(F, k), acc, (T*)smem);
}

// ---- exact coarse solve (option mg_exact).  A scene's level of at most
// BS_MG_EXACT_MAX cells (a 9-point Galerkin stencil on an nx x ny grid,
// cells numbered q = j ny + i) is a band matrix of half-bandwidth b = ny + 1.
// Once per step one block per scene factors it in FP64 (LU without pivoting,
// in shared memory: the Jacobi-scaled PPE and its Galerkin products are
// diagonally dominant M-matrices, whose pivots stay positive) and forms the
// inverse by m forward/back substitutions in parallel, one right-hand side
// per thread (the solution columns in global memory, coalesced across the
// threads).  Each visit of the level then is one mat-vec z = A^-1 r, a warp
// per row, in place of the Jacobi sweeps and the levels below.  Cells with
// no particle (zero diagonal) are decoupled rows whose z stays 0; if a
// pivot is not positive and finite the scene falls back to z = D^-1 r.
template <typename T>
__global__ void __launch_bounds__(1024) k_mg_exact_factor(Dev D, __grid_constant__ const MgExact E) {
    BS_PDL_ENTRY();
    const int k = blockIdx.x;
    const int l = E.l[k];
    if (l <= 0) return;
    const int nx = E.nx[k], ny = E.ny[k], m = nx * ny;
    if (m <= 0 || m > BS_MG_EXACT_MAX) return;
    const int b = ny + 1, W = 2 * b + 1;
    extern __shared__ double band[];   // row i: columns i-b .. i+b
    __shared__ int bad;
    const MgDev& M = D.mg;
    const T* __restrict__ A = (const T*)M.A[l];
    const long n = M.n[l];
    const int off = E.off[k];
    for (int e = threadIdx.x; e < m * W; e += blockDim.x) band[e] = 0.0;
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    for (int q = threadIdx.x; q < m; q += blockDim.x) {
        const int i = q % ny, j = q / ny;
        const double dq = (double)A[4 * n + off + q];
        if (dq == 0.0) {   // no particle in the cell: an identity row (its r is 0)
            band[q * W + b] = 1.0;
            continue;
        }
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const int ni = i + (t % 3) - 1, nj = j + (t / 3) - 1;
            if (ni < 0 || nj < 0 || ni >= ny || nj >= nx) continue;
            band[q * W + (nj * ny + ni - q + b)] = (double)A[t * n + off + q];
        }
    }
    __syncthreads();
    for (int kk = 0; kk < m; ++kk) {
        const double piv = band[kk * W + b];
        const int nr = min(m - 1, kk + b) - kk;
        if (threadIdx.x < nr) {
            const int i = kk + 1 + threadIdx.x;
            band[i * W + (kk - i + b)] /= piv;
        }
        if (threadIdx.x == 0 && !(piv > 0.0 && isfinite(piv))) bad = 1;
        __syncthreads();
        for (int e = threadIdx.x; e < nr * nr; e += blockDim.x) {
            const int i = kk + 1 + e / nr, jc = kk + 1 + e % nr;
            band[i * W + (jc - i + b)] -= band[i * W + (kk - i + b)] * band[kk * W + (jc - kk + b)];
        }
        __syncthreads();
    }
    double* X = M.xinv + (long)k * BS_MG_EXACT_MAX * BS_MG_EXACT_MAX;
    T* Ai = (T*)M.ainv + (long)k * BS_MG_EXACT_MAX * BS_MG_EXACT_MAX;
    if (bad) {
        const T* dinv = (const T*)M.dinv[l] + off;
        for (long e = threadIdx.x; e < (long)m * m; e += blockDim.x) Ai[e] = (e / m == e % m) ? dinv[e / m] : (T)0;
        return;
    }
    // column t of the inverse: L y = e_t (unit lower), then U x = y; X[i m + t]
    for (int t = threadIdx.x; t < m; t += blockDim.x) {
        for (int i = 0; i < m; ++i) {
            double y = (i == t) ? 1.0 : 0.0;
            for (int c = max(0, i - b); c < i; ++c) y -= band[i * W + (c - i + b)] * X[(long)c * m + t];
            X[(long)i * m + t] = y;
        }
        for (int i = m - 1; i >= 0; --i) {
            double x = X[(long)i * m + t];
            for (int c = i + 1; c <= min(m - 1, i + b); ++c) x -= band[i * W + (c - i + b)] * X[(long)c * m + t];
            X[(long)i * m + t] = x / band[i * W + b];
        }
    }
    __syncthreads();
    for (long e = threadIdx.x; e < (long)m * m; e += blockDim.x) Ai[e] = (T)X[e];
}

// z = A^-1 r on a scene's exactly solved level (added to z with acc): a warp
// per row, lanes over the row, a fixed-order sum
template <typename T>
__global__ void k_mg_exact_apply(Dev D, __grid_constant__ const MgLevel F, int acc) {
    BS_PDL_ENTRY();
    const int k = blockIdx.y;
    if (F.lev[k] != F.l) return;
    const int m = F.nx[k] * F.ny[k];
    const int lane = threadIdx.x & 31;
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= m) return;
    const T* __restrict__ Ai = (const T*)D.mg.ainv + (long)k * BS_MG_EXACT_MAX * BS_MG_EXACT_MAX + (long)q * m;
    const T* __restrict__ r = (const T*)D.mg.r[F.l] + F.off[k];
    T a = 0;
    for (int p = lane; p < m; p += 32) a += Ai[p] * r[p];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) {
        T* z = (T*)D.mg.z[F.l] + F.off[k];
        z[q] = acc ? z[q] + a : a;
    }
}

// ---- the levels from l0 down in one launch: one thread-block cluster per
// scene (cluster rank r, nt threads over the cluster, one cell per thread
// on the first level), the visit's level operations in order, a cluster
// barrier (release / acquire: the level arrays in global memory, L2
// resident) between them in place of a kernel boundary.  The coarsest-level
// solve runs in the cluster's first block.  Every thread reaches every
// barrier (no early exit).
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();   // (the aligned form needs the warp converged)
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned n;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return n;
}

template <typename T>
__global__ void __launch_bounds__(1024) k_mg_sub(Dev D, __grid_constant__ const MgSub S) {
    BS_PDL_ENTRY();
    extern __shared__ unsigned char smem[];
    const int cs = (int)cluster_size();
    const int k = blockIdx.x / cs, rank = blockIdx.x % cs;
    const int t = rank * blockDim.x + threadIdx.x, nt = cs * blockDim.x;
    for (int o = 0; o < S.nops; ++o) {
        const int l = S.lv[o];
        const MgLevel& F = S.G[l - S.l0];
        const LevelS f = view_of(F, k);
        switch (S.op[o]) {
            case 0: {   // down l -> l+1
                const LevelS c = view_of(S.G[l + 1 - S.l0], k);
                const int m = c.nx * c.ny;
                for (int q = t; q < m; q += nt) op_down<T>(D.mg, f, c, q);
                break;
            }
            case 1: {   // residual on l
                const int m = f.nx * f.ny;
                for (int q = t; q < m; q += nt) op_resid<T>(D.mg, f, q);
                break;
            }
            case 2: {   // up l+1 -> l (the coarse solve wrote the scene's coarsest level)
                if (l >= F.lev[k]) break;
                const LevelS c = view_of(S.G[l + 1 - S.l0], k);
                const int m = f.nx * f.ny;
                for (int q = t; q < m; q += nt) op_up<T>(D.mg, f, c, S.acc[o], q);
                break;
            }
            default:   // coarsest-level solve of the scenes whose coarsest level is l
                if (rank == 0 && F.lev[k] == l) op_coarse<T>(D.mg, f, S.acc[o], (T*)smem);
                break;
        }
        cluster_sync_all();
    }
}

// Level 0 post-sweep after the prolongation; writes the preconditioned
// vector (FP64).
// mode 0: one sweep from zz into out; with two post-sweeps (mg_post0 = 2)
// mode 1 sweeps zz into u (free after the prolongation) and mode 2 u into out.
template <typename T>
__global__ void k_mg_l0_up(Dev D, double* __restrict__ out, int mode, int fg) {
    BS_PDL_ENTRY();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = D.blk_scene[r / BS_ALIGN];
    if (mg_skip(D, s, fg)) return;
    if (r >= D.par[s].row0 + D.dyn[s].n) return;
    const T* __restrict__ zz = (const T*)(mode == 2 ? D.mg.u : D.mg.zz);
    const T* __restrict__ A = (const T*)(sizeof(T) == 8 ? D.aval : (void*)D.aval32);
    const int* __restrict__ idx = D.nidx;
    const T zr = zz[r];
    const T ax = ell_dot<T>(A, idx, zz, r, D.ncount[r], D.kmax, ((const T*)D.mg.adiagT)[r] * zr);
    const T x = ((const T*)D.mg.xin)[r];
    const T v = zr + (T)D.mg.omega * ((const T*)D.mg.dinv0)[r] * (x - ax);
    if (mode == 1) {
        ((T*)D.mg.u)[r] = v;
    } else {
        if (out) out[r] = (double)v;
        if (sizeof(T) == 4 && D.zf) D.zf[r] = (float)v;   // the double-float FGMRES pass reads it in FP32 (out null)
    }
}

inline unsigned gdiv(long a, int b) { return (unsigned)((a + b - 1) / b); }

// op list of one visit of level l (the recursion of cycle_t)
void sub_ops(const Dev& D, const Launch& L, int l, int acc, MgSub& S) {
    const unsigned char need = L.mgneed[l];
    if (!(need & 1)) return;
    auto push = [&](int op, int lv, int a) {
        if (S.nops < BS_MG_MAXOPS) {
            S.op[S.nops] = (unsigned char)op;
            S.lv[S.nops] = (unsigned char)lv;
            S.acc[S.nops] = (unsigned char)a;
        }
        S.nops++;
    };
    if (need & 4) push(3, l, acc);
    if (!(need & 2)) return;
    push(0, l, 0);
    sub_ops(D, L, l + 1, 0, S);
    if (l <= D.mg.wlev) {
        push(1, l + 1, 0);
        sub_ops(D, L, l + 1, 1, S);
    }
    push(2, l, acc);
}

// op list of `visits` visits (1, or 2 with the residual between them) of the
// chip level; false if it does not fit
bool chip_ops(const Dev& D, const Launch& L, int l0, int visits, MgChip& S) {
    MgSub V;
    V.nops = 0;
    sub_ops(D, L, l0, 0, V);
    if (visits == 2) {
        if (V.nops < BS_MG_MAXOPS) {
            V.op[V.nops] = 1;
            V.lv[V.nops] = (unsigned char)l0;
            V.acc[V.nops] = 0;
        }
        V.nops++;
        sub_ops(D, L, l0, 1, V);
    }
    S.nops = V.nops;
    if (V.nops > BS_MG_MAXOPS) return false;
    std::memcpy(S.op, V.op, sizeof(S.op));
    std::memcpy(S.lv, V.lv, sizeof(S.lv));
    std::memcpy(S.acc, V.acc, sizeof(S.acc));
    return true;
}

// the launch's tables: the visits' ops, the scenes' grids, offsets and layouts
template <typename T>
void chip_args(const Dev& D, const Launch& L, int visits, MgChip& S) {
    S.l0 = L.mgtail;
    S.cs = L.mgchip_cs;
    S.stride = L.mgchip_smem;
    S.lose = L.mgchip_lose;
    chip_ops(D, L, S.l0, visits, S);
    for (int k = 0; k < D.nscene; ++k) {
        const MgLevel& G = L.mglev[S.l0];
        S.nx[k] = G.nx[k];
        S.ny[k] = G.ny[k];
        S.lev[k] = G.nx[k] > 0 ? G.lev[k] : 0;
        for (int u = 0; u < BS_MG_SUBL; ++u) S.off[u][k] = S.l0 + u <= D.mg.nlev ? L.mglev[S.l0 + u].off[k] : 0;
        ChipLev V[BS_MG_SUBL];
        ChipGeo geo = {};
        if (S.lev[k] >= S.l0) chip_layout(V, &geo, S.lev[k] - S.l0 + 1, S.nx[k], S.ny[k], S.cs, 0, sizeof(T));
        S.d[k] = geo.d;
        S.zero[k] = geo.zero;
        S.zero0[k] = geo.zero0;
        S.img[k] = geo.img;
        S.img0[k] = geo.img0;
    }
}

template <typename T>
void chip_t(const Dev& D, const Launch& L, int visits, int fg) {
    MgChip S;
    chip_args<T>(D, L, visits, S);
    const int q = tbegin(L, K_MG_TAIL);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(D.nscene * S.cs));
    cfg.blockDim = dim3(BS_CHIP_THREADS);
    cfg.dynamicSmemBytes = (size_t)L.mgchip_smem;
    cfg.stream = L.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)S.cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, k_mg_chip<T>, D, S, fg);
    tend(L, q);
}

template <typename T>
void setup_t(const Dev& D, const Launch& L) {
    int q = tbegin(L, K_MG_GAL0);
    launch_pdl(L, k_mg_dinv0<T>, L.nblk_rows, BS_THREADS, 0, D);
    launch_pdl(L, k_mg_gal0<T>, gdiv((long)D.ncell_total * 32, BS_THREADS), BS_THREADS, 0, D);
    tend(L, q);
    *L.launches += 1;
    for (int l = 1; l < D.mg.nlev; ++l) {
        if (D.mg.exact && !(L.mgneed[l + 1] & 1)) break;   // below every scene's exact level
        q = tbegin(L, K_MG_GALC);
        launch_pdl(L, k_mg_galc<T>, gdiv(D.mg.n[l + 1], 128), 128, 0, D, l);
        tend(L, q);
    }
    if (L.mgtail) {
        MgChip S;
        chip_args<T>(D, L, 1, S);
        q = tbegin(L, K_MG_GALC);
        launch_pdl(L, k_mg_chip_pack<T>, (unsigned)(D.nscene * S.cs), BS_CHIP_THREADS, 0, D, S);
        tend(L, q);
    }
    if (D.mg.exact && L.exact) {
        q = tbegin(L, K_MG_GALC);
        launch_pdl(L, k_mg_exact_factor<T>, D.nscene, 1024, BS_MG_EXACT_BAND * sizeof(double), D, *L.exact);
        tend(L, q);
    }
}

// Cycle on level l >= 1 (input r[l], output z[l]); acc: add to z[l].
// Levels 1..wlev visit level l+1 twice (W), deeper levels once (V).
// Levels no scene needs launch nothing.  From the subtree level down, one
// clustered launch per visit.
template <typename T>
void cycle_t(const Dev& D, const Launch& L, int l, int acc, int fg) {
    const MgLevel* G = L.mglev;
    const unsigned char need = L.mgneed[l];
    if (!(need & 1)) return;
    int q;
    if (l == L.mgtail) {   // this level and everything below it on chip
        chip_t<T>(D, L, 1, fg);
        return;
    }
    if (l == L.mgsub_level) {   // this level and everything below: one clustered launch
        MgSub S;
        S.l0 = l;
        S.nops = 0;
        sub_ops(D, L, l, acc, S);
        for (int u = 0; u < BS_MG_SUBL && l + u <= D.mg.nlev; ++u) S.G[u] = G[l + u];
        q = tbegin(L, K_MG_SUB);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(D.nscene * L.mgsub_cs));
        cfg.blockDim = dim3(1024);
        cfg.dynamicSmemBytes = 2 * D.mg.coarse_max * sizeof(T);
        cfg.stream = L.stream;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)L.mgsub_cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 2;
        cudaLaunchKernelEx(&cfg, k_mg_sub<T>, D, S);
        tend(L, q);
        return;
    }
    if (need & 4) {
        q = tbegin(L, K_MG_COARSE);
        if (D.mg.exact)
            launch_pdl_2d(L, k_mg_exact_apply<T>, dim3(BS_MG_EXACT_MAX / 8, D.nscene), 256, 0, D, G[l], acc);
        else
            launch_pdl(L, k_mg_coarse<T>, D.nscene, 256, 2 * D.mg.coarse_max * sizeof(T), D, G[l], acc);
        tend(L, q);
    }
    if (!(need & 2)) return;
    q = tbegin(L, K_MG_DOWN);
    launch_pdl(L, k_mg_down<T>, gdiv(4L * D.mg.n[l + 1], 128), 128, 0, D, G[l], G[l + 1]);
    tend(L, q);
    if (l + 1 == L.mgtail && l <= D.mg.wlev) {
        chip_t<T>(D, L, 2, fg);   // both visits and the residual between them
    } else {
        cycle_t<T>(D, L, l + 1, 0, fg);
    }
    if (l <= D.mg.wlev && l + 1 != L.mgtail) {
        q = tbegin(L, K_MG_RESID);
        launch_pdl(L, k_mg_resid<T>, gdiv(D.mg.n[l + 1], 128), 128, 0, D, G[l + 1]);
        tend(L, q);
        cycle_t<T>(D, L, l + 1, 1, fg);
    }
    q = tbegin(L, K_MG_UP);
    launch_pdl(L, k_mg_up<T>, gdiv(D.mg.n[l], 128), 128, 0, D, G[l], G[l + 1], acc);
    tend(L, q);
}

template <typename T>
void apply_t(const Dev& D, const Launch& L, const double* in, double* out, int fg) {
    (void)in;   // the Krylov stream already wrote the input (mg_put_input)
    int q = tbegin(L, K_MG_L0DOWN);
    launch_pdl(L, k_mg_l0_resid<T>, row_blocks(L, L.mg0_tpb), L.mg0_tpb, 0, D, fg);
    tend(L, q);
    q = tbegin(L, K_MG_L0REST);
    launch_pdl(L, k_mg_l0_down<T>, gdiv((long)D.ncell_total * 4, 128), 128, 0, D, fg);
    tend(L, q);
    cycle_t<T>(D, L, 1, 0, fg);
    q = tbegin(L, K_MG_PROLONG);
    launch_pdl(L, k_mg_l0_prolong<T>, row_blocks(L, L.mg0_tpb), L.mg0_tpb, 0, D, fg);
    tend(L, q);
    q = tbegin(L, K_MG_L0UP);
    if (D.mg.post0 == 2) {
        launch_pdl(L, k_mg_l0_up<T>, row_blocks(L, L.mg0_tpb), L.mg0_tpb, 0, D, out, 1, fg);
        launch_pdl(L, k_mg_l0_up<T>, row_blocks(L, L.mg0_tpb), L.mg0_tpb, 0, D, out, 2, fg);
        *L.launches += 1;
    } else {
        launch_pdl(L, k_mg_l0_up<T>, row_blocks(L, L.mg0_tpb), L.mg0_tpb, 0, D, out, 0, fg);
    }
    tend(L, q);
}

}  // namespace

namespace bs {

// clusters of `cs` blocks of k_mg_sub that fit on the device at once (0: the
// cluster shape cannot be launched)
int mg_sub_max_clusters(int mg_precision, int cs, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cs);
    cfg.blockDim = dim3(1024);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    cudaError_t e;
    if (mg_precision == BS_PREC_MIXED) {
        if (cs > 8) cudaFuncSetAttribute(k_mg_sub<float>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        e = cudaOccupancyMaxActiveClusters(&n, k_mg_sub<float>, &cfg);
    } else {
        if (cs > 8) cudaFuncSetAttribute(k_mg_sub<double>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        e = cudaOccupancyMaxActiveClusters(&n, k_mg_sub<double>, &cfg);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int mg_exact_prepare() {
    const int bytes = BS_MG_EXACT_BAND * (int)sizeof(double);
    if (cudaFuncSetAttribute(k_mg_exact_factor<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_mg_exact_factor<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
            cudaSuccess)
        return BS_E_CUDA;
    return BS_OK;
}

void mg_setup(const Dev& D, const Launch& L, int mg_precision) {
    if (mg_precision == BS_PREC_MIXED) setup_t<float>(D, L);
    else setup_t<double>(D, L);
}

void mg_apply(const Dev& D, const Launch& L, int mg_precision, const double* in, double* out, int fg) {
    if (mg_precision == BS_PREC_MIXED) apply_t<float>(D, L, in, out, fg);
    else apply_t<double>(D, L, in, out, fg);
}

// Shared memory (bytes) of one block of the chip launch for a scene whose
// grid on the first level is nx x ny and whose coarsest level is nl - 1
// levels below, in clusters of cs; 0 when the split does not work out (the
// first solo level has fewer columns than the cluster has blocks).
size_t mg_chip_bytes(int mg_precision, int nl, int nx, int ny, int cs) {
    if (nl < 1 || nl > BS_MG_SUBL) return 0;
    ChipLev V[BS_MG_SUBL];
    ChipGeo G;
    const bool f32 = mg_precision == BS_PREC_MIXED;
    chip_layout(V, &G, nl, nx, ny, cs, 0, f32 ? 4 : 8);
    if (G.d > 0 && V[G.d].nx < cs) return 0;
    if (V[nl - 1].nx * V[nl - 1].ny > BS_CHIP_THREADS) return 0;   // the coarsest level: a cell per thread
    for (int u = 0; u < nl; ++u)   // a quad per thread; stored indices in 16 bits
        if (V[u].Q > BS_CHIP_THREADS || V[u].area / (f32 ? 4 : 8) >= 0xffff) return 0;
    return (size_t)G.img;
}

bool mg_chip_ops_fit(const Dev& D, const Launch& L, int l0, int visits) {
    MgChip S;
    return chip_ops(D, L, l0, visits, S);
}

// can a cluster of cs blocks with this much shared memory run at all?  (also
// allows the kernel that much, and clusters beyond the portable size)
bool mg_chip_prepare(int mg_precision, int cs, size_t smem) {
    const void* f = mg_precision == BS_PREC_MIXED ? (const void*)k_mg_chip<float> : (const void*)k_mg_chip<double>;
    int n = 0;
    bool ok = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, BS_CHIP_SMEM) == cudaSuccess &&
              (cs <= 8 || cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
    if (ok) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)cs);
        cfg.blockDim = dim3(BS_CHIP_THREADS);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        ok = cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess && n >= 1;
    }
    if (!ok) cudaGetLastError();
    return ok;
}

}  // namespace bs
