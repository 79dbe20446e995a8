// bs_solver.cu -- batched BiCGStab on the Jacobi-scaled PPE (bicgstab,
// solver.f90:129-254, on the padded-ELL operator spmv2, solver.f90:84-127).
//
// One iteration = three kernels over all scenes:
//   K1: p <- r + beta (p - omega v) folded into v <- A p  (gathers r,p,v)
//   K2: s <- r - alpha v folded into t <- A s            (gathers r,v)
//   K3: x <- x + alpha p + omega s ; r <- s - omega t
// Each kernel ends with per-scene FP64 dot products: block partials plus a
// deterministic finisher (the last block of the scene sums the partials in
// block order and updates the scene's scalars).  Converged scenes return at
// the top of every kernel.  FP64 mode: all vectors FP64.  Mixed mode: the
// inner iteration runs on FP32 vectors and FP32 matrix values; the outer
// loop recomputes the true residual with the FP64 matrix and corrects x
// (iterative refinement), with FP64 dots throughout.
#include <cstring>

#include "bs_internal.cuh"

namespace {

// Sum NV values over the scene's blocks; returns true in the finisher block
// (thread 0 holds the totals in tot[]).
template <int NV>
__device__ __forceinline__ bool scene_sum(const Dev& D, int s, double (&v)[NV], double (&tot)[NV]) {
    __shared__ double sh[NV * 32];
    __shared__ int last;
    const ScenePar& P = D.par[s];
    block_sum<NV>(v, sh);
    if (threadIdx.x == 0) {
        double* part = D.part + (long)blockIdx.x * BS_MAXDOT;
#pragma unroll
        for (int q = 0; q < NV; ++q) part[q] = v[q];
        __threadfence();
        const int prev = atomicAdd(&D.blk_done[s], 1);
        last = (prev == P.nblk - 1);
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double a[NV];
#pragma unroll
    for (int q = 0; q < NV; ++q) a[q] = 0.0;
    for (int b = threadIdx.x; b < P.nblk; b += blockDim.x) {
        const double* part = D.part + (long)(P.blk0 + b) * BS_MAXDOT;
#pragma unroll
        for (int q = 0; q < NV; ++q) a[q] += __ldcg(part + q);
    }
    __syncthreads();
    block_sum<NV>(a, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) tot[q] = a[q];
        D.blk_done[s] = 0;
    }
    return true;
}

__device__ __forceinline__ bool scene_done(const Dev& D, int s) { return D.dyn[s].converged != 0; }

// ---------------------------------------------------------------- FP64
__global__ void k_init64(Dev D, int* nconv) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double v[2] = {0.0, 0.0};
    if (r < P.row0 + D.dyn[s].n) {
        const double* A = (const double*)D.aval;
        double acc = D.adiag[r] * D.p[r];
        const int n = D.ncount[r];
        for (int k = 0; k < n; ++k) {
            const long e = ell(r, k, D.kmax);
            acc += A[e] * D.p[D.nidx[e]];
        }
        const double b = D.rhs[r];
        const double rr = b - acc;
        D.sr[r] = rr;
        D.srhat[r] = rr;
        D.sp[r] = 0.0;
        D.sv[r] = 0.0;
        v[0] = b * b;
        v[1] = rr * rr;
    }
    double tot[2];
    if (scene_sum<2>(D, s, v, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        Y.bnorm2 = tot[0];
        Y.rnorm2 = tot[1];
        Y.rho_old = tot[1];
        Y.alpha = 1.0;
        Y.omega = 1.0;
        Y.beta = 0.0;
        Y.iters = 0;
        Y.breakdown = 0;
        Y.outer = 0;
        Y.part_tmp = 0.0;
        const bool conv = (tot[0] == 0.0) || (tot[1] <= P.ppe_tol * P.ppe_tol * tot[0]);
        Y.converged = conv;
        if (conv) atomicAdd(nconv, 1);
    }
}

// KP: p = r + beta (p - omega v)   (streaming; beta = 0 on the first iteration);
// also writes the V-cycle input (mgmode 1: FP64, 2: FP32)
__global__ void k_pupd64(Dev D, int mgmode) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (scene_done(D, s)) return;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= D.par[s].row0 + D.dyn[s].n) return;
    const double beta = D.dyn[s].beta, omega = D.dyn[s].omega;
    const double p = D.sr[r] + beta * (D.sp[r] - omega * D.sv[r]);
    D.sp[r] = p;
    if (mgmode == 1) bs::mg_put_input<double>(D, r, p);
    else if (mgmode == 2) bs::mg_put_input<float>(D, r, p);
}

// y = A u for one row (1 DFMA per nonzero).  Latency: index, then value, in rounds;
// eight in a round instead of four, a two-step pass of the 13,681-row aquifer
// (30 neighbours, 73 columns a step) 6.10 -> 5.91 ms.
__device__ __forceinline__ double spmv_row64(const Dev& D, const double* __restrict__ u, int r) {
    const double* __restrict__ A = (const double*)D.aval;
    const int* __restrict__ idx = D.nidx;
    const int n = D.ncount[r];
    const int kmax = D.kmax;
    double acc = D.adiag[r] * u[r];
    long e = ell(r, 0, kmax);
    int k = 0;
    for (; k + 8 <= n; k += 8, e += 256) {   // eight independent gathers in flight
        int j[8];
        double a[8], v[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) j[m] = __ldg(idx + e + 32 * m);
#pragma unroll
        for (int m = 0; m < 8; ++m) a[m] = __ldg(A + e + 32 * m);
#pragma unroll
        for (int m = 0; m < 8; ++m) v[m] = u[j[m]];
#pragma unroll
        for (int m = 0; m < 8; ++m) acc = __fma_rn(a[m], v[m], acc);
    }
    for (; k + 4 <= n; k += 4, e += 128) {
        int j[4];
        double a[4], v[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) j[m] = __ldg(idx + e + 32 * m);
#pragma unroll
        for (int m = 0; m < 4; ++m) a[m] = __ldg(A + e + 32 * m);
#pragma unroll
        for (int m = 0; m < 4; ++m) v[m] = u[j[m]];
#pragma unroll
        for (int m = 0; m < 4; ++m) acc = __fma_rn(a[m], v[m], acc);
    }
    for (; k < n; ++k, e += 32) acc = __fma_rn(__ldg(A + e), u[__ldg(idx + e)], acc);
    return acc;
}

// K1: v = A u (u = p, or M^-1 p when preconditioned);  partial (rhat, v);
// finisher: alpha
__global__ void k_it1_64(Dev D, const double* __restrict__ u) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (scene_done(D, s)) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double q[1] = {0.0};
    if (r < P.row0 + D.dyn[s].n) {
        const double acc = spmv_row64(D, u, r);
        D.sv[r] = acc;
        q[0] = D.srhat[r] * acc;
    }
    double tot[1];
    if (scene_sum<1>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        if (tot[0] == 0.0 || !isfinite(tot[0])) {
            Y.breakdown = 1;
            Y.alpha = 0.0;
        } else {
            Y.alpha = Y.rho_old / tot[0];
        }
    }
}

// KS: s = r - alpha v   (streaming), plus the V-cycle input as in KP
__global__ void k_supd64(Dev D, int mgmode) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (scene_done(D, s)) return;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= D.par[s].row0 + D.dyn[s].n) return;
    const double v = D.sr[r] - D.dyn[s].alpha * D.sv[r];
    D.ss[r] = v;
    if (mgmode == 1) bs::mg_put_input<double>(D, r, v);
    else if (mgmode == 2) bs::mg_put_input<float>(D, r, v);
}

// K2: t = A u (u = s, or M^-1 s);  partials (t,s), (t,t);  finisher: omega
__global__ void k_it2_64(Dev D, const double* __restrict__ u) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (scene_done(D, s)) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (r < P.row0 + D.dyn[s].n) {
        const double acc = spmv_row64(D, u, r);
        D.st[r] = acc;
        const double si = D.ss[r];
        q[0] = acc * si;
        q[1] = acc * acc;
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        Y.omega = (tot[1] != 0.0) ? tot[0] / tot[1] : 0.0;
        if (tot[1] == 0.0) Y.breakdown = 1;
    }
}

// K3: x += alpha pu + omega su;  r = s - omega t;  partials (rhat, r), (r,r);
// finisher: beta, convergence
__global__ void k_it3_64(Dev D, const double* __restrict__ pu, const double* __restrict__ su, int* nconv) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (scene_done(D, s)) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const double alpha = D.dyn[s].alpha, omega = D.dyn[s].omega;
    double q[2] = {0.0, 0.0};
    double mrel = 0.0;
    if (r < P.row0 + D.dyn[s].n) {
        const double si = D.ss[r], ti = D.st[r];
        const double xo = D.p[r];
        const double xn = xo + alpha * pu[r] + omega * su[r];
        D.p[r] = xn;
        const double rr = si - omega * ti;
        D.sr[r] = rr;
        q[0] = D.srhat[r] * rr;
        q[1] = rr * rr;
        if (P.stop_rule == BS_STOP_REFERENCE) mrel = fabs((xn - xo) / (xo + BS_SP1EM5));
    }
    if (P.stop_rule == BS_STOP_REFERENCE) {
        __shared__ double shm[32];
        double mv[1] = {mrel};
        block_max<1>(mv, shm);
        __syncthreads();
        if (threadIdx.x == 0) atomicMax((unsigned long long*)&D.dyn[s].part_tmp, __double_as_longlong(mv[0]));
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        const double rho_new = tot[0];
        Y.beta = (rho_new / Y.rho_old) * (alpha / omega);
        Y.rho_old = rho_new;
        Y.rnorm2 = tot[1];
        Y.iters += 1;
        bool conv;
        if (P.stop_rule == BS_STOP_REFERENCE) {
            conv = Y.part_tmp <= (double)1e-2f;
            Y.part_tmp = 0.0;
        } else {
            conv = tot[1] <= P.ppe_tol * P.ppe_tol * Y.bnorm2;
        }
        if (!isfinite(tot[1])) {
            conv = true;
            set_err(D, s, BS_ERR_NONFINITE);
        }
        if (Y.breakdown) {
            conv = true;
            if (!(tot[1] <= P.ppe_tol * P.ppe_tol * Y.bnorm2)) set_err(D, s, BS_ERR_SOLVER_BREAK);
        }
        if (!conv && Y.iters >= P.maxit) {
            conv = true;
            set_err(D, s, BS_ERR_NOT_CONVERGED);
        }
        if (conv) {
            Y.converged = 1;
            atomicAdd(nconv, 1);
        }
    }
}

// ---------------------------------------------------------------- mixed
// Outer refinement: r64 = b - A64 x (FP64 matrix, FP64 vectors); the scene
// is done when ||r64|| <= tol ||b||.  Otherwise the inner FP32 BiCGStab
// solves A32 d = r64/||r64|| to inner_tol and x += ||r64|| d.
__global__ void k_mx_res(Dev D, int* nconv) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const ScenePar& P = D.par[s];
    SceneDyn& Y = D.dyn[s];
    if (Y.outer < 0) return;   // outer-converged
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (r < P.row0 + Y.n) {
        const double b = D.rhs[r];
        const double rr = b - spmv_row64(D, D.p, r);
        D.sxd[r] = rr;
        q[0] = rr * rr;
        q[1] = b * b;
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        Y.rtrue2 = tot[0];
        Y.bnorm2 = tot[1];
        Y.relres = (tot[1] > 0.0) ? sqrt(tot[0] / tot[1]) : sqrt(tot[0]);
        const bool done = (tot[1] == 0.0) || (tot[0] <= P.ppe_tol * P.ppe_tol * tot[1]) || !isfinite(tot[0]);
        if (!isfinite(tot[0])) set_err(D, s, BS_ERR_NONFINITE);
        if (done || Y.outer >= P.max_outer) {
            if (!done) set_err(D, s, BS_ERR_NOT_CONVERGED);
            Y.outer = -Y.outer - 1;   // mark outer-converged, keep the count
            Y.converged = 1;
            atomicAdd(nconv + 1, 1);
        } else {
            Y.rnorm2 = tot[0];
            Y.converged = 0;
            Y.outer += 1;
        }
    }
}

// inner init: r = r64 / ||r64|| in FP32, rhat = r, p = v = d = 0
__global__ void k_mx_init(Dev D, int* nconv) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const SceneDyn& Y0 = D.dyn[s];
    if (Y0.outer < 0) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const double scale = 1.0 / sqrt(Y0.rnorm2);
    double q[1] = {0.0};
    if (r < P.row0 + Y0.n) {
        const float rf = (float)(D.sxd[r] * scale);
        D.fr[r] = rf;
        D.frhat[r] = rf;
        D.fp[r] = 0.0f;
        D.fv[r] = 0.0f;
        D.fd[r] = 0.0f;
        q[0] = (double)rf * rf;
    }
    double tot[1];
    if (scene_sum<1>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        Y.rho_old = tot[0];
        Y.part_tmp = tot[0];   // inner ||r0||^2
        Y.alpha = 1.0;
        Y.omega = 1.0;
        Y.beta = 0.0;
        Y.breakdown = 0;
        if (tot[0] == 0.0) {
            Y.converged = 1;
            atomicAdd(nconv, 1);
        }
    }
}

__device__ __forceinline__ bool inner_done(const Dev& D, int s) {
    return D.dyn[s].outer < 0 || D.dyn[s].converged != 0;
}

// FP32 row of A32 applied to u_j = a_j + c (b_j - e g_j) evaluated on the fly
template <int MODE>
__device__ __forceinline__ float spmv_row32(const Dev& D, const float* __restrict__ a, const float* __restrict__ b,
                                            const float* __restrict__ g, float c, float e2, int r, float& own) {
    const float* __restrict__ A = (const float*)D.aval32;   // FP32 values (hi part)
    const int* __restrict__ idx = D.nidx;
    const int n = D.ncount[r];
    const int kmax = D.kmax;
    auto val = [&](int j) -> float {
        if (MODE == 0) return a[j] + c * (b[j] - e2 * g[j]);   // p = r + beta (p - omega v)
        return a[j] - c * b[j];                              // s = r - alpha v
    };
    own = val(r);
    float acc = (float)D.adiag[r] * own;
    long e = ell(r, 0, kmax);
    int k = 0;
    for (; k + 4 <= n; k += 4, e += 128) {
        const int j0 = __ldg(idx + e), j1 = __ldg(idx + e + 32), j2 = __ldg(idx + e + 64), j3 = __ldg(idx + e + 96);
        const float a0 = __ldg(A + e), a1 = __ldg(A + e + 32), a2 = __ldg(A + e + 64), a3 = __ldg(A + e + 96);
        const float u0 = val(j0), u1 = val(j1), u2 = val(j2), u3 = val(j3);
        acc = fmaf(a0, u0, acc);
        acc = fmaf(a1, u1, acc);
        acc = fmaf(a2, u2, acc);
        acc = fmaf(a3, u3, acc);
    }
    for (; k < n; ++k, e += 32) acc = fmaf(__ldg(A + e), val(__ldg(idx + e)), acc);
    return acc;
}

__global__ void k_mx_it1(Dev D, const float* __restrict__ p, const float* __restrict__ v, float* pn, float* vn) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (inner_done(D, s)) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const float beta = (float)D.dyn[s].beta, omega = (float)D.dyn[s].omega;
    double q[1] = {0.0};
    if (r < P.row0 + D.dyn[s].n) {
        float pi;
        const float acc = spmv_row32<0>(D, D.fr, p, v, beta, omega, r, pi);
        pn[r] = pi;
        vn[r] = acc;
        q[0] = (double)D.frhat[r] * acc;
    }
    double tot[1];
    if (scene_sum<1>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        if (tot[0] == 0.0 || !isfinite(tot[0])) {
            Y.breakdown = 1;
            Y.alpha = 0.0;
        } else {
            Y.alpha = Y.rho_old / tot[0];
        }
    }
}

__global__ void k_mx_it2(Dev D, const float* __restrict__ v) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (inner_done(D, s)) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const float alpha = (float)D.dyn[s].alpha;
    double q[2] = {0.0, 0.0};
    if (r < P.row0 + D.dyn[s].n) {
        float si;
        const float acc = spmv_row32<1>(D, D.fr, v, v, alpha, 0.0f, r, si);
        D.fs[r] = si;
        D.ft[r] = acc;
        q[0] = (double)acc * si;
        q[1] = (double)acc * acc;
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        Y.omega = (tot[1] != 0.0) ? tot[0] / tot[1] : 0.0;
        if (tot[1] == 0.0) Y.breakdown = 1;
    }
}

__global__ void k_mx_it3(Dev D, const float* __restrict__ p, int* nconv) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (inner_done(D, s)) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const float alpha = (float)D.dyn[s].alpha, omega = (float)D.dyn[s].omega;
    double q[2] = {0.0, 0.0};
    if (r < P.row0 + D.dyn[s].n) {
        const float si = D.fs[r], ti = D.ft[r];
        D.fd[r] = D.fd[r] + alpha * p[r] + omega * si;
        const float rr = si - omega * ti;
        D.fr[r] = rr;
        q[0] = (double)D.frhat[r] * rr;
        q[1] = (double)rr * rr;
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        const double rho_new = tot[0];
        Y.beta = (rho_new / Y.rho_old) * ((double)alpha / (double)omega);
        Y.rho_old = rho_new;
        Y.iters += 1;
        bool conv = tot[1] <= P.inner_tol * P.inner_tol * Y.part_tmp;
        if (!isfinite(tot[1]) || Y.breakdown) conv = true;
        if (Y.iters >= P.maxit) conv = true;
        if (conv) {
            Y.converged = 1;
            atomicAdd(nconv, 1);
        }
    }
}

// x += ||r64|| d
__global__ void k_mx_update(Dev D) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const SceneDyn& Y = D.dyn[s];
    if (Y.outer < 0) return;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= D.par[s].row0 + Y.n) return;
    D.p[r] = D.p[r] + sqrt(Y.rnorm2) * (double)D.fd[r];
}

// FP32 copy of the assembled FP64 matrix values (inner operator): hi part
// and the remainder; nothing to do where the mixed assembly already wrote them
__global__ void k_mx_convert(Dev D) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == D.par[s].row0) {
        D.dyn[s].outer = 0;
        D.dyn[s].iters = 0;
    }
    if (r >= D.par[s].row0 + D.dyn[s].n || D.dyn[s].asm_split) return;
    const double* A = (const double*)D.aval;
    float* F = D.aval32;
    const int n = D.ncount[r];
    for (int k = 0; k < n; ++k) {
        const long e = ell(r, k, D.kmax);
        const float h = (float)A[e];
        F[e] = h;
        D.aval_lo[e] = __double2float_rn(__dsub_rn(A[e], (double)h));
    }
}

// true FP64 residual ||b - A x|| / ||b|| for every scene (no early exit)
__global__ void k_true_res64(Dev D) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (r < P.row0 + D.dyn[s].n) {
        const double* A = (const double*)D.aval;
        double acc = D.adiag[r] * D.p[r];
        const int n = D.ncount[r];
        for (int k = 0; k < n; ++k) {
            const long e = ell(r, k, D.kmax);
            acc += A[e] * D.p[D.nidx[e]];
        }
        const double b = D.rhs[r];
        const double rr = b - acc;
        q[0] = rr * rr;
        q[1] = b * b;
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        Y.rtrue2 = tot[0];
        Y.relres = (tot[1] > 0.0) ? sqrt(tot[0] / tot[1]) : sqrt(tot[0]);
    }
}

// ---------------------------------------------------------------- FGMRES
// Restarted flexible GMRES (Saad, SIAM J. Sci. Comput. 14, 1993), the Krylov
// method of the reference's live solver (fgmres, solver.f90:306-350: MKL's
// RCI dfgmres with spmv2 as the operator, the previous pressure as the first
// guess, memory.f90:144, isph.f90:477).  Per scene: r0 = b - A x0, v0 =
// r0/||r0||; column j: z_j = M^-1 v_j (the multigrid cycle; z_j = v_j
// unpreconditioned), w = A z_j, classical Gram-Schmidt against v_0..v_j
// applied twice in two passes over the basis (the second projection from
// the basis' Gram matrix), h_{j+1,j} = ||w||, v_{j+1} = w / h_{j+1,j}; Givens rotations keep
// the least-squares residual |g_{j+1}| current.  The cycle ends when |g_{j+1}|
// <= ref, h_{j+1,j} <= 1e-12 (lucky breakdown), j+1 = m (restart) or at the
// iteration cap; then y = R^-1 g and x += Z y.  Scenes run their cycles in lock
// step; a scene whose cycle ended returns at the top of every column kernel,
// and the column index lives in the scene's state, so one captured chunk of
// columns serves every cycle.
//
// Two forms of a column.  FP64 basis (fg_df = 0): k_fg_put writes v_j and the
// V-cycle input, pass 1 (k_fg_arn1) the SpMV and the dots, pass 2
// (k_fg_arn2) the projection, the norm and, in its finisher, the
// rotations.  Double-float basis (fg_df = 1, the preconditioned mixed solve):
// the basis is stored as (hi, lo) FP32 pairs and its dots and projection run
// on the FP32 pipe; pass 1 (k_fg_arn1_df) also sums u.u and its finisher takes
// h_{j+1,j} from the Gram relation and runs the rotations, so pass 2
// (k_fg_arn2_df) streams v_{j+1} and the next V-cycle input with no reduction
// and k_fg_put runs once per cycle.

// Per-scene small storage: H [(m+1) x m] column-major (R of the rotated
// Hessenberg matrix), Gm [(m+1) x (m+1)] (the Gram matrix V^T V of the
// basis), cs[m], sn[m], g[m+1], y[m], hc[m+1] (the column's coefficients)
struct FgSmall {
    double *H, *Gm, *cs, *sn, *g, *y, *hc;
};
__device__ __forceinline__ FgSmall fg_small(const Dev& D, int s) {
    const int m = D.fg_m;
    double* b = D.fg_small + (long)s * D.fg_small_n;
    FgSmall f;
    f.H = b;
    b += (long)(m + 1) * m;
    f.Gm = b;
    b += (long)(m + 1) * (m + 1);
    f.cs = b;
    b += m;
    f.sn = b;
    b += m;
    f.g = b;
    b += m + 1;
    f.y = b;
    b += m;
    f.hc = b;
    return f;
}

__device__ __forceinline__ bool fg_running(const Dev& D, int s) {
    return D.dyn[s].converged == 0 && D.dyn[s].fg_state == 0;
}

__device__ __forceinline__ double warp_sum(double a) {
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// Double-float arithmetic (a value as an unevaluated sum hi + lo of two FP32
// numbers, 48 significant bits; Dekker 1971, Knuth's TwoSum, the FMA form of
// TwoProduct) for the Gram-Schmidt passes of the mixed solve: a basis element
// is 8 bytes as in FP64, and its products and sums run on the FP32 pipe, which
// on this part is ~60x faster than the FP64 pipe that bounds the FP64 form.
// Intrinsics keep every rounding explicit (no contraction).
__device__ __forceinline__ float2 df_split(double a) {
    const float h = __double2float_rn(a);
    return make_float2(h, __double2float_rn(__dsub_rn(a, (double)h)));
}
__device__ __forceinline__ double df_to_double(float2 a) { return __dadd_rn((double)a.x, (double)a.y); }
// s += a * b (products to ~2^-48 relative: TwoProduct of the high parts plus
// the cross terms; TwoSum into the running high part, errors into the low)
__device__ __forceinline__ void df_fma(float2& s, float2 a, float2 b) {
    const float ph = __fmul_rn(a.x, b.x);
    float pe = __fmaf_rn(a.x, b.x, -ph);
    pe = __fmaf_rn(a.x, b.y, pe);
    pe = __fmaf_rn(a.y, b.x, pe);
    const float t = __fadd_rn(s.x, ph);
    const float v = __fsub_rn(t, s.x);
    const float e = __fadd_rn(__fsub_rn(s.x, __fsub_rn(t, v)), __fsub_rn(ph, v));
    s.y = __fadd_rn(s.y, __fadd_rn(e, pe));
    s.x = t;
}
// a + b, renormalised
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
    const float t = __fadd_rn(a.x, b.x);
    const float v = __fsub_rn(t, a.x);
    float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(t, v)), __fsub_rn(b.x, v));
    e = __fadd_rn(e, __fadd_rn(a.y, b.y));
    const float h = __fadd_rn(t, e);
    return make_float2(h, __fsub_rn(e, __fsub_rn(h, t)));
}
__device__ __forceinline__ float2 df_shfl_xor(float2 a, int m) {
    return make_float2(__shfl_xor_sync(0xffffffffu, a.x, m), __shfl_xor_sync(0xffffffffu, a.y, m));
}

// Sum `cnt` rows of nv partials (row stride ld) in a fixed order: thread t
// takes value t % nv over rows q, q+Q, ... (q = t / nv, Q = 256 / nv), the
// Q sub-sums are added in q order.  The rows from `have` on are zeros (blocks
// without rows write nothing): they change nothing, so a scene's sums do not
// depend on its slot's capacity.  Eight loads in flight per thread.
__device__ __forceinline__ void fg_sum_rows(const double* __restrict__ src, int cnt, int have, int ld, int nv, double* out,
                                            double* scratch /*[BS_THREADS]*/) {
    const int t = threadIdx.x;
    if (nv <= BS_THREADS) {
        const int Q = BS_THREADS / nv;
        const int i = t % nv, q = t / nv;
        if (q < Q) {
            // four sub-sums over the rows that come in fours, the rest into the first; no operation for a row
            // of zeros (an FP64 instruction of a warp takes the SM's FP64 pipe 16 cycles)
            const int m = cnt > q ? (cnt - q + Q - 1) / Q : 0, full = m & ~3;
            const int mh = have > q ? (have - q + Q - 1) / Q : 0;
            double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
            for (int k = 0; k < mh; k += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = k + u < mh ? __ldcg(src + (long)(q + (k + u) * Q) * ld + i) : 0.0;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (k + u >= mh) break;
                    if ((u & 3) == 0 || k + u >= full) a0 += v[u];
                    else if ((u & 3) == 1) a1 += v[u];
                    else if ((u & 3) == 2) a2 += v[u];
                    else a3 += v[u];
                }
            }
            scratch[q * nv + i] = (a0 + a1) + (a2 + a3);
        }
        __syncthreads();
        if (t < nv) {
            double a = 0.0;
            for (int k = 0; k < Q; ++k) a += scratch[k * nv + t];
            out[t] = a;
        }
    } else {
        for (int i = t; i < nv; i += BS_THREADS) {
            const int full = cnt & ~1;
            double a0 = 0.0, a1 = 0.0;
            for (int k = 0; k < have; k += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = k + u < have ? __ldcg(src + (long)(k + u) * ld + i) : 0.0;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (k + u >= have) break;
                    if ((u & 1) && k + u < full) a1 += v[u];
                    else a0 += v[u];
                }
            }
            out[i] = a0 + a1;
        }
    }
    __syncthreads();
}

// The block's writes reach the device before its count: the writes are ordered
// before thread 0 by the block barrier and before the count by its fence; true
// in the block that counts last (its reads come after the others' writes).
__device__ __forceinline__ bool fg_count(int* counter, int total) {
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(counter, 1) == total - 1;
        if (last) {
            *counter = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return last != 0;
}

// Two-level scene sum of nv per-block values in vals[] (shared) over the
// scene's nact blocks that hold rows.  First level: the last block of each
// group of 32 row blocks sums the group into fg_gpart (tot: shared); true in
// that block.
__device__ __forceinline__ bool fg_group_sum(const Dev& D, int s, int nact, int nv, const double* vals, double* tot,
                                             double* scratch /*[BS_THREADS]*/) {
    const ScenePar& P = D.par[s];
    const int ld = bs::fg_part_ld(D.fg_m);
    const int grp = (blockIdx.x - P.blk0) >> 5, have = min(32, nact - (grp << 5));
    double* part = D.fg_part + (long)blockIdx.x * ld;
    for (int i = threadIdx.x; i < nv; i += BS_THREADS) part[i] = vals[i];
    if (!fg_count(&D.fg_gdone[P.grp0 + grp], have)) return false;
    fg_sum_rows(D.fg_part + (long)(P.blk0 + (grp << 5)) * ld, min(32, P.nblk - (grp << 5)), have, ld, nv, tot, scratch);
    double* gp = D.fg_gpart + (long)(P.grp0 + grp) * ld;
    for (int i = threadIdx.x; i < nv; i += BS_THREADS) gp[i] = tot[i];
    return true;
}
// Both levels: the last group of the scene sums the groups into tot[]; true in
// that block.  one_level: a small scene's last block sums its blocks' values
// itself (the order of the sums differs, so only where the solve does not
// multiply such a difference: without the FP32 preconditioner).  A column of an
// unpreconditioned solve with one level and with two, us: 3 blocks 46.6 and 49.5,
// 39 blocks 51.4 and 53.6, 54 blocks 52.8 and 53.0, 64 blocks 54.3 and 53.5, 79
// blocks 58.6 and 56.9, 235 blocks 110 and 93: they cross between 54 and 64.
#define BS_FG_ONE_LEVEL 64
__device__ __forceinline__ bool fg_scene_sum(const Dev& D, int s, int nact, int nv, const double* vals, double* tot,
                                             bool one_level) {
    __shared__ double scratch[BS_THREADS];
    const ScenePar& P = D.par[s];
    const int ld = bs::fg_part_ld(D.fg_m);
    if (one_level && nact <= BS_FG_ONE_LEVEL) {
        double* part = D.fg_part + (long)blockIdx.x * ld;
        for (int i = threadIdx.x; i < nv; i += BS_THREADS) part[i] = vals[i];
        if (!fg_count(&D.blk_done[s], nact)) return false;
        fg_sum_rows(D.fg_part + (long)P.blk0 * ld, nact, nact, ld, nv, tot, scratch);
        return true;
    }
    const int ngrp = (nact + 31) >> 5;
    if (!fg_group_sum(D, s, nact, nv, vals, tot, scratch)) return false;
    if (!fg_count(&D.blk_done[s], ngrp)) return false;
    fg_sum_rows(D.fg_gpart + (long)P.grp0 * ld, (P.nblk + 31) >> 5, ngrp, ld, nv, tot, scratch);
    return true;
}

// Cycle start: r = b - A x (into ss), ||r||, g = ||r|| e1.  first: every
// scene, sets the stopping threshold (tol ||r0|| or tol ||b||).
__global__ void k_fg_start(Dev D, int first, int* nconv, const int* cycle) {
    BS_PDL_ENTRY();
    if (cycle) first = (*cycle == 0);   // the captured solve counts its cycles on the device
    const int s = D.blk_scene[blockIdx.x];
    if (!first && D.dyn[s].converged) return;
    const ScenePar& P = D.par[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (r < P.row0 + D.dyn[s].n) {
        const double b = D.rhs[r];
        const double rr = b - spmv_row64(D, D.p, r);
        D.ss[r] = rr;
        q[0] = rr * rr;
        q[1] = b * b;
    }
    double tot[2];
    if (scene_sum<2>(D, s, q, tot) && threadIdx.x == 0) {
        SceneDyn& Y = D.dyn[s];
        const double beta = sqrt(tot[0]);
        if (first) {
            Y.bnorm2 = tot[1];
            Y.iters = 0;
            Y.outer = 0;
            Y.converged = 0;
            Y.breakdown = 0;
            Y.part_tmp = P.ppe_tol * (P.stop_rule == BS_STOP_RELRES ? sqrt(tot[1]) : beta);
        }
        Y.rnorm2 = tot[0];
        Y.rho_old = beta;   // norm of the vector the next column normalises
        Y.fg_rinv = beta > 0.0 ? 1.0 / beta : 0.0;
        Y.fg_j = 0;
        Y.fg_k = 0;
        fg_small(D, s).g[0] = beta;
        bool conv = tot[1] == 0.0 || beta <= Y.part_tmp;
        if (!isfinite(tot[0])) {
            conv = true;
            set_err(D, s, BS_ERR_NONFINITE);
        }
        if (conv) {
            Y.fg_state = 2;
            Y.converged = 1;
            atomicAdd(nconv, 1);
            atomicAdd(nconv + 1, 1);
        } else {
            Y.fg_state = 0;
            Y.outer += 1;   // cycles
        }
    }
}

// v_j = pending / its norm (into V), plus the V-cycle input (mgmode 1: FP64,
// 2: FP32); the scene's reciprocal norm is formed once by the producer (an
// FP64 division per row would bound this pass on this part)
__global__ void k_fg_put(Dev D, int mgmode) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (!fg_running(D, s)) return;
    const SceneDyn& Y = D.dyn[s];
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= D.par[s].row0 + Y.n) return;
    const double v = D.ss[r] * Y.fg_rinv;
    if (D.fg_df) reinterpret_cast<float2*>(D.fg_V)[(long)Y.fg_j * D.fg_ld + r] = df_split(v);
    else D.fg_V[(long)Y.fg_j * D.fg_ld + r] = v;
    if (mgmode == 1) bs::mg_put_input<double>(D, r, v);
    else if (mgmode == 2) bs::mg_put_input<float>(D, r, v);
}

// Column finisher (one block per scene): the new column h[0..j] of H, with
// h_{j+1,j} = hn below it, rotated by the cycle's earlier Givens rotations, a
// new rotation that zeroes hn, the residual estimate |g_{j+1}| and the cycle's
// state.  The value that runs down the column obeys t_{i+1} = -sn_i t_i +
// cs_i h_{i+1}.  scan: this chain of affine maps is composed by a prefix scan
// over the lanes of one warp (one after another they take 10 us at column 150);
// else one thread runs down it (in a block beside pass 2's streaming blocks,
// where its time does not count).  est_bad: hn was formed from the Gram
// relation rather than summed, and was not trusted (cancellation), so the
// cycle restarts from the true residual instead of going on.
__device__ void fg_finish_column(const Dev& D, int s, const FgSmall& f, int j, double hn, bool est_bad, bool scan,
                                 int* nconv) {
    constexpr int PER = (BS_FG_MAXM + 31) / 32;   // rotations per lane
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const ScenePar& P = D.par[s];
    const int m = D.fg_m;
    double* h = f.H + (long)j * (m + 1);
    double c[PER], sn[PER], b[PER];
    const int per = (j + 31) / 32, i0 = lane * per;   // this lane's rotations [i0, i0 + per) below j
    const double first = __ldcg(h);
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const bool in = q < per && i0 + q < j;
        c[q] = in ? __ldcg(f.cs + i0 + q) : 1.0;
        sn[q] = in ? __ldcg(f.sn + i0 + q) : 0.0;
        b[q] = in ? __ldcg(h + i0 + q + 1) : 0.0;
    }
    const double gj = lane == 0 ? __ldcg(f.g + j) : 0.0;
    double a;
    if (scan) {
        // the lane's map t -> A t + C over its rotations; a rotation beyond j leaves t as it is
        double A = 1.0, C = 0.0;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (q >= per || i0 + q >= j) continue;
            A = -sn[q] * A;
            C = -sn[q] * C + c[q] * b[q];
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {   // inclusive scan: the maps of lanes 0 .. lane
            const double Ap = __shfl_up_sync(0xffffffffu, A, o), Cp = __shfl_up_sync(0xffffffffu, C, o);
            if (lane >= o) {
                C = A * Cp + C;
                A = A * Ap;
            }
        }
        const double end = A * first + C;   // after this lane's rotations
        double t = __shfl_up_sync(0xffffffffu, end, 1);
        if (lane == 0) t = first;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            if (q >= per || i0 + q >= j) continue;
            h[i0 + q] = c[q] * t + sn[q] * b[q];
            t = -sn[q] * t + c[q] * b[q];
        }
        a = __shfl_sync(0xffffffffu, end, 31);
    } else {
        __shared__ double hcol[BS_FG_MAXM + 1], csh[BS_FG_MAXM], snh[BS_FG_MAXM];
#pragma unroll
        for (int q = 0; q < PER; ++q)
            if (q < per && i0 + q < j) {
                csh[i0 + q] = c[q];
                snh[i0 + q] = sn[q];
                hcol[i0 + q + 1] = b[q];
            }
        __syncwarp();
        a = first;
        if (lane == 0) {
            double hi = first;
            for (int i = 0; i < j; ++i) {
                const double bi = hcol[i + 1];
                hcol[i] = csh[i] * hi + snh[i] * bi;
                hi = -snh[i] * hi + csh[i] * bi;
            }
            a = hi;
        }
        __syncwarp();
        for (int i = lane; i < j; i += 32) h[i] = hcol[i];
    }
    if (lane == 0) {
        SceneDyn& Y = D.dyn[s];
        const double den = sqrt(a * a + hn * hn);
        const double cc = den > 0.0 ? a / den : 1.0, ss = den > 0.0 ? hn / den : 0.0;
        f.cs[j] = cc;
        f.sn[j] = ss;
        h[j] = den;
        h[j + 1] = 0.0;
        f.g[j] = cc * gj;
        f.g[j + 1] = -ss * gj;
        const double res = fabs(ss * gj);
        Y.rnorm2 = res * res;
        Y.rho_old = hn;
        Y.iters += 1;
        Y.fg_j = j + 1;
        int st = 0;
        if (!isfinite(res) || !isfinite(hn)) {
            st = 3;
            set_err(D, s, BS_ERR_NONFINITE);
        } else if (est_bad) {
            st = Y.iters >= P.maxit ? 3 : 1;
        } else if (res <= Y.part_tmp || hn <= 1e-12) {
            st = 2;
        } else if (Y.iters >= P.maxit) {
            st = 3;
        } else if (j + 1 == m) {
            st = 1;
        }
        Y.fg_state = st;
        if (st) atomicAdd(nconv, 1);
    }
}

// s += (a.x + a.y) z for an FP32 z: TwoProduct of the high part, the low
// part's product into the error, TwoSum into the running sum
__device__ __forceinline__ void df_fma1(float2& s, float2 a, float z) {
    const float ph = __fmul_rn(a.x, z);
    float pe = __fmaf_rn(a.x, z, -ph);
    pe = __fmaf_rn(a.y, z, pe);
    const float t = __fadd_rn(s.x, ph);
    const float v = __fsub_rn(t, s.x);
    const float e = __fadd_rn(__fsub_rn(s.x, __fsub_rn(t, v)), __fsub_rn(ph, v));
    s.y = __fadd_rn(s.y, __fadd_rn(e, pe));
    s.x = t;
}

// Row r of A z for an FP32-exact z (the mixed V-cycle output, zf): the
// off-diagonal values as double-float pairs (aval32 + aval_lo, 48 bits) and
// the products and sums on the FP32 pipe, eight gathers in flight; the diagonal
// term in FP64.  zr: z of the row in FP64.
__device__ __forceinline__ double spmv_row_df(const Dev& D, const float* z, int r, double& zr) {
    const float* __restrict__ Ah = D.aval32;
    const float* __restrict__ Al = D.aval_lo;
    const int* __restrict__ idx = D.nidx;
    const int n = D.ncount[r];
    const float zrow = z[r];
    float2 acc = make_float2(0.f, 0.f);
    long e = ell(r, 0, D.kmax);
    int k = 0;
    for (; k + 8 <= n; k += 8, e += 256) {
        int j[8];
        float2 a[8];
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) j[u] = __ldg(idx + e + 32 * u);
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u] = make_float2(__ldg(Ah + e + 32 * u), __ldg(Al + e + 32 * u));
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = z[j[u]];
#pragma unroll
        for (int u = 0; u < 8; ++u) df_fma1(acc, a[u], v[u]);
    }
    for (; k + 4 <= n; k += 4, e += 128) {
        int j[4];
        float2 a[4];
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) j[u] = __ldg(idx + e + 32 * u);
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = make_float2(__ldg(Ah + e + 32 * u), __ldg(Al + e + 32 * u));
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = z[j[u]];
#pragma unroll
        for (int u = 0; u < 4; ++u) df_fma1(acc, a[u], v[u]);
    }
    for (; k < n; ++k, e += 32) df_fma1(acc, make_float2(__ldg(Ah + e), __ldg(Al + e)), z[__ldg(idx + e)]);
    zr = (double)zrow;
    return __dadd_rn(__dmul_rn(D.adiag[r], zr), df_to_double(acc));
}

// Pass 1's finisher with the FP64 basis (the scene's last block; tsh: the summed
// dots h and c): the Gram column and the column's coefficients hc = (2I - Gm) h
// -- classical Gram-Schmidt applied twice, (I - V V^T)^2 = I - V (2I - V^T V) V^T,
// with the second projection taken from the Gram matrix instead of a second
// pass over V.
__device__ __forceinline__ void fg_arn1_finish(const Dev& D, int s, int j, const double* tsh) {
    const int nv = j + 1;
    const FgSmall f = fg_small(D, s);
    const int ldg = D.fg_m + 1;
    for (int i = threadIdx.x; i < nv; i += BS_THREADS) {
        f.Gm[i + (long)j * ldg] = tsh[nv + i];
        f.Gm[j + (long)i * ldg] = tsh[nv + i];
    }
    // Gm x for a vector x in shared memory, rows wid, wid + 8, ... by warp, four
    // rows' loads in flight (Gm is symmetric: row i is read as the contiguous
    // column i; its new row and column from tsh), the four sums over the lanes by
    // one transposing butterfly (6 FP64 adds instead of 20: this block's FP64
    // pipe sets its time); put(i, value) in one lane
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto gram = [&](const double* x, auto&& put) {
        for (int i0 = wid; i0 < nv; i0 += 4 * (BS_THREADS / 32)) {
            double a[4] = {0.0, 0.0, 0.0, 0.0};
            for (int k = lane; k < nv; k += 32) {
                double g[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i0 + u * (BS_THREADS / 32);
                    g[u] = i >= nv ? 0.0 : i == j ? tsh[nv + k] : k == j ? tsh[nv + i] : __ldcg(f.Gm + (long)i * ldg + k);
                }
                const double xk = x[k];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i0 + u * (BS_THREADS / 32) < nv) a[u] += g[u] * xk;
            }
            const bool b4 = lane & 16, b3 = lane & 8;
            double y[2];
#pragma unroll
            for (int u = 0; u < 2; ++u)
                y[u] = (b4 ? a[u + 2] : a[u]) + __shfl_xor_sync(0xffffffffu, b4 ? a[u] : a[u + 2], 16);
            double v = (b3 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, b3 ? y[0] : y[1], 8);
            v += __shfl_xor_sync(0xffffffffu, v, 4);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            const int i = i0 + ((b4 ? 2 : 0) + (b3 ? 1 : 0)) * (BS_THREADS / 32);
            if ((lane & 7) == 0 && i < nv) put(i, v);
        }
    };
    gram(tsh, [&](int i, double a) {
        const double acc = 2.0 * tsh[i] - a;
        f.hc[i] = acc;
        f.H[i + (long)j * ldg] = acc;
    });
}

// Column j, pass 1, FP64 basis: w = A z_j (z_j = the V-cycle output in sp2, kept
// as Z_j; or v_j) into sv; one read of v_0..v_j gives h = V^T w and the Gram
// column c = V^T v_j.
__global__ void __launch_bounds__(BS_THREADS, 5) k_fg_arn1(Dev D, int precond) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (!fg_running(D, s)) return;
    const int nact = (D.dyn[s].n + BS_THREADS - 1) / BS_THREADS;
    if ((int)blockIdx.x - D.par[s].blk0 >= nact) return;   // no rows
    __shared__ double ws[BS_THREADS], vs[BS_THREADS];
    __shared__ double dsh[2 * (BS_FG_MAXM + 1)];
    __shared__ double tsh[2 * (BS_FG_MAXM + 1)];
    const int j = D.dyn[s].fg_j, nv = j + 1;
    const int rend = D.par[s].row0 + D.dyn[s].n;
    const long r0 = (long)blockIdx.x * BS_THREADS;
    const int r = (int)r0 + threadIdx.x;
    const long col = (long)j * D.fg_ld;
    const double* u = precond ? D.sp2 : D.fg_V + col;
    double w = 0.0, vj = 0.0;
    if (r < rend) {
        w = spmv_row64(D, u, r);
        D.sv[r] = w;
        vj = D.fg_V[col + r];
        if (precond) D.fg_Z[col + r] = D.sp2[r];
    }
    ws[threadIdx.x] = w;
    vs[threadIdx.x] = vj;
    __syncthreads();
    // Warp w takes basis vectors w + 8 (4g + u), u = 0..3: lanes across the
    // block's rows (coalesced), 8 values per lane (4 vectors x 2 dots), summed
    // over the lanes by a transposing butterfly -- 9 FP64 adds per lane for
    // the 8 values rather than 5 per value (the FP64 pipe bounds this pass)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    for (int base = warp; base < nv; base += 4 * (BS_THREADS / 32)) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = base + (BS_THREADS / 32) * u;
            double a = 0.0, c = 0.0;
            if (i < nv) {
                const double* v = D.fg_V + (long)i * D.fg_ld + r0;
#pragma unroll
                for (int k = 0; k < BS_THREADS / 32; ++k) {
                    const int t = lane + 32 * k;
                    const double vi = (r0 + t < rend) ? v[t] : 0.0;
                    a += vi * ws[t];
                    c += vi * vs[t];
                }
            }
            x[2 * u] = a;
            x[2 * u + 1] = c;
        }
        double y[4], z[2];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            y[k] = (b4 ? x[k + 4] : x[k]) + __shfl_xor_sync(0xffffffffu, b4 ? x[k] : x[k + 4], 16);
#pragma unroll
        for (int k = 0; k < 2; ++k)
            z[k] = (b3 ? y[k + 2] : y[k]) + __shfl_xor_sync(0xffffffffu, b3 ? y[k] : y[k + 2], 8);
        double tv = (b2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b2 ? z[0] : z[1], 4);
        tv += __shfl_xor_sync(0xffffffffu, tv, 2);
        tv += __shfl_xor_sync(0xffffffffu, tv, 1);
        if ((lane & 3) == 0) {   // lane holds value q = lane / 4 = 2u + dot
            const int q = lane >> 2;
            const int i = base + (BS_THREADS / 32) * (q >> 1);
            if (i < nv) dsh[(q & 1) ? nv + i : i] = tv;
        }
    }
    __syncthreads();
    if (!fg_scene_sum(D, s, nact, 2 * nv, dsh, tsh, !precond)) return;
    fg_arn1_finish(D, s, j, tsh);
}

// Column j, pass 1, double-float basis: w = A z_j for the mixed V-cycle's output
// (zf; kept as Z_j) into sv, the dots of v_0..v_j with w and v_j, and w.w.
// Warp w takes the vectors w, w + 8, ...: 8 rows per lane loaded first, then two
// accumulation chains, w and v_j read from shared memory (48 registers, at 36
// bytes of spills: five blocks per SM).  The dots of four vectors (8 double-float values a lane) are
// summed over the lanes by a transposing butterfly, w.w of the eight warps by
// one warp likewise (9 FP64 adds instead of 40), each block's value converted
// to FP64 once for the FP64 scene sums.  Bound by HBM: 70 us for 312 MB at
// 0.71 M particles (cold, k_fg_fin not counted), 0.65 of the measured copy rate.  Measured and not kept: the
// basis fetched under the SpMV by bulk copies into a ring in shared memory
// (32 KB and 64 registers: four blocks per SM; 13.86 ms per step against 13.61,
// 4.20 against 4.06 at 0.18 M).
__global__ void __launch_bounds__(BS_THREADS, 5) k_fg_arn1_df(Dev D) {
    constexpr int NW = BS_THREADS / 32;
    __shared__ float2 wsd[BS_THREADS], vsd[BS_THREADS];
    __shared__ double wwp[BS_THREADS];
    __shared__ double dsh[2 * (BS_FG_MAXM + 1)];
    __shared__ double tsh[2 * (BS_FG_MAXM + 1)];
    const int s = D.blk_scene[blockIdx.x];
    const int blk0 = D.par[s].blk0;
    const int nact = (D.dyn[s].n + BS_THREADS - 1) / BS_THREADS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // (the scene's state and the basis were written at least two kernels ago)
    const bool running = fg_running(D, s);
    if (!running || (int)blockIdx.x - blk0 >= nact) {
        BS_PDL_ENTRY();
        return;
    }
    const int j = D.dyn[s].fg_j, nv = j + 1;
    const int rend = D.par[s].row0 + D.dyn[s].n;
    const long r0 = (long)blockIdx.x * BS_THREADS;
    const int r = (int)r0 + threadIdx.x;
    const long col = (long)j * D.fg_ld;
    const float2* Vb = reinterpret_cast<const float2*>(D.fg_V);
    const float2 vjd = r < rend ? __ldg(Vb + col + r) : make_float2(0.f, 0.f);
    BS_PDL_ENTRY();
    double w = 0.0;
    if (r < rend) {
        double zr;
        w = spmv_row_df(D, D.zf, r, zr);
        D.sv[r] = w;
        D.fg_Z[col + r] = zr;
    }
    wsd[threadIdx.x] = df_split(w);
    vsd[threadIdx.x] = vjd;
    wwp[threadIdx.x] = w * w;
    __syncthreads();
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    if (warp == NW - 1) {   // w.w: the sums over the lanes of each of the eight warps, then over the warps in order
        double x[8], y[4], z[2];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = wwp[32 * k + lane];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            y[k] = (b4 ? x[k + 4] : x[k]) + __shfl_xor_sync(0xffffffffu, b4 ? x[k] : x[k + 4], 16);
#pragma unroll
        for (int k = 0; k < 2; ++k)
            z[k] = (b3 ? y[k + 2] : y[k]) + __shfl_xor_sync(0xffffffffu, b3 ? y[k] : y[k + 2], 8);
        double t = (b2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b2 ? z[0] : z[1], 4);
        t += __shfl_xor_sync(0xffffffffu, t, 2);
        t += __shfl_xor_sync(0xffffffffu, t, 1);
        double a = 0.0;   // warp k's sum is in the lanes 4k .. 4k + 3 (k = 4 b4 + 2 b3 + b2)
#pragma unroll
        for (int k = 0; k < 8; ++k) a += __shfl_sync(0xffffffffu, t, 4 * k);
        if (lane == 0) dsh[2 * nv] = a;
    }
    for (int base = warp; base < nv; base += 4 * NW) {
        float2 x[8];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            float2 a = make_float2(0.f, 0.f), c = a;
            if (base + NW * u < nv) {
                const float2* v = Vb + (long)(base + NW * u) * D.fg_ld + r0;
                float2 vv[NW];
#pragma unroll
                for (int k = 0; k < NW; ++k) vv[k] = (r0 + lane + 32 * k < rend) ? v[lane + 32 * k] : make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    const int t = lane + 32 * k;
                    df_fma(a, vv[k], wsd[t]);
                    df_fma(c, vv[k], vsd[t]);
                }
            }
            x[2 * u] = a;
            x[2 * u + 1] = c;
        }
        float2 y[4], z[2];
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = df_add(b4 ? x[k + 4] : x[k], df_shfl_xor(b4 ? x[k] : x[k + 4], 16));
#pragma unroll
        for (int k = 0; k < 2; ++k) z[k] = df_add(b3 ? y[k + 2] : y[k], df_shfl_xor(b3 ? y[k] : y[k + 2], 8));
        float2 tv = df_add(b2 ? z[1] : z[0], df_shfl_xor(b2 ? z[0] : z[1], 4));
        tv = df_add(tv, df_shfl_xor(tv, 2));
        tv = df_add(tv, df_shfl_xor(tv, 1));
        if ((lane & 3) == 0) {
            const int qq = lane >> 2;
            const int i = base + NW * (qq >> 1);
            if (i < nv) dsh[(qq & 1) ? nv + i : i] = df_to_double(tv);
        }
    }
    __syncthreads();
    fg_group_sum(D, s, nact, 2 * nv + 1, dsh, tsh, wwp);   // (the scene's sums and the coefficients: k_fg_fin)
}

// The scene's sums and the column's coefficients with the double-float basis,
// one cluster of BS_FIN_BLOCKS blocks per scene (one block took 30 us of the
// 90 of pass 1 at 0.71 M particles: an FP64 instruction of a warp holds the
// SM's FP64 pipe for 16 cycles, and its loads came one chain after another).
// Each block sums its share of the 2 nv + 1 values over the groups (every
// sub-sum a thread's) and sends them to the others; the rows of the Gram
// products are shared out likewise, their old part loaded into registers before
// the wait for pass 1.  The orders of all sums are those of fg_sum_rows and of
// a warp per row.
//   hc = (2I - Gm) h (fg_arn1_finish), and h_{j+1,j} = ||w|| for w = u - V c
// without a pass over w: ||w||^2 = u.u - 2 c.h + c^T Gm c (u = A z_j, h = V^T u,
// Gm = V^T V, c = hc), so pass 2 can write v_{j+1} and the V-cycle input
// directly.  When that difference falls below 1e-6 u.u the estimate is not
// trusted and the cycle restarts from the true residual.  Pass 2 also runs the
// column's rotations (in a block of its own, beside the streaming ones).
#define BS_FIN_BLOCKS 8
__global__ void __launch_bounds__(BS_THREADS) k_fg_fin(Dev D) {
    constexpr int NB = BS_FIN_BLOCKS, NV = BS_FG_MAXM + 1;
    constexpr int RW = (NV + 8 * NB - 1) / (8 * NB), KL = (NV + 31) / 32;   // rows per warp, values per lane
    __shared__ double tot[2 * NV + 1], hcs[NV], gts[NV], eparts[8];
    __shared__ double scr[4 * BS_THREADS / NB + 4 * BS_THREADS], scr2[BS_THREADS / NB + BS_THREADS];
    const int s = blockIdx.x / NB, rank = (int)cluster_rank(), t = threadIdx.x;
    const int lane = t & 31, wid = t >> 5;
    SceneDyn& Y = D.dyn[s];
    if (!fg_running(D, s)) {   // (the state was written at least two kernels ago)
        BS_PDL_ENTRY();
        if (rank == 0 && t == 0) Y.fg_act = 0;   // no column for pass 2
        return;
    }
    const ScenePar& P = D.par[s];
    const FgSmall f = fg_small(D, s);
    const int j = Y.fg_j, nv = j + 1, nvals = 2 * nv + 1;
    const int ldg = D.fg_m + 1, ld = bs::fg_part_ld(D.fg_m);
    const int cnt = (P.nblk + 31) >> 5, have = ((Y.n + BS_THREADS - 1) / BS_THREADS + 31) >> 5;
    // this warp's rows of Gm: rank + NB (wid + 8 m); its new row and column come with the sums
    double g[RW][KL];
#pragma unroll
    for (int m = 0; m < RW; ++m) {
        const int i = rank + NB * (wid + 8 * m);
#pragma unroll
        for (int c = 0; c < KL; ++c) {
            const int k = lane + 32 * c;
            g[m][c] = i < j && k < j ? __ldcg(f.Gm + (long)i * ldg + k) : 0.0;
        }
    }
    cluster_arrive();   // every block of the cluster runs before remote stores
    BS_PDL_ENTRY();
    // this block's values [v0, v0 + nmine)
    const int per = (nvals + NB - 1) / NB, v0 = rank * per, nmine = max(0, min(per, nvals - v0));
    const double* __restrict__ src = D.fg_gpart + (long)P.grp0 * ld + v0;
    const int Q = nvals <= BS_THREADS ? BS_THREADS / nvals : 1;   // sub-sums of a value (rows q, q + Q, ...)
    const int A = nvals <= BS_THREADS ? 4 : 2;                    // accumulators of a sub-sum
    for (int e = t; e < nmine * Q * A; e += BS_THREADS) {
        const int i = e % nmine, qa = e / nmine, q = qa % Q, u = qa / Q;
        const int m = cnt > q ? (cnt - q + Q - 1) / Q : 0, full = m / A * A;
        const int mh = have > q ? (have - q + Q - 1) / Q : 0;
        double a = 0.0;
        for (int k0 = u; k0 < min(mh, full); k0 += 8 * A) {
            double v[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) v[x] = k0 + x * A < min(mh, full) ? __ldcg(src + (long)(q + (k0 + x * A) * Q) * ld + i) : 0.0;
#pragma unroll
            for (int x = 0; x < 8; ++x)
                if (k0 + x * A < min(mh, full)) a += v[x];
        }
        if (u == 0)
            for (int k = full; k < mh; ++k) a += __ldcg(src + (long)(q + k * Q) * ld + i);
        scr[e] = a;
    }
    __syncthreads();
    for (int e = t; e < nmine * Q; e += BS_THREADS) {
        const int st = nmine * Q;
        scr2[e] = A == 4 ? (scr[e] + scr[e + st]) + (scr[e + 2 * st] + scr[e + 3 * st]) : scr[e] + scr[e + st];
    }
    cluster_wait();
    __syncthreads();
    if (t < nmine) {
        double a = 0.0;
        if (A == 4)
            for (int q = 0; q < Q; ++q) a += scr2[q * nmine + t];
        else
            a = scr2[t];
        const unsigned p = (unsigned)__cvta_generic_to_shared(tot + v0 + t);
#pragma unroll
        for (int b = 0; b < NB; ++b) st_rank(p, b, a);
    }
    cluster_arrive();
    cluster_wait();
    // Gm x for a vector x in shared memory, one row after another of this warp
    auto gram = [&](const double* x, auto&& put) {
#pragma unroll
        for (int m = 0; m < RW; ++m) {
            const int i = rank + NB * (wid + 8 * m);
            if (i >= nv) break;
            double a = 0.0;
#pragma unroll
            for (int c = 0; c < KL; ++c) {
                const int k = lane + 32 * c;
                if (k < nv) a += (i == j ? tot[nv + k] : k == j ? tot[nv + i] : g[m][c]) * x[k];
            }
            a = warp_sum(a);
            put(i, a);
        }
    };
    gram(tot, [&](int i, double a) {
        const double acc = 2.0 * tot[i] - a;
        if (lane < NB) st_rank((unsigned)__cvta_generic_to_shared(hcs + i), lane, acc);
        if (lane == 0) {
            f.hc[i] = acc;
            f.H[i + (long)j * ldg] = acc;
            f.Gm[i + (long)j * ldg] = tot[nv + i];
            f.Gm[j + (long)i * ldg] = tot[nv + i];
        }
    });
    cluster_arrive();
    cluster_wait();
    gram(hcs, [&](int i, double a) {
        if (lane == 0) st_rank((unsigned)__cvta_generic_to_shared(gts + i), 0, a);
    });
    cluster_arrive();
    cluster_wait();
    if (rank != 0) return;
    if (t < 8) {   // the rows t, t + 8, ... in order, then these sums in order
        double part = 0.0;
        for (int i = t; i < nv; i += 8) part += hcs[i] * (gts[i] - 2.0 * tot[i]);
        eparts[t] = part;
    }
    __syncthreads();
    if (t == 0) {
        const double uu = tot[2 * nv];
        double eta2 = uu;
        for (int w = 0; w < 8; ++w) eta2 += eparts[w];
        const double hn = sqrt(fmax(eta2, 0.0));
        Y.fg_c = j;
        Y.fg_hn = hn;
        Y.fg_bad = !(eta2 > 1e-6 * uu);
        Y.fg_rinv = hn > 0.0 ? 1.0 / hn : 0.0;
        Y.fg_act = 1;
    }
}

// Column j, pass 2, FP64 basis: w -= V hc (the pending vector, into ss),
// h_{j+1,j} = ||w||; finisher: rotations, residual estimate, cycle end
__global__ void k_fg_arn2(Dev D, int* nconv, int mgmode) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    if (!fg_running(D, s)) return;
    __shared__ double hs[BS_FG_MAXM + 1];
    const ScenePar& P = D.par[s];
    const int j = D.dyn[s].fg_j;
    const int rend = P.row0 + D.dyn[s].n;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const FgSmall f = fg_small(D, s);
    for (int i = threadIdx.x; i <= j; i += BS_THREADS) hs[i] = f.hc[i];
    __syncthreads();
    double q[1] = {0.0};
    if (r < rend) {
        double w = D.sv[r];
        const double* v = D.fg_V + r;
        int i = 0;
        for (; i + 4 <= j + 1; i += 4) {   // four loads in flight
            const double v0 = v[(long)i * D.fg_ld], v1 = v[(long)(i + 1) * D.fg_ld];
            const double v2 = v[(long)(i + 2) * D.fg_ld], v3 = v[(long)(i + 3) * D.fg_ld];
            w -= hs[i] * v0;
            w -= hs[i + 1] * v1;
            w -= hs[i + 2] * v2;
            w -= hs[i + 3] * v3;
        }
        for (; i <= j; ++i) w -= hs[i] * v[(long)i * D.fg_ld];
        D.ss[r] = w;
        q[0] = w * w;
    }
    double tot[1];
    __shared__ double hns;
    if (!scene_sum<1>(D, s, q, tot)) return;
    if (threadIdx.x == 0) {
        hns = sqrt(tot[0]);
        D.dyn[s].fg_rinv = hns > 0.0 ? 1.0 / hns : 0.0;
    }
    __syncthreads();
    // (a preconditioned solve keeps the plain chain)
    fg_finish_column(D, s, f, j, hns, false, mgmode == 0, nconv);
}

// Column j, pass 2, double-float basis: v_{j+1} = (w - V hc) / h_{j+1,j} into
// the basis, and the V-cycle input (mgmode as k_fg_put), with no reduction.  Two
// rows per thread (16-byte loads of the basis), eight vectors in flight; per
// row four sums, the vectors in turn.  The first D.nscene blocks run the scenes'
// rotations (fg_finish_column) beside the streaming blocks; these read only
// what k_fg_fin left (fg_c, fg_act, fg_rinv), so a cycle that ends with this
// column has one vector too many.
#define BS_ARN2_THREADS (BS_ALIGN / 2)
__global__ void __launch_bounds__(BS_ARN2_THREADS) k_fg_arn2_df(Dev D, int* nconv, int mgmode) {
    BS_PDL_ENTRY();
    if ((int)blockIdx.x < D.nscene) {
        const SceneDyn& Y = D.dyn[blockIdx.x];
        if (Y.fg_act) fg_finish_column(D, blockIdx.x, fg_small(D, blockIdx.x), Y.fg_c, Y.fg_hn, Y.fg_bad != 0, false, nconv);
        return;
    }
    const int blk = blockIdx.x - D.nscene;
    const int s = D.blk_scene[blk];
    if (!D.dyn[s].fg_act) return;
    __shared__ float2 hsd[BS_FG_MAXM + 1];
    const int j = D.dyn[s].fg_c;
    const int rend = D.par[s].row0 + D.dyn[s].n;
    const int r = blk * BS_ALIGN + 2 * threadIdx.x;
    const FgSmall f = fg_small(D, s);
    for (int i = threadIdx.x; i <= j; i += BS_ARN2_THREADS) hsd[i] = df_split(f.hc[i]);
    __syncthreads();
    if (r >= rend) return;
    const double rinv = D.dyn[s].fg_rinv;
    const double2 w2 = *reinterpret_cast<const double2*>(D.sv + r);
    const long ld = D.fg_ld / 2;
    const float4* v = reinterpret_cast<const float4*>(D.fg_V) + r / 2;   // (x, y): the first row, (z, w): the second
    float2 a[4], b[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c] = b[c] = make_float2(0.f, 0.f);
    int i = 0;
    for (; i + 8 <= j + 1; i += 8) {
        float4 x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = v[(i + u) * ld];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float2 h = hsd[i + u];
            df_fma(a[u & 3], h, make_float2(x[u].x, x[u].y));
            df_fma(b[u & 3], h, make_float2(x[u].z, x[u].w));
        }
    }
    {   // the last ones: four in turn, then the rest into the first sum
        float4 x[7];
        const int left = j + 1 - i;
#pragma unroll
        for (int u = 0; u < 7; ++u) x[u] = u < left ? v[(i + u) * ld] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 7; ++u) {
            if (u >= left) break;
            const float2 h = hsd[i + u];
            const float2 p = make_float2(x[u].x, x[u].y), q = make_float2(x[u].z, x[u].w);
            if (u < 4 && left >= 4) {
                df_fma(a[u], h, p);
                df_fma(b[u], h, q);
            } else {
                df_fma(a[0], h, p);
                df_fma(b[0], h, q);
            }
        }
    }
    const double vn0 = __dsub_rn(w2.x, df_to_double(df_add(df_add(a[0], a[1]), df_add(a[2], a[3])))) * rinv;
    const double vn1 = __dsub_rn(w2.y, df_to_double(df_add(df_add(b[0], b[1]), df_add(b[2], b[3])))) * rinv;
    const float2 s0 = df_split(vn0), s1 = df_split(vn1);
    float2* out = reinterpret_cast<float2*>(D.fg_V) + (long)(j + 1) * D.fg_ld + r;
    auto put = [&](int q, double x) {
        if (mgmode == 1) bs::mg_put_input<double>(D, q, x);
        else if (mgmode == 2) bs::mg_put_input<float>(D, q, x);
    };
    out[0] = s0;
    put(r, vn0);
    if (r + 1 < rend) {
        out[1] = s1;
        put(r + 1, vn1);
    }
}

// One warp per scene: y = R^-1 g over the cycle's k columns; scenes that
// converged (or met the cap) in this cycle are marked done
__global__ void k_fg_solve(Dev D, int* nconv) {
    BS_PDL_ENTRY();
    const int s = blockIdx.x, lane = threadIdx.x;
    SceneDyn& Y = D.dyn[s];
    if (Y.converged) {
        if (lane == 0) Y.fg_k = 0;
        return;
    }
    __shared__ double ys[BS_FG_MAXM];
    const int k = Y.fg_j;
    const int ld = D.fg_m + 1;
    const FgSmall f = fg_small(D, s);
    // row i's entries right of the diagonal (lane: i + 1 + lane, + 32, ...), loaded a row ahead: a row
    // needs nothing of the one before it but its y
    constexpr int PER = (BS_FG_MAXM + 31) / 32;
    double h[PER], hn[PER], d = 0.0, g = 0.0, dn, gn;
    auto row = [&](int i, double (&v)[PER], double& di, double& gi) {
#pragma unroll
        for (int c = 0; c < PER; ++c) {
            const int l = i + 1 + lane + 32 * c;
            v[c] = i >= 0 && l < k ? __ldcg(f.H + i + (long)l * ld) : 0.0;
        }
        di = i >= 0 ? __ldcg(f.H + i + (long)i * ld) : 0.0;
        gi = i >= 0 ? __ldcg(f.g + i) : 0.0;
    };
    row(k - 1, h, d, g);
    for (int i = k - 1; i >= 0; --i) {
        row(i - 1, hn, dn, gn);
        double acc = 0.0;
#pragma unroll
        for (int c = 0; c < PER; ++c) {
            const int l = i + 1 + lane + 32 * c;
            if (l < k) acc += h[c] * ys[l];
        }
        // the sum over the lanes; the first k - 1 - i hold terms, the others 0
        const int terms = k - 1 - i;
        for (int o = 16; o > 0; o >>= 1)
            if (terms > o) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) ys[i] = d != 0.0 ? (g - acc) / d : 0.0;
        __syncwarp();
        d = dn;
        g = gn;
#pragma unroll
        for (int c = 0; c < PER; ++c) h[c] = hn[c];
    }
    for (int i = lane; i < k; i += 32) f.y[i] = ys[i];
    if (lane == 0) {
        Y.fg_k = k;
        if (Y.fg_state >= 2) {
            if (Y.fg_state == 3) set_err(D, s, BS_ERR_NOT_CONVERGED);
            Y.converged = 1;
            atomicAdd(nconv + 1, 1);
        }
    }
}

// x += Z y over the cycle's columns
__global__ void k_fg_update(Dev D, int precond) {
    BS_PDL_ENTRY();
    const int s = D.blk_scene[blockIdx.x];
    const int k = D.dyn[s].fg_k;
    if (k == 0) return;
    __shared__ double ys[BS_FG_MAXM];
    const FgSmall f = fg_small(D, s);
    for (int i = threadIdx.x; i < k; i += BS_THREADS) ys[i] = f.y[i];
    __syncthreads();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= D.par[s].row0 + D.dyn[s].n) return;
    const double* z = (precond ? D.fg_Z : D.fg_V) + r;
    double dx = 0.0;
    for (int i = 0; i < k; ++i) dx += ys[i] * z[(long)i * D.fg_ld];
    D.p[r] += dx;
}

}  // namespace

namespace bs {

// pass 1 of a column with the double-float basis: the row blocks, then the
// scenes' clusters
static void fg_pass1_df(const Dev& D, const Launch& L) {
    launch_pdl(L, k_fg_arn1_df, L.nblk_rows, BS_THREADS, 0, D);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(D.nscene * BS_FIN_BLOCKS));
    cfg.blockDim = dim3(BS_THREADS);
    cfg.stream = L.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = BS_FIN_BLOCKS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, k_fg_fin, D);
    *L.launches += 1;
}

// Host driver of the FP64 solve.  Checks the converged-scene counter every
// `check_every` iterations with one event sync, one chunk behind the launches
// so the GPU never idles on the host.
void solve_fp64(const Dev& D, const Launch& L, int maxit, int check_every, int precond, int mg_prec, int* d_nconv,
                int* h_nconv, cudaEvent_t ev) {
    int q;
    if (precond) {
        if (mg_prec == BS_PREC_MIXED) {
            q = tbegin(L, K_MX_CONV);
            launch_pdl(L, k_mx_convert, L.nblk_rows, BS_THREADS, 0, D);
            tend(L, q);
        }
        mg_setup(D, L, mg_prec);
    }
    const double* pu = precond ? D.sp2 : D.sp;   // M^-1 p
    const double* su = precond ? D.sv2 : D.ss;   // M^-1 s
    cudaMemsetAsync(d_nconv, 0, sizeof(int), L.stream);
    q = tbegin(L, K_BICG_INIT);
    launch_pdl(L, k_init64, L.nblk_rows, BS_THREADS, 0, D, d_nconv);
    tend(L, q);
    const int mgmode = precond ? (mg_prec == BS_PREC_MIXED ? 2 : 1) : 0;
    auto iteration = [&]() {
        int q2 = tbegin(L, K_BICG_PUPD);
        launch_pdl(L, k_pupd64, L.nblk_rows, BS_THREADS, 0, D, mgmode);
        tend(L, q2);
        if (precond) mg_apply(D, L, mg_prec, D.sp, D.sp2, 0);
        q2 = tbegin(L, K_BICG_IT1);
        launch_pdl(L, k_it1_64, L.nblk_rows, BS_THREADS, 0, D, pu);
        tend(L, q2);
        q2 = tbegin(L, K_BICG_SUPD);
        launch_pdl(L, k_supd64, L.nblk_rows, BS_THREADS, 0, D, mgmode);
        tend(L, q2);
        if (precond) mg_apply(D, L, mg_prec, D.ss, D.sv2, 0);
        q2 = tbegin(L, K_BICG_IT2);
        launch_pdl(L, k_it2_64, L.nblk_rows, BS_THREADS, 0, D, su);
        tend(L, q2);
        q2 = tbegin(L, K_BICG_IT3);
        launch_pdl(L, k_it3_64, L.nblk_rows, BS_THREADS, 0, D, pu, su, d_nconv);
        tend(L, q2);
    };
    // capture one convergence-check chunk (check_every iterations; an
    // iteration of a converged scene returns at once) as a CUDA graph, not
    // while per-kernel events are on
    IterGraph* G = L.graph;
    bool use_graph = G && !(L.timer && L.timer->mask);
    if (use_graph && !(G->valid && G->solver == BS_SOLVER_BICGSTAB && G->precond == precond && G->prec == mg_prec &&
                       G->chunk == check_every && std::memcmp(&G->key, &D, sizeof(Dev)) == 0)) {
        if (G->exec) cudaGraphExecDestroy(G->exec);
        G->exec = nullptr;
        G->valid = false;
        const int64_t before = *L.launches;
        cudaGraph_t gr = nullptr;
        if (cudaStreamBeginCapture(L.stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            for (int c = 0; c < check_every; ++c) iteration();
            if (cudaStreamEndCapture(L.stream, &gr) == cudaSuccess && gr &&
                cudaGraphInstantiate(&G->exec, gr, 0) == cudaSuccess) {
                G->valid = true;
                G->key = D;
                G->solver = BS_SOLVER_BICGSTAB;
                G->precond = precond;
                G->prec = mg_prec;
                G->chunk = check_every;
                G->nkernels = *L.launches - before;
            }
            if (gr) cudaGraphDestroy(gr);
        }
        *L.launches = before;
        cudaGetLastError();
        use_graph = G->valid;
    }
    int it = 0;
    while (it < maxit) {
        cudaMemcpyAsync(h_nconv, d_nconv, sizeof(int), cudaMemcpyDeviceToHost, L.stream);
        cudaEventRecord(ev, L.stream);
        if (use_graph) {
            cudaGraphLaunch(G->exec, L.stream);
            *L.launches += G->nkernels;
            it += check_every;
        } else {
            for (int c = 0; c < check_every && it < maxit; ++c, ++it) iteration();
        }
        cudaEventSynchronize(ev);
        timer_collect(L.timer, false);
        if (*h_nconv >= D.nscene) break;
    }
    q = tbegin(L, K_TRUERES);
    launch_pdl(L, k_true_res64, L.nblk_rows, BS_THREADS, 0, D);
    tend(L, q);
}

// Host driver of FGMRES: per restart cycle one start kernel and a host read
// of the converged count, then chunks of `check_every` columns (captured as
// one CUDA graph) until every scene's cycle has ended, then the small
// triangular solves and the update.  d_nconv[0] counts scenes whose cycle
// ended, d_nconv[1] converged scenes.
void solve_fgmres(const Dev& D, const Launch& L, int maxit, int check_every, int precond, int mg_prec,
                  int* d_nconv, int* h_nconv, cudaEvent_t ev) {
    int q;
    if (precond) {
        if (mg_prec == BS_PREC_MIXED) {
            q = tbegin(L, K_MX_CONV);
            launch_pdl(L, k_mx_convert, L.nblk_rows, BS_THREADS, 0, D);
            tend(L, q);
        }
        mg_setup(D, L, mg_prec);
    }
    const int mgmode = precond ? (mg_prec == BS_PREC_MIXED ? 2 : 1) : 0;
    // a column: [v_j and the V-cycle input], the V-cycle, pass 1, pass 2.  With
    // the double-float basis pass 2 writes v_{j+1} and the next input, so only
    // a cycle's first vector needs k_fg_put (after k_fg_start).
    auto put = [&]() {
        int q2 = tbegin(L, K_FG_PUT);
        launch_pdl(L, k_fg_put, L.nblk_rows, BS_THREADS, 0, D, mgmode);
        tend(L, q2);
    };
    auto column = [&]() {
        if (!D.fg_df) put();
        if (precond) mg_apply(D, L, mg_prec, D.fg_V, D.fg_df ? nullptr : D.sp2, 1);   // (pass 1 of the double-float form reads zf)
        int q2 = tbegin(L, K_FG_ARN);
        if (D.fg_df) fg_pass1_df(D, L);
        else launch_pdl(L, k_fg_arn1, L.nblk_rows, BS_THREADS, 0, D, precond);
        tend(L, q2);
        q2 = tbegin(L, K_FG_ORTH);
        if (D.fg_df) launch_pdl(L, k_fg_arn2_df, L.nblk_rows + D.nscene, BS_ARN2_THREADS, 0, D, d_nconv, mgmode);
        else launch_pdl(L, k_fg_arn2, L.nblk_rows, BS_THREADS, 0, D, d_nconv, mgmode);
        tend(L, q2);
    };
    IterGraph* G = L.graph;
    bool use_graph = G && !(L.timer && L.timer->mask);
    if (use_graph && !(G->valid && G->solver == BS_SOLVER_FGMRES && G->precond == precond && G->prec == mg_prec &&
                       G->chunk == check_every && std::memcmp(&G->key, &D, sizeof(Dev)) == 0)) {
        if (G->exec) cudaGraphExecDestroy(G->exec);
        G->exec = nullptr;
        G->valid = false;
        const int64_t before = *L.launches;
        cudaGraph_t gr = nullptr;
        if (cudaStreamBeginCapture(L.stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            for (int c = 0; c < check_every; ++c) column();
            if (cudaStreamEndCapture(L.stream, &gr) == cudaSuccess && gr &&
                cudaGraphInstantiate(&G->exec, gr, 0) == cudaSuccess) {
                G->valid = true;
                G->key = D;
                G->solver = BS_SOLVER_FGMRES;
                G->precond = precond;
                G->prec = mg_prec;
                G->chunk = check_every;
                G->nkernels = *L.launches - before;
            }
            if (gr) cudaGraphDestroy(gr);
        }
        *L.launches = before;
        cudaGetLastError();
        use_graph = G->valid;
    }
    cudaMemsetAsync(d_nconv, 0, 2 * sizeof(int), L.stream);
    // every cycle does at least one column of each scene it starts, and the
    // column kernels stop a scene at maxit columns
    for (int cycle = 0; cycle <= maxit; ++cycle) {
        cudaMemcpyAsync(d_nconv, d_nconv + 1, sizeof(int), cudaMemcpyDeviceToDevice, L.stream);
        q = tbegin(L, K_FG_START);
        launch_pdl(L, k_fg_start, L.nblk_rows, BS_THREADS, 0, D, cycle == 0 ? 1 : 0, d_nconv, (const int*)nullptr);
        tend(L, q);
        cudaMemcpyAsync(h_nconv, d_nconv, 2 * sizeof(int), cudaMemcpyDeviceToHost, L.stream);
        cudaStreamSynchronize(L.stream);
        timer_collect(L.timer, false);
        if (h_nconv[1] >= D.nscene) break;
        if (D.fg_df) put();
        int it = 0;
        while (it < D.fg_m) {
            cudaMemcpyAsync(h_nconv, d_nconv, sizeof(int), cudaMemcpyDeviceToHost, L.stream);
            cudaEventRecord(ev, L.stream);
            if (use_graph) {
                cudaGraphLaunch(G->exec, L.stream);
                *L.launches += G->nkernels;
                it += check_every;
            } else {
                for (int c = 0; c < check_every && it < D.fg_m; ++c, ++it) column();
            }
            cudaEventSynchronize(ev);
            timer_collect(L.timer, false);
            if (*h_nconv >= D.nscene) break;
        }
        q = tbegin(L, K_FG_UPD);
        launch_pdl(L, k_fg_solve, D.nscene, 32, 0, D, d_nconv);
        launch_pdl(L, k_fg_update, L.nblk_rows, BS_THREADS, 0, D, precond);
        tend(L, q);
    }
    q = tbegin(L, K_TRUERES);
    launch_pdl(L, k_true_res64, L.nblk_rows, BS_THREADS, 0, D);
    tend(L, q);
}

// Mixed solve: outer FP64 refinement around an FP32 BiCGStab.
void solve_mixed(const Dev& D, const Launch& L, int maxit, int check_every, int* d_nconv, int* h_nconv,
                 cudaEvent_t ev) {
    // FP32-inner iterative refinement (kept for systems whose condition number
    // times the FP32 unit round-off is well below one)
    int q = tbegin(L, K_MX_CONV);
    launch_pdl(L, k_mx_convert, L.nblk_rows, BS_THREADS, 0, D);
    tend(L, q);
    cudaMemsetAsync(d_nconv, 0, 2 * sizeof(int), L.stream);
    int max_outer = 0;
    cudaMemcpyAsync(h_nconv + 2, &D.par[0].max_outer, sizeof(int), cudaMemcpyDeviceToHost, L.stream);
    cudaStreamSynchronize(L.stream);
    max_outer = h_nconv[2];
    for (int outer = 0; outer <= max_outer; ++outer) {
        float *p = D.fp, *v = D.fv, *p2 = D.fp2, *v2 = D.fv2;   // k_mx_init zeroes fp, fv
        q = tbegin(L, K_MX_RES);
        launch_pdl(L, k_mx_res, L.nblk_rows, BS_THREADS, 0, D, d_nconv);
        tend(L, q);
        cudaMemcpyAsync(h_nconv, d_nconv, 2 * sizeof(int), cudaMemcpyDeviceToHost, L.stream);
        cudaStreamSynchronize(L.stream);
        if (h_nconv[1] >= D.nscene) break;
        cudaMemsetAsync(d_nconv, 0, sizeof(int), L.stream);
        // inner-converged counter starts with the outer-converged scenes
        cudaMemcpyAsync(d_nconv, d_nconv + 1, sizeof(int), cudaMemcpyDeviceToDevice, L.stream);
        q = tbegin(L, K_MX_INIT);
        launch_pdl(L, k_mx_init, L.nblk_rows, BS_THREADS, 0, D, d_nconv);
        tend(L, q);
        int it = 0;
        while (it < maxit) {
            cudaMemcpyAsync(h_nconv, d_nconv, sizeof(int), cudaMemcpyDeviceToHost, L.stream);
            cudaEventRecord(ev, L.stream);
            for (int c = 0; c < check_every && it < maxit; ++c, ++it) {
                q = tbegin(L, K_MX_IT1);
                launch_pdl(L, k_mx_it1, L.nblk_rows, BS_THREADS, 0, D, p, v, p2, v2);
                tend(L, q);
                q = tbegin(L, K_MX_IT2);
                launch_pdl(L, k_mx_it2, L.nblk_rows, BS_THREADS, 0, D, v2);
                tend(L, q);
                q = tbegin(L, K_MX_IT3);
                launch_pdl(L, k_mx_it3, L.nblk_rows, BS_THREADS, 0, D, p2, d_nconv);
                tend(L, q);
                float* t;
                t = p; p = p2; p2 = t;
                t = v; v = v2; v2 = t;
            }
            cudaEventSynchronize(ev);
            timer_collect(L.timer, false);
            if (*h_nconv >= D.nscene) break;
        }
        q = tbegin(L, K_MX_UPD);
        launch_pdl(L, k_mx_update, L.nblk_rows, BS_THREADS, 0, D);
        tend(L, q);
    }
}


// ---------------------------------------------------------------- captured solves
// The solves above check convergence on the host between chunks of
// iterations.  Inside a captured step the loops run on the device instead:
// a conditional while node repeats a chunk of iterations (or columns, or
// restart cycles) for as long as its condition kernel -- one thread, after
// the chunk -- finds a scene that has not converged and the iteration budget
// not spent.  Every loop is bounded by the same maxit / restart length as the
// host loops, so it ends even if no scene converges.

bool cond_handle(cudaStream_t st, unsigned init, cudaGraphConditionalHandle* h) {
    cudaStreamCaptureStatus cs;
    cudaGraph_t g = nullptr;
    if (cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr, nullptr) != cudaSuccess ||
        cs != cudaStreamCaptureStatusActive || !g)
        return false;
    return cudaGraphConditionalHandleCreate(h, g, init, cudaGraphCondAssignDefault) == cudaSuccess;
}

// BiCGStab chunk done: go on while a scene is not converged and it < maxit
__global__ void k_cond_iter(Dev D, const int* nconv, cudaGraphConditionalHandle h, int chunk, int maxit,
                            int body_kernels) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    LoopCtl* C = D.loop;
    C->kernels += (unsigned long long)body_kernels;
    C->it += chunk;
    cudaGraphSetConditional(h, (*nconv < D.nscene && C->it < maxit) ? 1u : 0u);
}

// FGMRES cycle started (k_fg_start ran): the cycle's columns run if a scene
// is not converged; another cycle follows while cycle <= maxit
__global__ void k_cond_cycle(Dev D, const int* nconv, cudaGraphConditionalHandle hloop,
                             cudaGraphConditionalHandle hbody, int maxit, int body_kernels) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    LoopCtl* C = D.loop;
    C->kernels += (unsigned long long)body_kernels;
    const bool go = nconv[1] < D.nscene;
    C->cycle += 1;
    cudaGraphSetConditional(hbody, go ? 1u : 0u);
    cudaGraphSetConditional(hloop, (go && C->cycle <= maxit) ? 1u : 0u);
}

// start of a cycle's columns: column counter 0, the column loop armed
__global__ void k_col_init(Dev D, cudaGraphConditionalHandle h, int body_kernels) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    LoopCtl* C = D.loop;
    C->kernels += (unsigned long long)body_kernels;
    C->col = 0;
    cudaGraphSetConditional(h, 1u);
}

// a chunk of columns done: go on while col < restart length and a scene's cycle is open
__global__ void k_cond_col(Dev D, const int* nconv, cudaGraphConditionalHandle h, int chunk, int body_kernels) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    LoopCtl* C = D.loop;
    C->kernels += (unsigned long long)body_kernels;
    C->col += chunk;
    cudaGraphSetConditional(h, (C->col < D.fg_m && nconv[0] < D.nscene) ? 1u : 0u);
}

namespace {

void bicg_iteration(const Dev& D, const Launch& L, int precond, int mg_prec, int* d_nconv) {
    const double* pu = precond ? D.sp2 : D.sp;
    const double* su = precond ? D.sv2 : D.ss;
    const int mgmode = precond ? (mg_prec == BS_PREC_MIXED ? 2 : 1) : 0;
    int q = tbegin(L, K_BICG_PUPD);
    launch_pdl(L, k_pupd64, L.nblk_rows, BS_THREADS, 0, D, mgmode);
    tend(L, q);
    if (precond) mg_apply(D, L, mg_prec, D.sp, D.sp2, 0);
    q = tbegin(L, K_BICG_IT1);
    launch_pdl(L, k_it1_64, L.nblk_rows, BS_THREADS, 0, D, pu);
    tend(L, q);
    q = tbegin(L, K_BICG_SUPD);
    launch_pdl(L, k_supd64, L.nblk_rows, BS_THREADS, 0, D, mgmode);
    tend(L, q);
    if (precond) mg_apply(D, L, mg_prec, D.ss, D.sv2, 0);
    q = tbegin(L, K_BICG_IT2);
    launch_pdl(L, k_it2_64, L.nblk_rows, BS_THREADS, 0, D, su);
    tend(L, q);
    q = tbegin(L, K_BICG_IT3);
    launch_pdl(L, k_it3_64, L.nblk_rows, BS_THREADS, 0, D, pu, su, d_nconv);
    tend(L, q);
}

void fg_put(const Dev& D, const Launch& L, int mgmode) {
    int q = tbegin(L, K_FG_PUT);
    launch_pdl(L, k_fg_put, L.nblk_rows, BS_THREADS, 0, D, mgmode);
    tend(L, q);
}

void fg_column(const Dev& D, const Launch& L, int precond, int mg_prec, int mgmode, int* d_nconv) {
    if (!D.fg_df) fg_put(D, L, mgmode);
    if (precond) mg_apply(D, L, mg_prec, D.fg_V, D.fg_df ? nullptr : D.sp2, 1);   // (pass 1 of the double-float form reads zf)
    int q = tbegin(L, K_FG_ARN);
    if (D.fg_df) fg_pass1_df(D, L);
    else launch_pdl(L, k_fg_arn1, L.nblk_rows, BS_THREADS, 0, D, precond);
    tend(L, q);
    q = tbegin(L, K_FG_ORTH);
    if (D.fg_df) launch_pdl(L, k_fg_arn2_df, L.nblk_rows + D.nscene, BS_ARN2_THREADS, 0, D, d_nconv, mgmode);
    else launch_pdl(L, k_fg_arn2, L.nblk_rows, BS_THREADS, 0, D, d_nconv, mgmode);
    tend(L, q);
}

void precond_setup(const Dev& D, const Launch& L, int precond, int mg_prec) {
    if (!precond) return;
    if (mg_prec == BS_PREC_MIXED) {
        const int q = tbegin(L, K_MX_CONV);
        launch_pdl(L, k_mx_convert, L.nblk_rows, BS_THREADS, 0, D);
        tend(L, q);
    }
    mg_setup(D, L, mg_prec);
}

Launch on_stream(const Launch& L, cudaStream_t st) {
    Launch B = L;
    B.stream = st;
    return B;
}

}  // namespace

bool capture_fp64(const Dev& D, const Launch& L, const cudaStream_t* side, int maxit, int check_every, int precond,
                  int mg_prec, int* d_nconv) {
    precond_setup(D, L, precond, mg_prec);
    cudaMemsetAsync(d_nconv, 0, sizeof(int), L.stream);
    int q = tbegin(L, K_BICG_INIT);
    launch_pdl(L, k_init64, L.nblk_rows, BS_THREADS, 0, D, d_nconv);
    tend(L, q);
    cudaMemsetAsync(&D.loop->it, 0, sizeof(int), L.stream);
    cudaGraphConditionalHandle h;
    if (!cond_handle(L.stream, 1, &h)) return false;
    const bool ok = cond_node(L.stream, side[0], cudaGraphCondTypeWhile, h, [&]() {
        const Launch B = on_stream(L, side[0]);
        const int64_t b0 = *L.launches;
        for (int c = 0; c < check_every; ++c) bicg_iteration(D, B, precond, mg_prec, d_nconv);
        const int nk = (int)(*L.launches - b0) + 1;
        k_cond_iter<<<1, 32, 0, side[0]>>>(D, d_nconv, h, check_every, maxit, nk);
        *L.launches = b0;   // counted on the device per iteration of the loop
        return cudaGetLastError() == cudaSuccess;
    });
    q = tbegin(L, K_TRUERES);
    launch_pdl(L, k_true_res64, L.nblk_rows, BS_THREADS, 0, D);
    tend(L, q);
    return ok;
}

bool capture_fgmres(const Dev& D, const Launch& L, const cudaStream_t* side, int maxit, int check_every,
                    int precond, int mg_prec, int* d_nconv) {
    precond_setup(D, L, precond, mg_prec);
    const int mgmode = precond ? (mg_prec == BS_PREC_MIXED ? 2 : 1) : 0;
    cudaMemsetAsync(d_nconv, 0, 2 * sizeof(int), L.stream);
    cudaMemsetAsync(&D.loop->cycle, 0, sizeof(int), L.stream);
    cudaGraphConditionalHandle hc, hif, hcol;
    if (!cond_handle(L.stream, 1, &hc)) return false;
    const bool ok = cond_node(L.stream, side[0], cudaGraphCondTypeWhile, hc, [&]() {
        // one restart cycle: start (true residual, norms), then its columns
        const Launch B0 = on_stream(L, side[0]);
        const int64_t b0 = *L.launches;
        cudaMemcpyAsync(d_nconv, d_nconv + 1, sizeof(int), cudaMemcpyDeviceToDevice, side[0]);
        int q0 = tbegin(B0, K_FG_START);
        launch_pdl(B0, k_fg_start, L.nblk_rows, BS_THREADS, 0, D, 0, d_nconv, (const int*)&D.loop->cycle);
        tend(B0, q0);
        if (!cond_handle(side[0], 0, &hif)) return false;
        k_cond_cycle<<<1, 32, 0, side[0]>>>(D, d_nconv, hc, hif, maxit, 2);
        const bool ok1 = cond_node(side[0], side[1], cudaGraphCondTypeIf, hif, [&]() {
            const Launch B1 = on_stream(L, side[1]);
            if (D.fg_df) fg_put(D, B1, mgmode);
            if (!cond_handle(side[1], 1, &hcol)) return false;
            // the cycle's own kernels: put (double-float basis), this one, the solve and the update
            k_col_init<<<1, 32, 0, side[1]>>>(D, hcol, (D.fg_df ? 1 : 0) + 3);
            const bool ok2 = cond_node(side[1], side[2], cudaGraphCondTypeWhile, hcol, [&]() {
                const Launch B2 = on_stream(L, side[2]);
                const int64_t b2 = *L.launches;
                for (int c = 0; c < check_every; ++c) fg_column(D, B2, precond, mg_prec, mgmode, d_nconv);
                const int nk = (int)(*L.launches - b2) + 1;
                k_cond_col<<<1, 32, 0, side[2]>>>(D, d_nconv, hcol, check_every, nk);
                *L.launches = b2;
                return cudaGetLastError() == cudaSuccess;
            });
            int q1 = tbegin(B1, K_FG_UPD);
            launch_pdl(B1, k_fg_solve, D.nscene, 32, 0, D, d_nconv);
            launch_pdl(B1, k_fg_update, L.nblk_rows, BS_THREADS, 0, D, precond);
            tend(B1, q1);
            return ok2 && cudaGetLastError() == cudaSuccess;
        });
        *L.launches = b0;
        return ok1 && cudaGetLastError() == cudaSuccess;
    });
    int q = tbegin(L, K_TRUERES);
    launch_pdl(L, k_true_res64, L.nblk_rows, BS_THREADS, 0, D);
    tend(L, q);
    return ok;
}

// scalar sub-step pairs of the captured step
__global__ void k_cond_scalar(Dev D, cudaGraphConditionalHandle h, int body_kernels) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    LoopCtl* C = D.loop;
    C->kernels += (unsigned long long)body_kernels;
    C->j += 2;
    int mx = 1;
    for (int s = 0; s < D.nscene; ++s) mx = max(mx, D.dyn[s].solsteps);
    // the same sub-step count as the host loop (bounded: solsteps is finite)
    cudaGraphSetConditional(h, C->j < mx ? 1u : 0u);
}

void cond_scalar(const Dev& D, cudaStream_t st, cudaGraphConditionalHandle h, int body_kernels) {
    k_cond_scalar<<<1, 32, 0, st>>>(D, h, body_kernels);
}

}  // namespace bs
