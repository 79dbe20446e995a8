// bs_static.cu -- BiCGStab on a caller-owned device CSR system that
// allocates nothing.
//
// Some callers cannot let a library call cudaMalloc/cudaFree: hosts whose
// device memory is owned by their own pool allocator (a framework that
// reserves HBM up front and forbids third-party allocations), or code that
// must not stall -- cudaMalloc and cudaFree may synchronise the device and
// take unbounded time.  This entry point keeps all of its solver scratch
// (the six Krylov vectors, block partial sums and the scalars) in one
// file-scope device array of fixed size, so a call only launches kernels and
// copies a few scalars back to the host.
//
// Limits and rules:
//  * n <= BS_STATIC_MAX_ROWS (65,536) rows; larger systems are rejected with
//    BS_E_CAPACITY before any work.
//  * The array (about 3.2 MB) is part of the library's device image: every
//    GPU that loads the library holds it until the process exits.
//  * Every call shares the array and it keeps the last call's contents; each
//    call clears what must start at zero (p, v, the converged flag).  Calls
//    whose work overlaps on the GPU (different streams, or host threads
//    without ordering) race on the array: serialise them.
//  * The device address of the array is looked up with cudaGetSymbolAddress
//    on the first call on each device (that device current) and cached; make
//    that first call before any stream capture begins.
//  * Convergence is judged on the recursive residual, as bs_bicgstab_csr
//    judges it; *relres reports the true residual ||b - A x|| / ||b||
//    computed after the last iteration.  The flag is read back to the host
//    every BS_STATIC_CHUNK iterations (the call waits for its stream there),
//    so the call cannot run on a stream that is being captured.
//  * The iterations are one cooperative launch, which starts when all of its
//    blocks (one per 256 rows, up to 204 KB of shared memory each) fit on the
//    device at once: beside other streams' kernels it waits for theirs to end.
//    Where such a launch is refused (a partition of the device, a green context)
//    the phases of an iteration are launches of their own.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "bs_internal.cuh"

#define BS_STATIC_MAX_ROWS 65536
#define BS_STATIC_THREADS 256
#define BS_STATIC_MAX_BLOCKS (BS_STATIC_MAX_ROWS / BS_STATIC_THREADS)
#define BS_STATIC_NPART 4
#define BS_STATIC_CHUNK 256   // iterations of one launch

// scratch layout (doubles): r, rhat, p, v, s, t [MAX_ROWS each] |
// partials [2 sets of MAX_BLOCKS * NPART] | scalars [32] (the last 8: the grid barrier)
#define BS_STATIC_VEC (6L * BS_STATIC_MAX_ROWS)
#define BS_STATIC_WORDS (BS_STATIC_VEC + 2 * BS_STATIC_MAX_BLOCKS * BS_STATIC_NPART + 32)

static __device__ __align__(256) double bs_static_scratch[BS_STATIC_WORDS];

namespace {

// scalar slots
enum { S_RHO = 0, S_ALPHA, S_OMEGA, S_BETA, S_BNORM2, S_RNORM2, S_CONV, S_ITERS, S_RTRUE2, S_BREAK };

struct Csr {
    int n;
    const int* rp;
    const int* col;
    const double* val;
};

struct Scr {
    double *r, *rh, *p, *v, *s, *t, *part, *sc;
};

__host__ __device__ inline Scr carve(double* base) {
    Scr q;
    q.r = base;
    q.rh = base + BS_STATIC_MAX_ROWS;
    q.p = base + 2L * BS_STATIC_MAX_ROWS;
    q.v = base + 3L * BS_STATIC_MAX_ROWS;
    q.s = base + 4L * BS_STATIC_MAX_ROWS;
    q.t = base + 5L * BS_STATIC_MAX_ROWS;
    q.part = base + BS_STATIC_VEC;
    q.sc = q.part + 2 * BS_STATIC_MAX_BLOCKS * BS_STATIC_NPART;
    return q;
}

// One cooperative launch runs the whole solve (up to `chunk` iterations): the
// blocks hold 256 rows each, cross a grid barrier where a product needs a
// vector's neighbours or a dot is summed (five per iteration), and keep their
// rows of the matrix in shared memory and of the vectors in registers.  Measured
// at 60,025 rows of 21 entries: 61 us per iteration with a launch per phase
// (eight, the sums by a block of their own), 25 now; 19 at 9,801 rows, 15 at 30.
// Bound now by latencies: the five barriers (1 to 1.7 us each), six
// block sums, three divisions (0.4 us each), and the FP64 pipe (2 x 21 fused
// multiply-adds per row at 16 cycles per warp, two blocks on an SM at 60,025
// rows: 6 us).  Every sum runs in the order of the launch-per-phase form (256-row
// blocks, then the blocks by 256 threads), with the products fused alike: the
// iterates are the same.
struct Grid {
    unsigned* count;    // arrivals, counted up over the launch
    unsigned* broken;   // 1: a wait ran out (the launch gives up)
    unsigned target;
};
// all blocks' writes before it are visible to all blocks after it; false: gave
// up.  The block barriers order the block's accesses before thread 0's release
// and after its acquire (which also drops the SM's stale L1 lines).
__device__ __forceinline__ bool grid_barrier(Grid& G) {
    __shared__ int ok;
    __syncthreads();
    if (gridDim.x == 1) return true;
    G.target += gridDim.x;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(G.count) : "memory");
        unsigned now = 0;
        int left = 1 << 21;   // bounded: a wait of a second or two
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(G.count) : "memory");
        } while ((int)(now - G.target) < 0 && --left > 0);
        ok = left > 0;
        if (!ok) atomicExch(G.broken, 1u);
    }
    __syncthreads();
    return ok != 0;
}

// block_sum of two values over the block's 256 threads by one warp, in block_sum's
// order (halves over 16, 8, 4, 2, 1 lanes, then over the warps): two lanes hold a
// warp's values and add them without exchanges, so 15 + 1 + 3 FP64 instructions
// instead of 90 (one holds the SM's FP64 pipe for 16 cycles) and a chain of four
// shuffled adds instead of eight.  Warp 0 returns true and has the sums.
// Rows of 34: the 16 lanes of a 64-bit read fall into 16 bank pairs.
constexpr int SUM_LD = 34;
__device__ __forceinline__ bool sum2(double (&q)[2], double* buf /*[16 * SUM_LD]*/) {
    const int t = threadIdx.x, lane = t & 31;
    buf[(t >> 5) * SUM_LD + lane] = q[0];
    buf[(8 + (t >> 5)) * SUM_LD + lane] = q[1];
    __syncthreads();
    if (t >= 32) return false;
    const double* in = buf + (lane >> 1) * SUM_LD + (lane & 1);
    double x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = in[2 * k];
#pragma unroll
    for (int m = 8; m > 0; m >>= 1)
#pragma unroll
        for (int k = 0; k < m; ++k) x[k] += x[k + m];
    double v = x[0];   // lane 16 q + 2 w (+ 1): value q, warp w
#pragma unroll
    for (int o : {1, 8, 4, 2}) v += __shfl_xor_sync(0xffffffffu, v, o);
    q[0] = __shfl_sync(0xffffffffu, v, 0);
    q[1] = __shfl_sync(0xffffffffu, v, 16);
    return true;
}

__global__ void __launch_bounds__(BS_STATIC_THREADS) ks_solve(Csr A, const double* b, double* x, double* base, int nblk,
                                                             double tol, int maxit, int chunk, int first, int cap) {
    constexpr int NT = BS_STATIC_THREADS;
    extern __shared__ __align__(16) unsigned char rows_smem[];
    __shared__ double sh[2][16 * SUM_LD], sc[16], ratio;
    __shared__ int rp[NT + 1];
    const Scr S = carve(base);
    double* const sval = (double*)rows_smem;
    int* const scol = (int*)(sval + cap);
    const int t = threadIdx.x;
    // the block's rows of the matrix into shared memory (if they fit)
    const int i0 = blockIdx.x * NT;
    const int nr = min(NT, A.n - i0);
    for (int k = t; k <= nr; k += NT) rp[k] = A.rp[i0 + k];
    __syncthreads();
    const int e0 = rp[0], ne = rp[nr] - e0;
    const bool held = ne <= cap;
    if (held)
        for (int e = t; e < ne; e += NT) {
            sval[e] = A.val[e0 + e];
            scol[e] = A.col[e0 + e];
        }
    Grid G{(unsigned*)(S.sc + 24), (unsigned*)(S.sc + 25), 0};
    if (t < 16) sc[t] = S.sc[t];
    __syncthreads();
    const int i = i0 + t;   // this thread's row
    const bool in = i < A.n;
    // (A u)_i; twelve gathers in flight, the sum in entry order
    auto row = [&](const double* u) {
        constexpr int B = 12;
        double acc = 0.0;
        if (held) {
            const int end = rp[t + 1] - e0;
            for (int e = rp[t] - e0; e < end; e += B) {
                double ue[B];
#pragma unroll
                for (int k = 0; k < B; ++k) ue[k] = e + k < end ? u[scol[e + k]] : 0.0;
#pragma unroll
                for (int k = 0; k < B; ++k)
                    if (e + k < end) acc = __fma_rn(sval[e + k], ue[k], acc);
            }
        } else {
            for (int e = A.rp[i]; e < A.rp[i + 1]; ++e) acc = __fma_rn(A.val[e], u[A.col[e]], acc);
        }
        return acc;
    };
    // the block's sums of q[]: partials of phase k's set (two sets: a block may be one barrier ahead)
    int phase = 0;
    auto partial = [&](double (&q)[2]) {
        if (sum2(q, sh[0]) && t == 0) {
            double* p = S.part + ((long)(phase & 1) * BS_STATIC_MAX_BLOCKS + blockIdx.x) * BS_STATIC_NPART;
            p[0] = q[0];
            p[1] = q[1];
        }
    };
    // the barrier, then the sums over the blocks
    auto total = [&](double (&a)[2]) {
        if (!grid_barrier(G)) return false;
        a[0] = a[1] = 0.0;
        const double* p = S.part + (long)(phase & 1) * BS_STATIC_MAX_BLOCKS * BS_STATIC_NPART;
        for (int k = t; k < nblk; k += NT) {
            a[0] += __ldcg(p + k * BS_STATIC_NPART);
            a[1] += __ldcg(p + k * BS_STATIC_NPART + 1);
        }
        sum2(a, sh[1]);   // thread 0 has them
        ++phase;
        return true;
    };
    double r = 0.0, rh = 0.0, p = 0.0, v = 0.0, s = 0.0, w = 0.0, xi = 0.0;
    if (in) {
        xi = x[i];
        if (!first) {
            r = S.r[i];
            rh = S.rh[i];
            p = S.p[i];
            v = S.v[i];
        }
    }
    double a[2];
    if (first) {
        double q[2] = {0.0, 0.0};
        if (in) {
            const double bi = b[i];
            r = rh = bi - row(x);
            S.rh[i] = rh;
            q[0] = __dmul_rn(bi, bi);
            q[1] = __dmul_rn(r, r);
        }
        partial(q);
        if (!total(a)) return;
        if (t == 0) {
            sc[S_BNORM2] = a[0];
            sc[S_RNORM2] = a[1];
            sc[S_RHO] = a[1];
            sc[S_ALPHA] = 1.0;
            sc[S_OMEGA] = 1.0;
            sc[S_BETA] = 0.0;
            sc[S_ITERS] = 0.0;
            sc[S_BREAK] = 0.0;
            sc[S_CONV] = (a[0] == 0.0 || a[1] <= tol * tol * a[0]) ? 1.0 : 0.0;
        }
        __syncthreads();
    }
    for (int it = 0; it < chunk && sc[S_CONV] == 0.0; ++it) {
        const double beta = sc[S_BETA], omega0 = sc[S_OMEGA];
        if (in) S.p[i] = p = __fma_rn(beta, __fma_rn(-omega0, v, p), r);
        if (!grid_barrier(G)) return;
        double q[2] = {0.0, 0.0};
        if (in) {   // v = A p, (rh, v) -> alpha
            v = row(S.p);
            q[0] = __dmul_rn(rh, v);
        }
        partial(q);
        if (!total(a)) return;
        if (t == 0) {
            if (a[0] == 0.0 || !isfinite(a[0])) {
                sc[S_BREAK] = 1.0;
                sc[S_ALPHA] = 0.0;
            } else {
                sc[S_ALPHA] = sc[S_RHO] / a[0];
            }
        }
        __syncthreads();
        const double alpha = sc[S_ALPHA];
        if (in) S.s[i] = s = __fma_rn(-alpha, v, r);
        if (!grid_barrier(G)) return;
        q[0] = q[1] = 0.0;
        if (in) {   // t = A s, (t, s) and (t, t) -> omega
            w = row(S.s);
            q[0] = __dmul_rn(w, s);
            q[1] = __dmul_rn(w, w);
        }
        partial(q);
        if (!total(a)) return;
        if (t == 0) {
            sc[S_OMEGA] = (a[1] != 0.0) ? a[0] / a[1] : 0.0;
            if (a[1] == 0.0) sc[S_BREAK] = 1.0;
        }
        __syncthreads();
        const double omega = sc[S_OMEGA];
        if (t == NT - 1) ratio = alpha / omega;   // (beside the other warps; a division takes 500 cycles)
        q[0] = q[1] = 0.0;
        if (in) {   // x, r; (rh, r) and (r, r) -> beta, the stopping test
            xi = __fma_rn(omega, s, __fma_rn(alpha, p, xi));
            r = __fma_rn(-omega, w, s);
            q[0] = __dmul_rn(rh, r);
            q[1] = __dmul_rn(r, r);
        }
        partial(q);
        if (!total(a)) return;
        if (t == 0) {
            sc[S_BETA] = __dmul_rn(a[0] / sc[S_RHO], ratio);
            sc[S_RHO] = a[0];
            sc[S_RNORM2] = a[1];
            sc[S_ITERS] += 1.0;
            const bool conv = a[1] <= tol * tol * sc[S_BNORM2] || !isfinite(a[1]) || sc[S_BREAK] != 0.0 ||
                              sc[S_ITERS] >= (double)maxit;
            sc[S_CONV] = conv ? 1.0 : 0.0;
        }
        __syncthreads();
    }
    if (in) {
        x[i] = xi;
        S.r[i] = r;
        S.v[i] = v;
    }
    if (sc[S_CONV] != 0.0) {   // the true residual
        if (!grid_barrier(G)) return;
        double q[2] = {0.0, 0.0};
        if (in) {
            const double ri = b[i] - row(x);
            q[0] = __dmul_rn(ri, ri);
        }
        partial(q);
        if (!total(a)) return;
        if (t == 0) sc[S_RTRUE2] = a[0];
    }
    __syncthreads();
    if (blockIdx.x == 0 && t < 16) S.sc[t] = sc[t];
}

// ---- launch per phase: where the cooperative launch is not to be had (fewer
// resident blocks than row blocks: a partition of the device, a green context).
// It resumes from what ks_solve leaves between its launches (r, rhat, p, v, the
// scalars), and gives the same iterates.
__device__ __forceinline__ double csr_row(const Csr& A, const double* __restrict__ u, int i) {
    double acc = 0.0;
    for (int e = A.rp[i]; e < A.rp[i + 1]; ++e) acc += A.val[e] * u[A.col[e]];
    return acc;
}

template <int NV>
__device__ __forceinline__ void block_partials(double (&v)[NV], double* part) {
    __shared__ double sh[NV * 32];
    block_sum<NV>(v, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) part[blockIdx.x * BS_STATIC_NPART + q] = v[q];
}

__device__ __forceinline__ bool done(const Scr& S) { return S.sc[S_CONV] != 0.0; }

__global__ void ks_init(Csr A, const double* __restrict__ b, const double* __restrict__ x, double* base) {
    const Scr S = carve(base);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (i < A.n) {
        const double ri = b[i] - csr_row(A, x, i);
        S.r[i] = ri;
        S.rh[i] = ri;
        S.p[i] = 0.0;
        S.v[i] = 0.0;
        q[0] = b[i] * b[i];
        q[1] = ri * ri;
    }
    block_partials<2>(q, S.part);
}

// single block: sum the partials in block order and update the scalars
__global__ void ks_reduce(int nblk, int phase, double tol, int maxit, double* base) {
    const Scr S = carve(base);
    // the host launches iterations in groups: once a solve has converged the
    // iteration phases of the rest of the group leave every scalar (and the
    // iteration count) as they are; the flag is read by the whole block, so
    // the early return is uniform
    if (phase >= 1 && phase <= 3 && S.sc[S_CONV] != 0.0) return;
    __shared__ double sh[3 * 32];
    double a[3] = {0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < nblk; b += blockDim.x)
        for (int q = 0; q < 3; ++q) a[q] += S.part[b * BS_STATIC_NPART + q];
    block_sum<3>(a, sh);
    if (threadIdx.x != 0) return;
    double* sc = S.sc;
    if (phase == 0) {   // init: (b,b), (r,r)
        sc[S_BNORM2] = a[0];
        sc[S_RNORM2] = a[1];
        sc[S_RHO] = a[1];
        sc[S_ALPHA] = 1.0;
        sc[S_OMEGA] = 1.0;
        sc[S_BETA] = 0.0;
        sc[S_ITERS] = 0.0;
        sc[S_BREAK] = 0.0;
        sc[S_CONV] = (a[0] == 0.0 || a[1] <= tol * tol * a[0]) ? 1.0 : 0.0;
    } else if (phase == 1) {   // (rhat, v) -> alpha
        if (a[0] == 0.0 || !isfinite(a[0])) {
            sc[S_BREAK] = 1.0;
            sc[S_ALPHA] = 0.0;
        } else {
            sc[S_ALPHA] = sc[S_RHO] / a[0];
        }
    } else if (phase == 2) {   // (t,s), (t,t) -> omega
        sc[S_OMEGA] = (a[1] != 0.0) ? a[0] / a[1] : 0.0;
        if (a[1] == 0.0) sc[S_BREAK] = 1.0;
    } else if (phase == 3) {   // (rhat, r), (r,r) -> beta, convergence
        sc[S_BETA] = (a[0] / sc[S_RHO]) * (sc[S_ALPHA] / sc[S_OMEGA]);
        sc[S_RHO] = a[0];
        sc[S_RNORM2] = a[1];
        sc[S_ITERS] += 1.0;
        const bool conv = a[1] <= tol * tol * sc[S_BNORM2] || !isfinite(a[1]) || sc[S_BREAK] != 0.0 ||
                          sc[S_ITERS] >= (double)maxit;
        sc[S_CONV] = conv ? 1.0 : 0.0;
    } else {   // true residual
        sc[S_RTRUE2] = a[0];
    }
}

__global__ void ks_p(Csr A, double* base) {
    const Scr S = carve(base);
    if (done(S)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    S.p[i] = S.r[i] + S.sc[S_BETA] * (S.p[i] - S.sc[S_OMEGA] * S.v[i]);
}

__global__ void ks_v(Csr A, double* base) {
    const Scr S = carve(base);
    if (done(S)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double q[1] = {0.0};
    if (i < A.n) {
        const double vi = csr_row(A, S.p, i);
        S.v[i] = vi;
        q[0] = S.rh[i] * vi;
    }
    block_partials<1>(q, S.part);
}

__global__ void ks_s(Csr A, double* base) {
    const Scr S = carve(base);
    if (done(S)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.n) return;
    S.s[i] = S.r[i] - S.sc[S_ALPHA] * S.v[i];
}

__global__ void ks_t(Csr A, double* base) {
    const Scr S = carve(base);
    if (done(S)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (i < A.n) {
        const double ti = csr_row(A, S.s, i);
        S.t[i] = ti;
        q[0] = ti * S.s[i];
        q[1] = ti * ti;
    }
    block_partials<2>(q, S.part);
}

__global__ void ks_x(Csr A, double* __restrict__ x, double* base) {
    const Scr S = carve(base);
    if (done(S)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double q[2] = {0.0, 0.0};
    if (i < A.n) {
        const double a = S.sc[S_ALPHA], w = S.sc[S_OMEGA];
        x[i] = x[i] + a * S.p[i] + w * S.s[i];
        const double ri = S.s[i] - w * S.t[i];
        S.r[i] = ri;
        q[0] = S.rh[i] * ri;
        q[1] = ri * ri;
    }
    block_partials<2>(q, S.part);
}

__global__ void ks_true(Csr A, const double* __restrict__ b, const double* __restrict__ x, double* base) {
    const Scr S = carve(base);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double q[1] = {0.0};
    if (i < A.n) {
        const double ri = b[i] - csr_row(A, x, i);
        q[0] = ri * ri;
    }
    block_partials<1>(q, S.part);
}

// device address of the scratch array, looked up once per device
std::mutex g_mu;
double* g_addr[64] = {};

int scratch_for_current_device(double** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BS_E_CUDA;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, bs_static_scratch);
        if (e != cudaSuccess || !p) return BS_E_CUDA;
        g_addr[dev] = (double*)p;
    }
    *out = g_addr[dev];
    return BS_OK;
}

}  // namespace

// form 0: one cooperative launch where it is to be had; 1: the launches per phase
static int solve_noalloc(int32_t n, const int32_t* d_row_ptr, const int32_t* d_col, const double* d_val,
                         const double* d_b, double* d_x, double tol, int32_t maxit, void* stream, int32_t* iters,
                         double* relres, int form) {
    if (n <= 0 || !d_row_ptr || !d_col || !d_val || !d_b || !d_x || maxit <= 0 || !(tol >= 0.0)) return BS_E_ARG;
    if (n > BS_STATIC_MAX_ROWS) return BS_E_CAPACITY;
    double* base = nullptr;
    int rc = scratch_for_current_device(&base);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const Csr A{n, d_row_ptr, d_col, d_val};
    const int nb = (n + BS_STATIC_THREADS - 1) / BS_STATIC_THREADS;
    // entries of the matrix a block can hold: two blocks share an SM when there are more blocks than SMs
    int dev = 0, sms = 0, per = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return BS_E_CUDA;
    const int most = 17000, cap = nb <= sms ? most : 8000, smem = cap * 12;
    // (the kernel's limit is the same on every call: calls of other sizes may be running)
    bool coop = form == 0 &&
                cudaFuncSetAttribute(ks_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, most * 12) == cudaSuccess &&
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ks_solve, BS_STATIC_THREADS, smem) == cudaSuccess;
    if (form == 0 && !coop) cudaGetLastError();
    if ((long)per * sms < nb) coop = false;
    double sc[32];
    const Scr S = carve(base);
    int first = 1, chunk = BS_STATIC_CHUNK;
    for (long it = 0;;) {
        if (coop) {
            if (cudaMemsetAsync(S.sc + 24, 0, 2 * sizeof(double), st) != cudaSuccess) return BS_E_CUDA;
            void* args[] = {(void*)&A, (void*)&d_b, (void*)&d_x, (void*)&base, (void*)&nb, (void*)&tol, (void*)&maxit,
                            (void*)&chunk, (void*)&first, (void*)&cap};
            if (cudaLaunchCooperativeKernel((const void*)ks_solve, dim3(nb), dim3(BS_STATIC_THREADS), args, smem, st) !=
                cudaSuccess) {   // (the stream's share of the device is smaller than the device)
                cudaGetLastError();
                coop = false;
                continue;
            }
            it += chunk;
        } else {
            if (first) {
                ks_init<<<nb, BS_STATIC_THREADS, 0, st>>>(A, d_b, d_x, base);
                ks_reduce<<<1, 256, 0, st>>>(nb, 0, tol, maxit, base);
            }
            // check every 4 iterations; kernels of a converged solve return at once
            for (int c = 0; c < 4; ++c, ++it) {
                ks_p<<<nb, BS_STATIC_THREADS, 0, st>>>(A, base);
                ks_v<<<nb, BS_STATIC_THREADS, 0, st>>>(A, base);
                ks_reduce<<<1, 256, 0, st>>>(nb, 1, tol, maxit, base);
                ks_s<<<nb, BS_STATIC_THREADS, 0, st>>>(A, base);
                ks_t<<<nb, BS_STATIC_THREADS, 0, st>>>(A, base);
                ks_reduce<<<1, 256, 0, st>>>(nb, 2, tol, maxit, base);
                ks_x<<<nb, BS_STATIC_THREADS, 0, st>>>(A, d_x, base);
                ks_reduce<<<1, 256, 0, st>>>(nb, 3, tol, maxit, base);
            }
        }
        if (cudaMemcpyAsync(sc, S.sc, sizeof(sc), cudaMemcpyDeviceToHost, st) != cudaSuccess) return BS_E_CUDA;
        if (cudaStreamSynchronize(st) != cudaSuccess) return BS_E_CUDA;
        unsigned broken = 0;
        if (coop) std::memcpy(&broken, sc + 25, sizeof(broken));
        if (broken) return BS_E_CUDA;   // a block's wait for the others ran out
        first = 0;
        if (sc[S_CONV] != 0.0 || it >= maxit) break;
    }
    if (!coop) {
        ks_true<<<nb, BS_STATIC_THREADS, 0, st>>>(A, d_b, d_x, base);
        ks_reduce<<<1, 256, 0, st>>>(nb, 4, tol, maxit, base);
        if (cudaMemcpyAsync(sc, S.sc, sizeof(sc), cudaMemcpyDeviceToHost, st) != cudaSuccess) return BS_E_CUDA;
        if (cudaStreamSynchronize(st) != cudaSuccess) return BS_E_CUDA;
    }
    if (cudaGetLastError() != cudaSuccess) return BS_E_CUDA;
    if (iters) *iters = (int32_t)sc[S_ITERS];
    if (relres) *relres = sc[S_BNORM2] > 0.0 ? std::sqrt(sc[S_RTRUE2] / sc[S_BNORM2]) : std::sqrt(sc[S_RTRUE2]);
    const bool ok = sc[S_BNORM2] == 0.0 || sc[S_RNORM2] <= tol * tol * sc[S_BNORM2];
    return ok ? BS_OK : BS_E_NOTCONV;
}

extern "C" int bs_bicgstab_csr_noalloc(int32_t n, const int32_t* d_row_ptr, const int32_t* d_col,
                                       const double* d_val, const double* d_b, double* d_x, double tol,
                                       int32_t maxit, void* stream, int32_t* iters, double* relres) {
    return solve_noalloc(n, d_row_ptr, d_col, d_val, d_b, d_x, tol, maxit, stream, iters, relres, 0);
}

// the launches per phase on any device (not in the public header: their tests)
extern "C" int bs_bicgstab_csr_noalloc_phases(int32_t n, const int32_t* d_row_ptr, const int32_t* d_col,
                                              const double* d_val, const double* d_b, double* d_x, double tol,
                                              int32_t maxit, void* stream, int32_t* iters, double* relres) {
    return solve_noalloc(n, d_row_ptr, d_col, d_val, d_b, d_x, tol, maxit, stream, iters, relres, 1);
}
