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
//
// With fewer resident blocks than row blocks (a device shared out) a block takes
// several in turn, its vectors in memory.
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

template <bool ONE>
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
    // the block's first rows of the matrix into shared memory (if they fit)
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
    // (A u)_i, i = vb * NT + t; twelve gathers in flight, the sum in entry order
    auto row = [&](int vb, const double* u) {
        constexpr int B = 12;
        double acc = 0.0;
        const int i = vb * NT + t;
        if (held && (ONE || vb == (int)blockIdx.x)) {
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
    // the sums of q[] over a row block: partials of phase k's set (two sets: a block may be one barrier ahead)
    int phase = 0;
    auto partial = [&](int vb, double (&q)[2]) {
        if (!ONE) __syncthreads();   // sh[0] is read of the row block before
        if (sum2(q, sh[0]) && t == 0) {
            double* p = S.part + ((long)(phase & 1) * BS_STATIC_MAX_BLOCKS + vb) * BS_STATIC_NPART;
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
    double r = 0.0, rh = 0.0, p = 0.0, v = 0.0, s = 0.0, w = 0.0, xi = 0.0;   // ONE: this thread's row
    const int ir = i0 + t;
    const bool in1 = ir < A.n;
    if (ONE && in1) {
        xi = x[ir];
        if (!first) {
            r = S.r[ir];
            rh = S.rh[ir];
            p = S.p[ir];
            v = S.v[ir];
        }
    }
#define FOR_ROWS                                                    \
    for (int vb = blockIdx.x; vb < nblk; vb += gridDim.x)           \
        for (int i = vb * NT + t, in = i < A.n, go = 1; go; go = 0)
    double a[2];
    if (first) {
        FOR_ROWS {
            double q[2] = {0.0, 0.0};
            if (in) {
                const double bi = b[i];
                const double ri = bi - row(vb, x);
                S.r[i] = ri;
                S.rh[i] = ri;
                S.p[i] = 0.0;
                S.v[i] = 0.0;
                if (ONE) r = rh = ri;
                q[0] = __dmul_rn(bi, bi);
                q[1] = __dmul_rn(ri, ri);
            }
            partial(vb, q);
        }
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
        FOR_ROWS if (in) {
            if (ONE) p = __fma_rn(beta, __fma_rn(-omega0, v, p), r);
            S.p[i] = ONE ? p : __fma_rn(beta, __fma_rn(-omega0, S.v[i], S.p[i]), S.r[i]);
        }
        if (!grid_barrier(G)) return;
        FOR_ROWS {   // v = A p, (rh, v) -> alpha
            double q[2] = {0.0, 0.0};
            if (in) {
                const double vi = row(vb, S.p);
                if (ONE) v = vi;
                else S.v[i] = vi;
                q[0] = __dmul_rn(ONE ? rh : S.rh[i], vi);
            }
            partial(vb, q);
        }
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
        FOR_ROWS if (in) {
            if (ONE) s = __fma_rn(-alpha, v, r);
            S.s[i] = ONE ? s : __fma_rn(-alpha, S.v[i], S.r[i]);
        }
        if (!grid_barrier(G)) return;
        FOR_ROWS {   // t = A s, (t, s) and (t, t) -> omega
            double q[2] = {0.0, 0.0};
            if (in) {
                const double ti = row(vb, S.s);
                if (ONE) w = ti;
                else S.t[i] = ti;
                q[0] = __dmul_rn(ti, ONE ? s : S.s[i]);
                q[1] = __dmul_rn(ti, ti);
            }
            partial(vb, q);
        }
        if (!total(a)) return;
        if (t == 0) {
            sc[S_OMEGA] = (a[1] != 0.0) ? a[0] / a[1] : 0.0;
            if (a[1] == 0.0) sc[S_BREAK] = 1.0;
        }
        __syncthreads();
        const double omega = sc[S_OMEGA];
        if (t == NT - 1) ratio = alpha / omega;   // (beside the other warps; a division takes 500 cycles)
        FOR_ROWS {   // x, r; (rh, r) and (r, r) -> beta, the stopping test
            double q[2] = {0.0, 0.0};
            if (in) {
                const double si = ONE ? s : S.s[i];
                if (ONE) xi = __fma_rn(omega, s, __fma_rn(alpha, p, xi));
                else x[i] = __fma_rn(omega, si, __fma_rn(alpha, S.p[i], x[i]));
                const double ri = __fma_rn(-omega, ONE ? w : S.t[i], si);
                if (ONE) r = ri;
                else S.r[i] = ri;
                q[0] = __dmul_rn(ONE ? rh : S.rh[i], ri);
                q[1] = __dmul_rn(ri, ri);
            }
            partial(vb, q);
        }
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
    if (ONE && in1) {
        x[ir] = xi;
        S.r[ir] = r;
        S.v[ir] = v;
    }
    if (sc[S_CONV] != 0.0) {   // the true residual
        if (!grid_barrier(G)) return;
        FOR_ROWS {
            double q[2] = {0.0, 0.0};
            if (in) {
                const double ri = b[i] - row(vb, x);
                q[0] = __dmul_rn(ri, ri);
            }
            partial(vb, q);
        }
        if (!total(a)) return;
        if (t == 0) sc[S_RTRUE2] = a[0];
    }
#undef FOR_ROWS
    __syncthreads();
    if (blockIdx.x == 0 && t < 16) S.sc[t] = sc[t];
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

extern "C" int bs_bicgstab_csr_noalloc(int32_t n, const int32_t* d_row_ptr, const int32_t* d_col,
                                       const double* d_val, const double* d_b, double* d_x, double tol,
                                       int32_t maxit, void* stream, int32_t* iters, double* relres) {
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
    const int cap = nb <= sms ? 17000 : 8000, smem = cap * 12;
    auto most = [&](auto kernel) {   // resident blocks of the kernel
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
               cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, BS_STATIC_THREADS, smem) == cudaSuccess;
    };
    if (!most(ks_solve<true>)) return BS_E_CUDA;
    const bool one = (long)per * sms >= nb;
    if (!one && !most(ks_solve<false>)) return BS_E_CUDA;
    int grid = (int)std::min<long>(nb, (long)per * sms);
    if (grid < 1) return BS_E_CUDA;
    double sc[32];
    const Scr S = carve(base);
    int first = 1, chunk = BS_STATIC_CHUNK;
    while (true) {
        if (cudaMemsetAsync(S.sc + 24, 0, 2 * sizeof(double), st) != cudaSuccess) return BS_E_CUDA;
        void* args[] = {(void*)&A, (void*)&d_b, (void*)&d_x, (void*)&base, (void*)&nb, (void*)&tol, (void*)&maxit,
                        (void*)&chunk, (void*)&first, (void*)&cap};
        if (cudaLaunchCooperativeKernel(one ? (const void*)ks_solve<true> : (const void*)ks_solve<false>, dim3(grid),
                                        dim3(BS_STATIC_THREADS), args, smem, st) != cudaSuccess)
            return BS_E_CUDA;
        if (cudaMemcpyAsync(sc, S.sc, sizeof(sc), cudaMemcpyDeviceToHost, st) != cudaSuccess) return BS_E_CUDA;
        if (cudaStreamSynchronize(st) != cudaSuccess) return BS_E_CUDA;
        unsigned broken;
        std::memcpy(&broken, sc + 25, sizeof(broken));
        if (broken) return BS_E_CUDA;   // a block's wait for the others ran out
        if (sc[S_CONV] != 0.0) break;
        first = 0;
    }
    if (cudaGetLastError() != cudaSuccess) return BS_E_CUDA;
    if (iters) *iters = (int32_t)sc[S_ITERS];
    if (relres) *relres = sc[S_BNORM2] > 0.0 ? std::sqrt(sc[S_RTRUE2] / sc[S_BNORM2]) : std::sqrt(sc[S_RTRUE2]);
    const bool ok = sc[S_BNORM2] == 0.0 || sc[S_RNORM2] <= tol * tol * sc[S_BNORM2];
    return ok ? BS_OK : BS_E_NOTCONV;
}
