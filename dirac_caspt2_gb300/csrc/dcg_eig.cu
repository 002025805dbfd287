// Hermitian eigensolver on the device (FP64), the replacement of the reference's ZHEEV /
// DSYEV calls (src/diag.F90:43,109).  Eigenvalues come out ascending, as there.
//
// Three phases, each written from the published algorithm:
//   1. Householder reduction of the Hermitian matrix to a real symmetric tridiagonal
//      (Golub & Van Loan, Matrix Computations, 4th ed., 8.3.1) with the complex reflector
//      of LAPACK's documented xLARFG definition (beta real).
//   2. Cuppen's divide and conquer on the tridiagonal (GVL 8.4.4): the tridiagonal is torn
//      into 1x1 leaves by rank-one modifications; sibling blocks are merged level by level.
//      Each merge deflates (small rank-one components, and Givens rotations for pairs of
//      close poles: Dongarra & Sorensen, SIAM J. Sci. Stat. Comput. 8 (1987) s139), solves
//      the secular equation one root per warp with a bracketed two-pole rational model
//      (Bunch, Nielsen & Sorensen, Numer. Math. 31 (1978) 31), recomputes the rank-one
//      vector from the roots so the eigenvectors stay orthogonal (Gu & Eisenstat, SIAM J.
//      Matrix Anal. Appl. 16 (1995) 172), and applies the merge's eigenvector matrix with one
//      batched GEMM per level.
//   3. Back-transformation of the requested eigenvectors by the stored reflectors.
//
// The merge tree is the power-of-two tree: at level l a node covers columns
// [i 2^l, min((i+1) 2^l, n)) and is split after its first 2^(l-1) columns, so a node's
// geometry follows from (l, i) and no tree is stored.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>

#include <chrono>
#include <condition_variable>
#include <deque>
#include <map>

#include "dcg_common.cuh"
#include "dcg_deflate.cuh"

namespace dcg {

constexpr double kUnitRoundoff = 1.1102230246251565e-16;   // 2^-53
constexpr int kSecularMaxIter = 100;

__device__ __forceinline__ double eig_warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);   // lane 0's value in every lane
}
__device__ __forceinline__ double eig_warp_prod(double v) {
    for (int o = 16; o > 0; o >>= 1) v *= __shfl_down_sync(0xffffffffu, v, o);
    return __shfl_sync(0xffffffffu, v, 0);
}
__device__ __forceinline__ double eig_warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return __shfl_sync(0xffffffffu, v, 0);
}

// Deterministic block sum (fixed tree); every thread gets the result.  sh >= 32 doubles.
__device__ double eig_block_sum(double v, double *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = eig_warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double t = 0.0;
    if (wid == 0) {
        t = lane < nw ? sh[lane] : 0.0;
        t = eig_warp_sum(t);
        if (lane == 0) sh[0] = t;
    }
    __syncthreads();
    t = sh[0];
    __syncthreads();
    return t;
}

__device__ double eig_block_max(double v, double *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = eig_warp_max(v);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double t = 0.0;
    if (wid == 0) {
        t = lane < nw ? sh[lane] : 0.0;
        t = eig_warp_max(t);
        if (lane == 0) sh[0] = t;
    }
    __syncthreads();
    t = sh[0];
    __syncthreads();
    return t;
}

// ===================================================================== 1. tridiagonal reduction
// Step k: reflector for column k (rows k+1..n-1), v stored in A(k+1:n-1, k) with v0 = 1.
__global__ void hh_gen_kernel(int n, int k, cplx *A, int64_t lda, double *d, double *e, cplx *tau) {
    __shared__ double sh[32];
    __shared__ cplx s_scale;
    __shared__ int s_skip;
    const int m = n - k - 1;
    cplx *x = A + (k + 1) + (int64_t)k * lda;
    double s = 0.0;
    for (int i = 1 + threadIdx.x; i < m; i += blockDim.x) s += cabs2(x[i]);
    s = eig_block_sum(s, sh);
    if (threadIdx.x == 0) {
        cplx alpha = x[0];
        double xnorm = sqrt(s);
        cplx t;
        double beta;
        if (xnorm == 0.0 && alpha.y == 0.0) {
            t = mk(0.0, 0.0);
            beta = alpha.x;
            s_skip = 1;
        } else {
            double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm * xnorm);
            beta = alpha.x >= 0.0 ? -nrm : nrm;
            t = mk((beta - alpha.x) / beta, -alpha.y / beta);
            s_scale = cdiv(mk(1.0, 0.0), mk(alpha.x - beta, alpha.y));
            s_skip = 0;
        }
        tau[k] = t;
        e[k] = beta;
        d[k] = A[k + (int64_t)k * lda].x;
    }
    __syncthreads();
    if (!s_skip)
        for (int i = 1 + threadIdx.x; i < m; i += blockDim.x) x[i] = cmul(x[i], s_scale);
    __syncthreads();
    if (threadIdx.x == 0) x[0] = mk(1.0, 0.0);
}

// partial p(i) = sum_{j in chunk} A(k+1+i, k+1+j) v(j)
constexpr int HH_CHUNK = 256;
__global__ void hh_matvec_kernel(int n, int k, const cplx *__restrict__ A, int64_t lda, const cplx *__restrict__ tau,
                                 cplx *ppart) {
    __shared__ cplx vs[HH_CHUNK];
    const int m = n - k - 1;
    const cplx t = tau[k];
    const int j0 = blockIdx.y * HH_CHUNK;
    const int j1 = min(m, j0 + HH_CHUNK);
    const cplx *v = A + (k + 1) + (int64_t)k * lda;
    for (int j = threadIdx.x; j < j1 - j0; j += blockDim.x) vs[j] = v[j0 + j];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    cplx acc = mk(0.0, 0.0);
    if (t.x != 0.0 || t.y != 0.0) {
        const cplx *Ai = A + (k + 1 + i) + (int64_t)(k + 1) * lda;
        for (int j = j0; j < j1; j++) cfma(acc, Ai[(int64_t)j * lda], vs[j - j0]);
    }
    ppart[(int64_t)blockIdx.y * n + i] = acc;
}

// w = tau*p + alpha v,  alpha = -1/2 tau (x^H v) with x = tau*p
__global__ void hh_w_kernel(int n, int k, const cplx *A, int64_t lda, const cplx *tau, const cplx *ppart,
                            int nchunk, cplx *w) {
    __shared__ double sh[32];
    const int m = n - k - 1;
    const cplx t = tau[k];
    const cplx *v = A + (k + 1) + (int64_t)k * lda;
    double sr = 0.0, si = 0.0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        cplx p = mk(0.0, 0.0);
        for (int c = 0; c < nchunk; c++) p = cadd(p, ppart[(int64_t)c * n + i]);
        cplx x = cmul(t, p);
        w[i] = x;
        cplx xv = cmul(cconj(x), v[i]);
        sr += xv.x;
        si += xv.y;
    }
    sr = eig_block_sum(sr, sh);
    si = eig_block_sum(si, sh);
    cplx alpha = cmul(mk(-0.5, 0.0), cmul(t, mk(sr, si)));
    for (int i = threadIdx.x; i < m; i += blockDim.x) w[i] = cadd(w[i], cmul(alpha, v[i]));
}

// A(k+1:, k+1:) -= v w^H + w v^H
__global__ void hh_update_kernel(int n, int k, cplx *A, int64_t lda, const cplx *w) {
    const int m = n - k - 1;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if (i >= m || j >= m) return;
    const cplx *v = A + (k + 1) + (int64_t)k * lda;
    cplx vi = v[i], vj = v[j], wi = w[i], wj = w[j];
    int64_t o = (k + 1 + i) + (int64_t)(k + 1 + j) * lda;
    cplx a = A[o];
    a = csub(a, cmulc(vi, wj));
    a = csub(a, cmulc(wi, vj));
    if (i == j) a.y = 0.0;
    A[o] = a;
}

__global__ void hh_last_kernel(int n, const cplx *A, int64_t lda, double *d) {
    d[n - 1] = A[(n - 1) + (int64_t)(n - 1) * lda].x;
}

// ---- persistent form: one cooperative launch for all columns, two grid barriers per column.
// Every block recomputes the reflector of column k (identical arithmetic in every block) and
// stages v in shared memory; a warp per column computes p = A22 v (A22 Hermitian, so
// p_i = column i of A22, conjugated, dotted with v); after the first barrier every block
// forms w = tau p + alpha v and applies A22 -= v w^H + w v^H to its columns.  Data written by
// other blocks is read with ld.global.cg so no stale L1 line is used.
struct GridBar {
    unsigned count;
    unsigned gen;
    int err;       // 1: a barrier wait exceeded its time limit
    unsigned long long limit_ns;   // time limit of one wait (set by the host before the launch)
};

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier for a cooperative launch: one monotonically increasing arrival counter
// (count), so a barrier costs one fence, one atomic and an acquire poll.  Each wait is bounded
// (gb->limit_ns, 5 s by default, the clock read every 16 polls); a block that gives up sets
// gb->err and every waiting block then leaves the kernel.
constexpr uint64_t kBarrierLimitNs = 5000000000ull;
__device__ __forceinline__ bool grid_barrier(GridBar *gb, unsigned nblocks) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        __threadfence();
        const unsigned arrive = atomicAdd(&gb->count, 1u);
        const unsigned target = (arrive / nblocks + 1u) * nblocks;
        unsigned cur;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(&gb->count) : "memory");
        if ((int)(cur - target) < 0) {
            const uint64_t t0 = globaltimer_ns();
            unsigned spins = 0;
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(cur) : "l"(&gb->count) : "memory");
                if ((int)(cur - target) >= 0) break;
                if ((++spins & 15u) == 0) {
                    if (*(volatile int *)&gb->err) {
                        ok = 0;
                        break;
                    }
                    if (globaltimer_ns() - t0 > gb->limit_ns) {
                        atomicExch(&gb->err, 1);
                        ok = 0;
                        break;
                    }
                }
            }
        }
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ cplx ldcg(const cplx *p) { return __ldcg(p); }

constexpr int TRD_THREADS = 512;
constexpr int TRD_UNROLL = 8;
constexpr int kTridiagPersistentMaxN = 7000;   // v and w staged in shared memory: 32 bytes per row

__global__ void __launch_bounds__(TRD_THREADS) tridiag_persistent_kernel(int n, cplx *A, int64_t lda, double *d,
                                                                         double *e, cplx *tau, cplx *pbuf,
                                                                         double2 *part, GridBar *gb) {
    extern __shared__ cplx tsm[];
    __shared__ double red[32];
    __shared__ cplx s_scale, s_tau, s_alpha;
    __shared__ double s_beta;
    __shared__ int s_skip;
    const unsigned nb = gridDim.x;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwb = blockDim.x >> 5;
    const int gw = blockIdx.x * nwb + wib, nw = nb * nwb;
    cplx *sv = tsm, *sw = tsm + (n > 1 ? n - 1 : 1);
    for (int k = 0; k + 1 < n; k++) {
        const int m = n - k - 1;
        cplx *x = A + (k + 1) + (int64_t)k * lda;
        // reflector of column k (same in every block)
        double ss = 0.0;
        for (int i = 1 + threadIdx.x; i < m; i += blockDim.x) ss += cabs2(ldcg(x + i));
        ss = eig_block_sum(ss, red);
        if (threadIdx.x == 0) {
            const cplx alpha = ldcg(x);
            const double xnorm = sqrt(ss);
            if (xnorm == 0.0 && alpha.y == 0.0) {
                s_tau = mk(0.0, 0.0);
                s_beta = alpha.x;
                s_skip = 1;
                s_scale = mk(1.0, 0.0);
            } else {
                const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm * xnorm);
                const double beta = alpha.x >= 0.0 ? -nrm : nrm;
                s_tau = mk((beta - alpha.x) / beta, -alpha.y / beta);
                s_beta = beta;
                s_scale = cdiv(mk(1.0, 0.0), mk(alpha.x - beta, alpha.y));
                s_skip = 0;
            }
        }
        __syncthreads();
        const cplx t = s_tau, sc = s_scale;
        const bool active = !s_skip;
        for (int i = threadIdx.x; i < m; i += blockDim.x) sv[i] = i == 0 ? mk(1.0, 0.0) : (active ? cmul(ldcg(x + i), sc) : ldcg(x + i));
        __syncthreads();
        // p = tau * A22 v (warp per column), partial x^H v with x = tau p
        double pr = 0.0, pim = 0.0;
        if (active) {
            for (int i = gw; i < m; i += nw) {
                const cplx *col = A + (k + 1) + (int64_t)(k + 1 + i) * lda;
                // conj(column) . v with TRD_UNROLL loads in flight per lane (the loop is L2-latency bound)
                double arr[TRD_UNROLL], aii[TRD_UNROLL];
#pragma unroll
                for (int u = 0; u < TRD_UNROLL; u++) arr[u] = aii[u] = 0.0;
                int j = lane;
                for (; j + 32 * (TRD_UNROLL - 1) < m; j += 32 * TRD_UNROLL) {
                    cplx a[TRD_UNROLL];
#pragma unroll
                    for (int u = 0; u < TRD_UNROLL; u++) a[u] = ldcg(col + j + 32 * u);
#pragma unroll
                    for (int u = 0; u < TRD_UNROLL; u++) {
                        const cplx v = sv[j + 32 * u];
                        arr[u] += a[u].x * v.x + a[u].y * v.y;
                        aii[u] += a[u].x * v.y - a[u].y * v.x;
                    }
                }
                for (; j < m; j += 32) {
                    const cplx a = ldcg(col + j), v = sv[j];
                    arr[0] += a.x * v.x + a.y * v.y;
                    aii[0] += a.x * v.y - a.y * v.x;
                }
                double ar = 0.0, ai = 0.0;
#pragma unroll
                for (int u = 0; u < TRD_UNROLL; u++) {
                    ar += arr[u];
                    ai += aii[u];
                }
                for (int o = 16; o > 0; o >>= 1) {
                    ar += __shfl_down_sync(0xffffffffu, ar, o);
                    ai += __shfl_down_sync(0xffffffffu, ai, o);
                }
                if (lane == 0) {
                    const cplx xp = cmul(t, mk(ar, ai));
                    pbuf[i] = xp;
                    const cplx xv = cmul(cconj(xp), sv[i]);
                    pr += xv.x;
                    pim += xv.y;
                }
            }
        }
        pr = eig_block_sum(pr, red);
        pim = eig_block_sum(pim, red);
        if (threadIdx.x == 0) part[blockIdx.x] = make_double2(pr, pim);
        if (!grid_barrier(gb, nb)) return;
        if (active) {
            double sr = 0.0, si = 0.0;
            for (unsigned b = threadIdx.x; b < nb; b += blockDim.x) {
                const double2 q = __ldcg(part + b);
                sr += q.x;
                si += q.y;
            }
            sr = eig_block_sum(sr, red);
            si = eig_block_sum(si, red);
            if (threadIdx.x == 0) s_alpha = cmul(mk(-0.5, 0.0), cmul(t, mk(sr, si)));
            __syncthreads();
            const cplx al = s_alpha;
            for (int i = threadIdx.x; i < m; i += blockDim.x) sw[i] = cadd(ldcg(pbuf + i), cmul(al, sv[i]));
            __syncthreads();
            for (int j = gw; j < m; j += nw) {
                const cplx vj = sv[j], wj = sw[j];
                cplx *col = A + (k + 1) + (int64_t)(k + 1 + j) * lda;
                int i = lane;
                for (; i + 32 * (TRD_UNROLL - 1) < m; i += 32 * TRD_UNROLL) {
                    cplx a[TRD_UNROLL];
#pragma unroll
                    for (int u = 0; u < TRD_UNROLL; u++) a[u] = ldcg(col + i + 32 * u);
#pragma unroll
                    for (int u = 0; u < TRD_UNROLL; u++) {
                        const int r = i + 32 * u;
                        cplx x = csub(a[u], cmulc(sv[r], wj));
                        x = csub(x, cmulc(sw[r], vj));
                        if (r == j) x.y = 0.0;
                        col[r] = x;
                    }
                }
                for (; i < m; i += 32) {
                    cplx a = ldcg(col + i);
                    a = csub(a, cmulc(sv[i], wj));
                    a = csub(a, cmulc(sw[i], vj));
                    if (i == j) a.y = 0.0;
                    col[i] = a;
                }
            }
        }
        if (blockIdx.x == 0) {
            for (int i = threadIdx.x; i < m; i += blockDim.x) x[i] = sv[i];
            if (threadIdx.x == 0) {
                d[k] = ldcg(A + k + (int64_t)k * lda).x;
                e[k] = s_beta;
                tau[k] = t;
            }
        }
        if (!grid_barrier(gb, nb)) return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) d[n - 1] = ldcg(A + (n - 1) + (int64_t)(n - 1) * lda).x;
}

// ---- shared-memory-resident form (n up to kTridiagSmemMaxN): the matrix lives in the blocks'
// shared memory for the whole reduction, block b owning columns b, b + nb, ...  Per column k the
// blocks exchange the reflector v (from the owner of column k) and x = tau A22 v (one entry per
// column, from its owner); the matvec and the rank-2 update run from shared memory.
//
// What bounds it is the chain of a column (the column's update, its way to every block, the
// matvec, x to every block, the next column's update) and the FP64 unit (a warp's FP64
// instruction holds a quarter of the SM for 70 to 77 clocks, whether one lane is active or all).  So:
//   - the column and x travel as 16-byte words that carry their own flag (the column's number
//     above each half of a double): a reader polls the data itself, one trip through L2 instead
//     of data, fence, counter and data again.
//   - the column goes out unscaled as soon as it is updated (u; v = sc u below a unit first
//     element).  Every block multiplies with u while a seventeenth warp of the owner forms tau
//     and sc from the norm, which follow as the header: conj(column) . v = sc (conj(column) . u)
//     + conj(A(k+1, j)), and tau sc = -1 / beta.
//   - every column's rows are dealt in pieces of 32 to the four quarters of the SM, shifted by
//     the column, so matvec and update load the quarters evenly for any number of columns.
//   - four warps (one per quarter) carry the chain: they receive u and x, scale v while x is
//     under way, and in the block that owns column k+1 update that column before all others.
//   - x^H v = conj(tau) v^H A22 v has a known phase, so only its real part is summed: w = x + al v
//     has a real al, which the update needs for its own columns alone.
// A sum's order depends on the matrix alone (rows and pieces), never on the number of
// blocks: the same bits alone, merged with other matrices or in a cluster.
// Measured, reduction alone: order 70 0.35 ms (5.0 us a column, the chain), order 791 9.5 ms (12 us a
// column, of which about 8 are FP64 issue), two of order 792 together 13.2 ms; before, with a
// grid barrier and a published-reflector wait per column, one warp per column and the reflector
// by one warp: order 791 17.7 ms, two of 792 21.2 ms.
constexpr int kTridiagSmemMaxN = 1400;
constexpr int kTrdRows = (kTridiagSmemMaxN + 127) / 128;   // rows of one of the four chain warps' lanes
constexpr int kTrdMaxJobs = 32;

// One problem of a batched launch: its matrix, outputs, exchange buffers and the block range
// [b0, b0 + nb) that reduces it.
struct TrdJob {
    cplx *A;
    int64_t lda;
    double *d, *e;
    cplx *tau;
    ulonglong2 *ll;      // trd_ll_words(n) words, zero before the launch
    unsigned long long limit_ns;   // time limit of one wait (its context's, also in a merged launch)
    int n, b0, nb, real;
};
struct TrdTable {
    TrdJob j[kTrdMaxJobs];
    int njobs;
    int *err;   // per job: nonzero when a wait ran out (zero before the launch)
};
// exchange words of one problem: by column parity x (2 n), u (2 n) and the header (8)
__host__ __device__ inline size_t trd_ll_words(int n) { return 8 * (size_t)n + 16; }

// A double in one 16-byte word: two 64-bit elements, each a half of it with the flag above it.  (Data
// words that carry their own flag are the low-latency exchange known from communication
// libraries.)  A vector access is one access per element in no given order, and a 64-bit element
// is read and written whole, so each flag vouches for the half beside it.
__device__ __forceinline__ void ll_store(ulonglong2 *p, double v, unsigned flag) {
    const unsigned long long f = (unsigned long long)flag << 32;
    asm volatile("st.volatile.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(f | (unsigned)__double2loint(v)),
                 "l"(f | (unsigned)__double2hiint(v))
                 : "memory");
}
__device__ __forceinline__ bool ll_load(const ulonglong2 *p, unsigned flag, double &v) {
    unsigned long long lo, hi;
    asm volatile("ld.volatile.global.v2.b64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    v = __hiloint2double((int)(unsigned)hi, (int)(unsigned)lo);
    return (unsigned)(lo >> 32) == flag && (unsigned)(hi >> 32) == flag;
}

// A bounded wait of one thread (the clock and the problem's error flag are read every 4 polls).
struct LlWait {
    uint64_t t0 = 0;
    unsigned spins = 0;
    __device__ __forceinline__ bool give_up(int *err, unsigned long long limit_ns) {
        if (spins++ == 0) t0 = globaltimer_ns();
        if ((spins & 3u) != 0) return false;
        if (*(volatile int *)err) return true;
        if (globaltimer_ns() - t0 <= limit_ns) return false;
        atomicExch(err, 1);
        return true;
    }
};

// Reflector of the column alpha, x with ss = |x|^2 (LAPACK's documented xLARFG, beta real): tau,
// beta, the scale sc = 1 / (alpha - beta) of x, and mib = tau sc = -1 / beta (0 for tau = 0).
__device__ __forceinline__ void trd_scalars(cplx alpha, double ss, cplx &tau, double &beta, cplx &scale, double &mib) {
    if (ss == 0.0 && alpha.y == 0.0) {
        tau = mk(0.0, 0.0);
        beta = alpha.x;
        scale = mk(1.0, 0.0);
        mib = 0.0;
        return;
    }
    const double a2 = cabs2(alpha), N2 = a2 + ss;
    if (N2 > 1e-280 && N2 < 1e280) {
        const double rs = fast_rsqrt(N2), s = alpha.x >= 0.0 ? -1.0 : 1.0, ib = s * rs;
        beta = s * (N2 * rs);
        tau = mk(fma(-alpha.x, ib, 1.0), -alpha.y * ib);
        const double gx = alpha.x - beta, r = fast_rcp(fma(gx, gx, alpha.y * alpha.y));
        scale = mk(gx * r, -alpha.y * r);
        mib = -ib;
    } else {   // outside the safe range of the squares: the plain formulas
        const double nrm = sqrt(N2);
        beta = alpha.x >= 0.0 ? -nrm : nrm;
        tau = mk((beta - alpha.x) / beta, -alpha.y / beta);
        scale = cdiv(mk(1.0, 0.0), mk(alpha.x - beta, alpha.y));
        mib = -1.0 / beta;
    }
}

__device__ __forceinline__ void chain_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }   // the four chain warps
__device__ __forceinline__ void column_sync() { asm volatile("bar.sync 2, 512;" ::: "memory"); }  // all but the header warp
// the chain warps of a column's owner tell the header warp that its sums are there
__device__ __forceinline__ void sums_ready() { asm volatile("bar.arrive 3, 160;" ::: "memory"); }
__device__ __forceinline__ void sums_wait() { asm volatile("bar.sync 3, 160;" ::: "memory"); }

// GLB: the columns stay in global memory (L2, or HBM beyond it) and u has a row of shared memory of
// its own; otherwise ROWS >= n / 128 and the chain warps hold u and v in registers.
template <bool REAL, int ROWS, bool GLB>
__device__ void tridiag_smem_body(const TrdJob &J, const int b, int *err) {
    extern __shared__ cplx tsm2[];
    __shared__ double s_sum[4], s_ss[4], s_hdr[5], s_al;
    __shared__ cplx s_alpha;
    const int n = J.n, nb = J.nb;
    const unsigned long long limit_ns = J.limit_ns;
    cplx *A = J.A;
    const int64_t lda = J.lda;
    ulonglong2 *xb = J.ll, *ub = xb + 4 * (size_t)n, *hb = ub + 4 * (size_t)n;   // [parity][n][2], [parity][n][2], [parity][8]
    const int tid = threadIdx.x, lane = tid & 31, q = (tid >> 5) & 3, s = tid >> 7;   // quarter, and warp within it
    const bool chain = s == 0, header = s == 4;
    const int nown = (n - b + nb - 1) / nb;   // columns b, b+nb, ...
    cplx *sv = GLB ? tsm2 : tsm2 + (size_t)nown * n, *sw = sv + n;   // v (not GLB: first u) and x
    cplx *su = GLB ? sw + n : sv;
    double *part = reinterpret_cast<double *>(sw + (GLB ? 2 : 1) * (size_t)n);   // [nown][4 quarters][2]
    auto column = [&](int c) { return GLB ? A + (int64_t)(b + c * nb) * lda : tsm2 + (size_t)c * n; };   // owned column
    if (!GLB) {
        for (int64_t x = tid; x < (int64_t)nown * n; x += blockDim.x) {
            const int c = (int)(x / n), r = (int)(x % n);
            tsm2[x] = A[r + (int64_t)(b + c * nb) * lda];
        }
    }
    __syncthreads();
    cplx vr[GLB ? 1 : ROWS];   // chain warps, not GLB: rows 32 (4 i + q) + lane of u, then of v
    const int NI = (n + 127) / 128;
    // the rows of a chain warp's lane, in groups of ROWS (not GLB: one group)
#define TRD_GROUPS(i0) for (int i0 = 0; i0 < (GLB ? NI : 1); i0 += ROWS)
#define TRD_ROWS(i0, i, r, from)                                                                \
    _Pragma("unroll") for (int i = 0; i < ROWS; i++)                                            \
        if (const int r = 32 * (4 * ((i0) + i) + q) + lane; (i0) + i < NI && r >= (from) && r < n)
    // Chain warps of the block that owns column k1: subtract the rank-2 term of the previous
    // column when upd, publish what lies below the reflector's first row, and leave that row's
    // element (alpha) and the parts of the squared norm for the header warp.
    auto panel = [&](int k1, bool upd) {
        const cplx *col = column((k1 - b) / nb);
        cplx vj = mk(0.0, 0.0), yj = mk(0.0, 0.0);
        if (upd) {
            vj = sv[k1];
            const cplx x = sw[k1];
            const double a2 = 2.0 * s_al;
            yj = mk(fma(a2, vj.x, x.x), fma(a2, vj.y, x.y));
        }
        ulonglong2 *uo = ub + (size_t)(k1 & 1) * 2 * n;
        const unsigned flag = (unsigned)k1 + 1u;
        double s0 = 0.0, s1 = 0.0;
        TRD_GROUPS(i0) TRD_ROWS(i0, i, r, k1) {
            cplx a = col[r];
            if (upd) {
                const cplx v = GLB ? sv[r] : vr[GLB ? 0 : i], x = sw[r];
                a.x = fma(-x.x, vj.x, a.x);
                a.x = fma(-v.x, yj.x, a.x);
                if (!REAL) {
                    a.y = fma(-x.y, vj.x, a.y);
                    a.x = fma(-x.y, vj.y, a.x);
                    a.y = fma(x.x, vj.y, a.y);
                    a.x = fma(-v.y, yj.y, a.x);
                    a.y = fma(-v.y, yj.x, a.y);
                    a.y = fma(v.x, yj.y, a.y);
                }
            }
            if (r == k1) J.d[k1] = a.x;
            if (r == k1 + 1) s_alpha = a;
            if (r <= k1 + 1) {
                a = mk(0.0, 0.0);
            } else if (nb > 1) {
                ll_store(uo + 2 * (size_t)r, a.x, flag);
                if (!REAL) ll_store(uo + 2 * (size_t)r + 1, a.y, flag);
            }
            if (GLB) su[r] = a;
            else vr[GLB ? 0 : i] = a;
            s0 = fma(a.x, a.x, s0);
            if (!REAL) s1 = fma(a.y, a.y, s1);
        }
        if (!REAL) s0 += s1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        if (lane == 0) s_ss[q] = s0;
        if (k1 + 1 < n) sums_ready();
    };
    if (b == 0 && chain) panel(0, false);
    for (int k = 0; k + 1 < n; k++) {
        // First owned column index > k.  A block without one leaves after its own last column.
        // An exchange word is written again two columns later, when every block still in the
        // loop has answered the column between (its x is needed for the next reflector), so it
        // has read the old word.
        const int c0 = k + 1 > b ? (k + 1 - b + nb - 1) / nb : 0;
        const bool owner = b == k % nb;
        if (c0 >= nown && !owner) return;
        const unsigned flag = (unsigned)k + 1u;
        const int par = k & 1;
        if (chain && !owner) {   // u, straight from its words: one row until it is there, then all
            const ulonglong2 *ui = ub + (size_t)par * 2 * n;
            LlWait wt;
            TRD_GROUPS(i0) {
                unsigned pend = 0;
                TRD_ROWS(i0, i, r, k + 2) pend |= 1u << i;
                bool all = i0 > 0;
                while (pend) {
                    const unsigned first = pend & (0u - pend);
                    all = all || (pend & (pend - 1)) == 0;
                    const unsigned look = all ? pend : first;
                    const unsigned before = pend;
                    TRD_ROWS(i0, i, r, k + 2) {
                        if (look >> i & 1u) {
                            double x, y = 0.0;
                            bool got = ll_load(ui + 2 * (size_t)r, flag, x);
                            if (!REAL) got = ll_load(ui + 2 * (size_t)r + 1, flag, y) && got;
                            if (got) {
                                if (GLB) su[r] = mk(x, y);
                                else vr[GLB ? 0 : i] = mk(x, y);
                                pend &= ~(1u << i);
                            }
                        }
                    }
                    all = pend != before;
                    // once a wait has run out the problem's error flag is set and every wait of its
                    // blocks ends at once: the loop runs out on whatever values there are
                    if (pend && wt.give_up(err, limit_ns)) break;
                }
            }
        }
        if (!header) {
            if (!GLB) {
                column_sync();   // the previous column's update is done: sv may change
                if (chain) TRD_ROWS(0, i, r, k + 1) sv[r] = r == k + 1 ? mk(0.0, 0.0) : vr[GLB ? 0 : i];
            }
            column_sync();
        }
        const int p0 = (k + 2) >> 5, pe = (n + 31) >> 5;   // pieces of 32 rows with rows > k + 1
        if (header) {   // the reflector's scalars: from the owner's sums, or its words
            if (owner) {
                cplx t, sc;
                double beta, mib;
                sums_wait();
                trd_scalars(s_alpha, (s_ss[0] + s_ss[1]) + (s_ss[2] + s_ss[3]), t, beta, sc, mib);
                if (lane < 5) {
                    const double h = lane == 0 ? sc.x : lane == 1 ? sc.y : lane == 2 ? t.x : lane == 3 ? t.y : mib;
                    if (nb > 1) ll_store(hb + 8 * par + lane, h, flag);
                    s_hdr[lane] = h;
                }
                if (lane == 0) {
                    J.tau[k] = t;
                    J.e[k] = beta;
                }
            } else if (lane < 5) {
                LlWait wt;
                double h;
                while (!ll_load(hb + 8 * par + lane, flag, h))
                    if (wt.give_up(err, limit_ns)) break;
                s_hdr[lane] = h;
            }
        } else {
            // matvec: conj(column) . u over this quarter's pieces, two columns at a time
            for (int c = c0 + ((s - c0) & 3); c < nown; c += 8) {
                double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
                const bool two = c + 4 < nown;
                {
                    const int j = b + c * nb;
                    const cplx *col = column(c);
#pragma unroll 2
                    for (int p = p0 + ((q - j - p0) & 3); p < pe; p += 4) {
                        const int r = 32 * p + lane;
                        if (r > k + 1 && r < n) {
                            const cplx a = col[r], v = su[r];
                            a0 = fma(a.x, v.x, a0);
                            if (!REAL) {
                                a1 = fma(a.x, v.y, a1);
                                a0 = fma(a.y, v.y, a0);
                                a1 = fma(-a.y, v.x, a1);
                            }
                        }
                    }
                }
                if (two) {
                    const int j = b + (c + 4) * nb;
                    const cplx *col = column(c + 4);
#pragma unroll 2
                    for (int p = p0 + ((q - j - p0) & 3); p < pe; p += 4) {
                        const int r = 32 * p + lane;
                        if (r > k + 1 && r < n) {
                            const cplx a = col[r], v = su[r];
                            a2 = fma(a.x, v.x, a2);
                            if (!REAL) {
                                a3 = fma(a.x, v.y, a3);
                                a2 = fma(a.y, v.y, a2);
                                a3 = fma(-a.y, v.x, a3);
                            }
                        }
                    }
                }
                // the four sums over the warp: halves exchanged first, then eighths, so every sum is
                // added over lane distances 16, 8, 4, 2, 1 whichever column it belongs to
                const bool hi = lane & 16, lo = lane & 8;
                double u = hi ? a2 : a0, w = hi ? a3 : a1;
                if (two) {
                    u += __shfl_xor_sync(0xffffffffu, hi ? a0 : a2, 16);
                    if (!REAL) w += __shfl_xor_sync(0xffffffffu, hi ? a1 : a3, 16);
                } else {
                    u = a0 + __shfl_xor_sync(0xffffffffu, a0, 16);
                    if (!REAL) w = a1 + __shfl_xor_sync(0xffffffffu, a1, 16);
                }
                double y;
                if (REAL) {
                    y = u + __shfl_xor_sync(0xffffffffu, u, 8);
                } else {
                    y = lo ? w : u;
                    y += __shfl_xor_sync(0xffffffffu, lo ? u : w, 8);
                }
                y += __shfl_xor_sync(0xffffffffu, y, 4);
                y += __shfl_xor_sync(0xffffffffu, y, 2);
                y += __shfl_xor_sync(0xffffffffu, y, 1);
                if ((lane & 7) == 0 && (two || !hi)) part[((size_t)(c + (hi ? 4 : 0)) * 4 + q) * 2 + (lo ? 1 : 0)] = y;
            }
        }
        __syncthreads();
        const double sx = s_hdr[0], sy = s_hdr[1], tr = s_hdr[2], ti = s_hdr[3], mib = s_hdr[4];
        if (s >= 1 && !header) {
            // x = tau p = mib (conj(column) . u) + tau conj(A(k+1, j)) of the own columns, to every block
            ulonglong2 *xo = xb + (size_t)par * 2 * n;
            const int cnt = 2 * (nown - c0);
            for (int t = tid - 128; t < ((cnt + 31) & ~31); t += 384) {
                const int c = c0 + (t >> 1), comp = t & 1, j = b + c * nb;
                double y = 0.0;
                cplx a = mk(0.0, 0.0);
                if (t < cnt) {
                    a = column(c)[k + 1];
                    const double *p = part + (size_t)c * 8 + comp;
                    if (!REAL || comp == 0) y = (p[0] + p[2]) + (p[4] + p[6]);
                }
                const double x = REAL ? (comp ? 0.0 : fma(mib, y, tr * a.x))
                                      : fma(mib, y, comp ? fma(ti, a.x, -tr * a.y) : fma(tr, a.x, ti * a.y));
                if (t < cnt) {
                    if (nb > 1) {
                        if (!REAL || comp == 0) ll_store(xo + 2 * (size_t)j + comp, x, flag);
                    } else {
                        reinterpret_cast<double *>(sw)[2 * j + comp] = x;
                    }
                }
            }
        }
        if (chain) {   // v = sc u below its first row
            TRD_GROUPS(i0) TRD_ROWS(i0, i, r, k + 1) {
                const cplx u = GLB ? su[r] : vr[GLB ? 0 : i];
                const cplx v = r == k + 1 ? mk(1.0, 0.0)
                                          : (REAL ? mk(u.x * sx, 0.0)
                                                  : mk(fma(u.x, sx, -u.y * sy), fma(u.x, sy, u.y * sx)));
                if (!GLB) vr[GLB ? 0 : i] = v;
                sv[r] = v;
                if (owner) A[r + (int64_t)k * lda] = v;
            }
        }
        if (c0 >= nown) return;   // the owner of column k was left for this
        if (nb == 1) __syncthreads();
        if (chain) {   // gather x, and al of w = x + al v: al = -1/2 tau x^H v = -|tau|^2 / (2 Re tau) Re(x^H v)
            const double f = tr != 0.0 ? -0.5 * fma(tr, tr, ti * ti) * fast_rcp(tr) : 0.0;
            if (nb > 1) {
                const ulonglong2 *xi = xb + (size_t)par * 2 * n;
                LlWait wt;
                TRD_GROUPS(i0) {
                    unsigned pend = 0;
                    TRD_ROWS(i0, i, r, k + 1) pend |= 1u << i;
                    bool all = true;
                    while (pend) {
                        const unsigned look = all ? pend : (pend & (0u - pend)), before = pend;
                        TRD_ROWS(i0, i, r, k + 1) {
                            if (look >> i & 1u) {
                                double x, y = 0.0;
                                bool got = ll_load(xi + 2 * (size_t)r, flag, x);
                                if (!REAL) got = ll_load(xi + 2 * (size_t)r + 1, flag, y) && got;
                                if (got) {
                                    sw[r] = mk(x, y);
                                    pend &= ~(1u << i);
                                }
                            }
                        }
                        all = pend != before;
                        if (pend && wt.give_up(err, limit_ns)) break;
                    }
                }
            }
            double z0 = 0.0, z1 = 0.0, z2 = 0.0, z3 = 0.0;
            TRD_GROUPS(i0) TRD_ROWS(i0, i, r, k + 1) {
                const cplx x = sw[r], v = GLB ? sv[r] : vr[GLB ? 0 : i];
                if (i & 1) {
                    z2 = fma(x.x, v.x, z2);
                    if (!REAL) z3 = fma(x.y, v.y, z3);
                } else {
                    z0 = fma(x.x, v.x, z0);
                    if (!REAL) z1 = fma(x.y, v.y, z1);
                }
            }
            double z = REAL ? z0 + z2 : (z0 + z1) + (z2 + z3);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            if (lane == 0) s_sum[q] = z;
            chain_sync();
            if (tid == 0) s_al = f * ((s_sum[0] + s_sum[1]) + (s_sum[2] + s_sum[3]));
        }
        __syncthreads();
        // the next column's owner updates it before its other columns and publishes it
        if (chain && b == (k + 1) % nb) panel(k + 1, true);
        // update of the other columns, rows > k+1: with w = x + al v,
        //   a - v conj(w_j) - w conj(v_j) = a - v conj(x_j + 2 al v_j) - x conj(v_j)
        if (!header) {
            const int c1 = k + 2 > b ? (k + 2 - b + nb - 1) / nb : 0;
            const double a2 = 2.0 * s_al;
            for (int c = c1 + ((s - c1) & 3); c < nown; c += 4) {
                const int j = b + c * nb;
                cplx *col = column(c);
                const cplx vj = sv[j], xj = sw[j];
                const cplx yj = mk(fma(a2, vj.x, xj.x), fma(a2, vj.y, xj.y));
#pragma unroll 2
                for (int p = p0 + ((q - j - p0) & 3); p < pe; p += 4) {
                    const int r = 32 * p + lane;
                    if (r > k + 1 && r < n) {
                        const cplx v = sv[r], x = sw[r];
                        cplx a = col[r];
                        a.x = fma(-v.x, yj.x, a.x);
                        if (!REAL) {
                            a.y = fma(-v.y, yj.x, a.y);
                            a.x = fma(-v.y, yj.y, a.x);
                            a.y = fma(v.x, yj.y, a.y);
                            a.x = fma(-x.y, vj.y, a.x);
                            a.y = fma(-x.y, vj.x, a.y);
                            a.y = fma(x.x, vj.y, a.y);
                        }
                        a.x = fma(-x.x, vj.x, a.x);
                        if (r == j) a.y = 0.0;
                        col[r] = a;
                    }
                }
            }
        }
    }
#undef TRD_ROWS
#undef TRD_GROUPS
}

// Batched tridiagonalisation: several Hermitian matrices in one launch, each reduced by its own
// group of blocks (all resident at once: a cooperative launch, or a cluster per matrix), so the
// latency-bound column loops of independent problems overlap instead of running one after
// another.
constexpr int TRS_THREADS = 544;   // sixteen warps for the columns and one for the header
__global__ void __launch_bounds__(TRS_THREADS) tridiag_smem_batched_kernel(const __grid_constant__ TrdTable T) {
    int j = 0;
    while (j + 1 < T.njobs && (int)blockIdx.x >= T.j[j + 1].b0) j++;
    const TrdJob &J = T.j[j];
    const int b = (int)blockIdx.x - J.b0;
    if (J.n <= 512) {
        if (J.real) tridiag_smem_body<true, 4, false>(J, b, T.err + j);
        else tridiag_smem_body<false, 4, false>(J, b, T.err + j);
    } else if (J.n <= 1024) {
        if (J.real) tridiag_smem_body<true, 8, false>(J, b, T.err + j);
        else tridiag_smem_body<false, 8, false>(J, b, T.err + j);
    } else {
        if (J.real) tridiag_smem_body<true, kTrdRows, false>(J, b, T.err + j);
        else tridiag_smem_body<false, kTrdRows, false>(J, b, T.err + j);
    }
}

// One matrix beyond the blocks' shared memory, over every SM: the same column loop on columns in
// global memory.  Bound by the FP64 unit (12 FMAs an element and column: 66 ms at order 2002 at
// 485 GFMA/s), the three passes over the trailing matrix a column from L2 or HBM beside it.
// Measured against the kernel with two grid barriers a column that every block's reflector waits
// for: order 1300 44 -> 27 ms, 2002 210 -> 82 ms, 2744 437 -> 191 ms.
__global__ void __launch_bounds__(TRS_THREADS) tridiag_global_kernel(const __grid_constant__ TrdTable T) {
    const TrdJob &J = T.j[0];
    if (J.real) tridiag_smem_body<true, 8, true>(J, (int)blockIdx.x, T.err);
    else tridiag_smem_body<false, 8, true>(J, (int)blockIdx.x, T.err);
}

// ===================================================================== 2. divide and conquer
// Per-level scratch, every array of length n and sliced by node (a node owns [s, s+N)).
struct DcBufs {
    double *lamA, *lamB;      // eigenvalues of the current / next level
    double *QA, *QB;          // eigenvector matrices (n x n, ld n), block diagonal by node
    double *U;                // merge eigenvector matrices, block diagonal (n x n, ld n)
    double *dK, *zK;          // undeflated poles and rank-one components (compact, per node)
    double *dv;               // deflated eigenvalues (per node)
    int *Kl, *defl;           // node-local column of each undeflated / deflated entry
    int *rp, *rn;             // Givens rotation column pairs
    double *rc, *rs;          // and their cosines / sines
    int *ord;                 // origin pole of each secular root (before that, the folded entries)
    double *tau, *lamK;       // root offset from its origin, root value
    double *zh;               // recomputed rank-one vector
    int *outc;                // output column of each node entry in the next level
    int *top, *bot;           // undeflated entries whose column reaches the node's first / second half
    int *k0, *flag, *half;    // prep scratch: entries past the z test, close pairs, halves reached
    int *kcnt, *ndef, *nrot;  // per node: undeflated count (-1: pass-through), deflated, rotations
    int *ntop, *nbot;         // per node: lengths of top and bot
    double *rho;              // per node
    int *status;              // nonzero: a merge met an inconsistent pole order
};

// Sums of four values over groups of G lanes; every lane of a group gets all four.  The first two
// exchange steps halve the number of values a lane carries, so 32 lanes take six FP64 additions
// instead of twenty (each holds a quarter SM for 77 clocks).
template <int G>
__device__ __forceinline__ void dc_sum4(double &v0, double &v1, double &v2, double &v3) {
    const int lane = threadIdx.x & 31;
    if (G == 4) {
        // lane g of the group ends with value g
        const bool h2 = lane & 2, h1 = lane & 1;
        double a = h2 ? v2 : v0, b = h2 ? v3 : v1;
        a += __shfl_xor_sync(0xffffffffu, h2 ? v0 : v2, 2);
        b += __shfl_xor_sync(0xffffffffu, h2 ? v1 : v3, 2);
        double x = h1 ? b : a;
        x += __shfl_xor_sync(0xffffffffu, h1 ? a : b, 1);
        v0 = __shfl_sync(0xffffffffu, x, 0, 4);
        v1 = __shfl_sync(0xffffffffu, x, 1, 4);
        v2 = __shfl_sync(0xffffffffu, x, 2, 4);
        v3 = __shfl_sync(0xffffffffu, x, 3, 4);
    } else {
        const bool hi = lane & (G / 2), lo = lane & (G / 4);
        double a = hi ? v2 : v0, b = hi ? v3 : v1;
        a += __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, G / 2);
        b += __shfl_xor_sync(0xffffffffu, hi ? v1 : v3, G / 2);
        double x = lo ? b : a;
        x += __shfl_xor_sync(0xffffffffu, lo ? a : b, G / 4);
#pragma unroll
        for (int o = G / 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        v0 = __shfl_sync(0xffffffffu, x, 0, G);
        v1 = __shfl_sync(0xffffffffu, x, G / 4, G);
        v2 = __shfl_sync(0xffffffffu, x, G / 2, G);
        v3 = __shfl_sync(0xffffffffu, x, 3 * G / 4, G);
    }
}
template <int G>
__device__ __forceinline__ double dc_group_sum(double v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int G>
__device__ __forceinline__ double dc_group_prod(double v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v *= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sqrt(max(x, 0)) for a model's discriminant: FP64 operations on the pipe are what a step costs.
__device__ __forceinline__ double dc_sqrt(double x) { return x > 1e-280 ? x * fast_rsqrt(x) : x > 0.0 ? sqrt(x) : 0.0; }

// Secular root j of 1/rho + sum_i z_i^2 / (d_i - lambda) = 0 by a group of G lanes (all lanes of
// the warp call, `act` false for groups without a root).  The root lies in (d_j, d_{j+1}) (the
// last one in (d_{k-1}, d_{k-1} + rho |z|^2)) and is found as an offset tau from the nearer pole
// d_o, so that d_i - lambda = (d_i - d_o) - tau keeps full accuracy.  The start solves the
// equation with its two nearest poles and the other terms frozen at the middle of the
// interval; each step fits c + s1/(dL - x) + s2/(dR - x) to the value and slope of the two
// partial sums at tau and takes that model's root; steps leaving the bracket bisect.  One of dL,
// dR is zero, and with s1, s2 > 0 the root between the poles is C/q for B > 0 and q/A
// otherwise (A x^2 - B x + C = 0, q its larger-magnitude half sum), so a step takes one square
// root and one division besides the pole sums.  All lanes of a group hold identical scalars.
template <int G>
__device__ void dc_secular_root(int k, int j, bool act, const double *dk, const double *zk, double rho, int &o_out,
                                double &tau_out, double &lam_out, int *status) {
    const int gl = threadIdx.x & (G - 1);
    const int kk = act ? k : 0;
    const double rhoinv = act ? 1.0 / rho : 1.0;
    const bool last = j >= k - 1;
    const double dl = act ? dk[j] : 0.0, dr = act && !last ? dk[j + 1] : 0.0;
    if (act && !last && !(dr > dl)) {   // poles out of order: give up on this root
        if (gl == 0) atomicExch(status, 1);
        o_out = j;
        tau_out = 0.0;
        lam_out = dl;
        act = false;
    }
    const double hg = last ? 0.0 : 0.5 * (dr - dl);
    const double zj2 = act ? zk[j] * zk[j] : 0.0, zr2 = act && !last ? zk[j + 1] * zk[j + 1] : 0.0;
    double x = 0.0;   // sum of the other terms at the middle of the interval, or |z|^2
    for (int i = gl; i < kk; i += G) {
        const double z2 = zk[i] * zk[i];
        if (last) x += z2;
        else if (i != j && i != j + 1) x += z2 * fast_rcp((dk[i] - dl) - hg);
    }
    x = dc_group_sum<G>(x);
    int o = j;
    double lo = 0.0, hi = 1.0, c0 = rhoinv + x;
    if (!last) {
        const double g = c0 + (zr2 - zj2) / (act ? hg : 1.0);
        if (g > 0.0) {
            hi = hg;
        } else {
            o = j + 1;
            lo = -hg;
            hi = 0.0;
        }
    } else {
        hi = rho * x;
        // the other terms at the upper end: z_j^2 / c0 is a lower bound of the root there
        double y = 0.0;
        for (int i = gl; i < kk; i += G)
            if (i != j) y += zk[i] * zk[i] * fast_rcp((dk[i] - dl) - hi);
        c0 = y;
    }
    {   // uniform shuffle for the groups of both kinds
        const double y = dc_group_sum<G>(last ? c0 : 0.0);
        if (last) c0 = rhoinv + y;
    }
    const double d_o = act ? dk[o] : 0.0;
    const double dL = dl - d_o, dR = last ? 0.0 : dr - d_o;
    double tau;
    {
        const double s1 = zj2, s2 = zr2;
        if (last) {
            tau = fmin(s1 * fast_rcp(c0), hi);
        } else {
            const double B = c0 * (dL + dR) + s1 + s2, C = s1 * dR + s2 * dL;
            const double q = 0.5 * (B + copysign(dc_sqrt(fma(B, B, -4.0 * c0 * C)), B));
            tau = B > 0.0 ? C * fast_rcp(q) : q * fast_rcp(c0);
        }
        if (!(tau > lo && (tau < hi || (last && tau == hi)))) tau = 0.5 * (lo + hi);
    }
    bool run = act;
    for (int it = 0; it < kSecularMaxIter; it++) {
        if (!__any_sync(0xffffffffu, run)) break;
        double ps = 0.0, ph = 0.0, dps = 0.0, dph = 0.0;
        if (run) {
            const int nL = j + 1;
            int i = gl;
            for (; i < nL; i += G) {
                const double r = fast_rcp((dk[i] - d_o) - tau);
                const double t = zk[i] * zk[i] * r;
                ps += t;
                dps = fma(t, r, dps);
            }
            for (; i < kk; i += G) {
                const double r = fast_rcp((dk[i] - d_o) - tau);
                const double t = zk[i] * zk[i] * r;
                ph += t;
                dph = fma(t, r, dph);
            }
        }
        dc_sum4<G>(ps, ph, dps, dph);
        if (!run) continue;
        const double g = rhoinv + ps + ph;
        const double err = 8.0 * (ph - ps) + rhoinv + fabs(tau) * (dps + dph);
        if (hi - lo <= 2.0 * kUnitRoundoff * fmax(fabs(lo), fabs(hi))) {
            run = false;
            continue;
        }
        // close enough for this step to be the last one: the model's root is quadratically closer
        if (fabs(g) <= 4.0 * kUnitRoundoff * err * k) run = false;
        if (g < 0.0) lo = tau;
        else hi = tau;
        const double a1 = dps * (dL - tau), s1 = a1 * (dL - tau);
        double cc = rhoinv + ps - a1, y;
        if (!last) {
            const double a2 = dph * (dR - tau), s2 = a2 * (dR - tau);
            cc += ph - a2;
            const double B = cc * (dL + dR) + s1 + s2, C = s1 * dR + s2 * dL;
            const double q = 0.5 * (B + copysign(dc_sqrt(fma(B, B, -4.0 * cc * C)), B));
            y = B > 0.0 ? C * fast_rcp(q) : q * fast_rcp(cc);
        } else {
            y = cc > 0.0 ? fmin(fma(s1, fast_rcp(cc), dL), hi) : NAN;   // the upper end itself is a root when k = 1
        }
        if (!(y > lo && (y < hi || (last && y == hi)))) {
            if (!run) continue;   // the last step stays where it is
            y = 0.5 * (lo + hi);
        }
        tau = y;
    }
    if (act) {
        o_out = o;
        tau_out = tau;
        lam_out = d_o + tau;
    }
}

// Levels up to nodes of kDcBase columns in one launch: a block of 128 threads merges its columns
// level by level in shared memory, four lanes per secular root.  The same steps as the level
// kernels below; separate launches took about 0.1 ms a level whatever the size (five levels
// of a 70-column problem 0.5 ms), bound by launches, scalar FP64 chains and padded tiles.
constexpr int kDcBase = 32;
__global__ void __launch_bounds__(128) dc_base_kernel(int n, const double *__restrict__ d, const double *__restrict__ e,
                                                      DcBufs b) {
    __shared__ double Q0[kDcBase][kDcBase + 1], Q1[kDcBase][kDcBase + 1], U[kDcBase][kDcBase + 1];
    __shared__ double lam[kDcBase], pd[kDcBase], pz[kDcBase], dk[kDcBase], zk[kDcBase], dv[kDcBase], lk[kDcBase],
        tau[kDcBase], zh[kDcBase], s_rho[kDcBase], rc[kDcBase], rs[kDcBase], rows[kDcBase];
    __shared__ int sp[kDcBase], st[kDcBase], kl[kDcBase], df[kDcBase], ord[kDcBase], outc[kDcBase], rp[kDcBase],
        rn[kDcBase], kcnt[kDcBase], nrot[kDcBase];
    const int c0 = blockIdx.x * kDcBase, nb = min(kDcBase, n - c0);
    const int tid = threadIdx.x, lane = tid & 31;
    double(*QA)[kDcBase + 1] = Q0, (*QB)[kDcBase + 1] = Q1;
    for (int x = tid; x < kDcBase * kDcBase; x += 128) QA[x >> 5][x & 31] = (x >> 5) == (x & 31) ? 1.0 : 0.0;
    if (tid < kDcBase) {
        const int i = c0 + tid;
        double v = 0.0;
        if (tid < nb) {
            v = d[i];
            if (i > 0) v -= fabs(e[i - 1]);
            if (i < n - 1) v -= fabs(e[i]);
        }
        lam[tid] = v;
    }
    __syncthreads();
    for (int half = 1; half < nb; half *= 2) {
        const int full = 2 * half;
        for (int x = tid; x < kDcBase * kDcBase; x += 128) QB[x >> 5][x & 31] = 0.0;
        if (tid < 32) {   // rank-one vector, merged order, deflation: lane = column, then merged position
            const int s = lane & ~(full - 1), i = lane - s, N = min(full, nb - s);
            const bool mrg = N > half, in = lane < nb && mrg;
            const unsigned nodemask = (full == 32 ? 0xffffffffu : (1u << full) - 1u) << s;
            const unsigned lt = (1u << lane) - 1u;
            const double beta = mrg ? e[c0 + s + half - 1] : 0.0;
            const double rho = 2.0 * fabs(beta), sg = beta < 0.0 ? -1.0 : 1.0;
            const double vd = lane < nb ? lam[lane] : 0.0;
            double vz = 0.0;
            if (in) vz = (i < half ? QA[s + half - 1][lane] : sg * QA[s + half][lane]) * 0.70710678118654752440;
            double mx = in ? fmax(fabs(vd), fabs(vz)) : 0.0;
            for (int o = half; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const double tol = 8.0 * kUnitRoundoff * mx;
            int pos = i < half ? i : i - half;
            for (int t = 0; t < half; t++) {   // stable merge of the two ascending halves
                const int other = i < half ? s + half + t : s + t;
                const double u = __shfl_sync(0xffffffffu, vd, other & 31);
                if (in && other < s + N) pos += i < half ? u < vd : u <= vd;
            }
            sp[lane] = lane;
            __syncwarp();
            if (in) sp[s + min(pos, N - 1)] = lane;
            __syncwarp();
            const int j = sp[lane];
            const double dj = __shfl_sync(0xffffffffu, vd, j), zj = __shfl_sync(0xffffffffu, vz, j);
            const bool keep = in && !(rho * fabs(zj) <= tol);
            const unsigned km = __ballot_sync(0xffffffffu, keep) & nodemask;
            const unsigned before = km & lt;
            const int prev = before ? 31 - __clz(before) : lane;
            const double dp = __shfl_sync(0xffffffffu, dj, prev), zp = __shfl_sync(0xffffffffu, zj, prev);
            const bool close = keep && before && dc_close(dj - dp, zp, zj, tol);
            const unsigned rm = __ballot_sync(0xffffffffu, close) & nodemask;
            pd[lane] = dj;
            pz[lane] = zj;
            st[lane] = keep;
            if (i == 0) nrot[lane] = 0;
            __syncwarp();
            if (i == 0 && rm) {   // a pair rotates: this node's first lane scans its merged order
                int nr = 0, pj = -1;
                for (int t = s; t < s + N; t++) {
                    if (!st[t]) continue;
                    if (pj >= 0 && dc_close(pd[t] - pd[pj], pz[pj], pz[t], tol)) {
                        double C, S, zt = pz[t], a = pd[pj], c = pd[t];
                        dc_rotate(a, pz[pj], c, zt, C, S);
                        rp[s + nr] = sp[pj];
                        rn[s + nr] = sp[t];
                        rc[s + nr] = C;
                        rs[s + nr] = S;
                        nr++;
                        pz[t] = zt;
                        pd[pj] = a;
                        pd[t] = c;
                        st[pj] = 0;
                    }
                    pj = t;
                }
                nrot[s] = nr;
            }
            __syncwarp();
            const bool kept = in && st[lane];
            const unsigned kf = __ballot_sync(0xffffffffu, kept) & nodemask;
            const unsigned dm = __ballot_sync(0xffffffffu, in && !kept) & nodemask;
            if (kept) {
                const int m = s + __popc(kf & lt);
                kl[m] = j;
                dk[m] = pd[lane];
                zk[m] = pz[lane];
            } else if (in) {
                const int m = s + __popc(dm & lt);
                df[m] = j;
                dv[m] = pd[lane];
            }
            if (i == 0) {
                kcnt[lane] = mrg ? __popc(kf) : -1;
                s_rho[lane] = rho;
            }
        }
        __syncthreads();
        if (tid < nb) {   // rotations of the node's columns, one row per thread
            const int s = tid & ~(full - 1);
            const int nr = kcnt[s] >= 0 ? nrot[s] : 0;
            for (int q = 0; q < nr; q++) {
                const int p = rp[s + q], r = rn[s + q];
                const double C = rc[s + q], S = rs[s + q], x = QA[tid][p], y = QA[tid][r];
                QA[tid][p] = C * x + S * y;
                QA[tid][r] = C * y - S * x;
            }
        }
        const int c = tid >> 2, gl = tid & 3, s = c & ~(full - 1), i = c - s, N = min(full, nb - s);
        const int k = c < nb ? kcnt[s] : -1;
        int o = 0;
        double tv = 0.0, lv = 0.0;
        const bool root = c < nb && i < k;
        dc_secular_root<4>(k, i, root, dk + s, zk + s, s_rho[s], o, tv, lv, b.status);
        if (root && gl == 0) {
            ord[c] = o;
            tau[c] = tv;
            lk[c] = lv;
        }
        __syncthreads();
        double p = 1.0;   // zhat_i^2 = prod_j |d_i - lambda_j| / prod_{j != i} |d_i - d_j|
        if (root) {
            const double di = dk[c];
            for (int j = gl; j < k; j += 4) {
                const double dl = fabs((di - dk[s + ord[s + j]]) - tau[s + j]);
                p *= j == i ? dl : dl * fast_rcp(fabs(dk[s + j] - di));
            }
        }
        p = dc_group_prod<4>(p);
        if (root && gl == 0) zh[c] = copysign(sqrt(p), zk[c]);
        const double v = c < nb && k >= 0 ? (i < k ? lk[c] : dv[c - k]) : 0.0;
        int r = 0;   // rank in the merged ascending order
        if (c < nb && k >= 0)
            for (int m = gl; m < N; m += 4) {
                const double u = m < k ? lk[s + m] : dv[s + m - k];
                r += (u < v) || (u == v && m < i);
            }
        r += __shfl_xor_sync(0xffffffffu, r, 1);
        r += __shfl_xor_sync(0xffffffffu, r, 2);
        if (gl == 0) outc[c] = c < nb && k >= 0 ? s + min(r, N - 1) : c;
        __syncthreads();
        double ss = 0.0;   // eigenvectors of the merge
        if (root) {
            const double dO = dk[s + ord[c]], t = tau[c];
            for (int m = gl; m < k; m += 4) {
                const double u = zh[s + m] * fast_rcp((dk[s + m] - dO) - t);
                U[s + m][c] = u;
                ss = fma(u, u, ss);
            }
        }
        ss = dc_group_sum<4>(ss);
        if (root) {
            const double inv = 1.0 / sqrt(ss);
            for (int m = gl; m < k; m += 4) U[s + m][c] *= inv;
        }
        if (gl == 0 && c < nb) rows[outc[c]] = k >= 0 ? v : lam[c];
        __syncthreads();
        if (c < nb) {
            const int oc = outc[c];
            for (int row = s + gl; row < s + N; row += 4) {
                double a = 0.0;
                if (k < 0) a = QA[row][c];
                else if (i >= k) a = QA[row][df[c - k]];
                else
                    for (int m = 0; m < k; m++) a = fma(QA[row][kl[s + m]], U[s + m][c], a);
                QB[row][oc] = a;
            }
        }
        __syncthreads();
        if (tid < kDcBase) lam[tid] = tid < nb ? rows[tid] : 0.0;
        double(*T)[kDcBase + 1] = QA;
        QA = QB;
        QB = T;
        __syncthreads();
    }
    for (int x = tid; x < nb * nb; x += 128) {
        const int r = x % nb, cc = x / nb;
        b.QA[(c0 + r) + (int64_t)(c0 + cc) * n] = QA[r][cc];
    }
    if (tid < nb) b.lamA[c0 + tid] = lam[tid];
}

// Exclusive block prefix sum of one int per thread (blockDim.x <= 1024); total gets the sum.
// Every thread of the block must call it.
__device__ int dc_block_excl_scan(int v, int *wsum, int &total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int t = lane < nw ? wsum[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        __syncwarp();
        wsum[lane] = t;
    }
    __syncthreads();
    total = wsum[nw - 1];
    const int base = (wid > 0 ? wsum[wid - 1] : 0) + x - v;
    __syncthreads();
    return base;
}

// One block per node: rank-one vector, merge order, deflation.  Deflation runs in parallel: the
// z test of every entry, then the rotation test of every neighbouring kept pair on the unrotated
// values; each maximal run of qualifying pairs is scanned by one thread, with the rotated
// values, until a test past the run's end fails (dc_deflate_scan).  A scan that reaches the next
// run would change that run's input; the block then repeats the scan in thread 0 alone.  The rotations
// themselves are applied to the eigenvector columns by dc_merge_kernel, which has the rows
// of the node spread over many blocks.  Dynamic shared memory: 20 bytes per node column.
__global__ void dc_prep_kernel(int n, int half, int full, const double *__restrict__ e, DcBufs b) {
    extern __shared__ double smem[];
    __shared__ double red[32];
    __shared__ int s_wsum[32], s_rot, s_conflict;
    const int node = blockIdx.x;
    const int s = node * full;
    const int N = min(full, n - s);
    const int n1 = half, n2 = N - half;
    if (n2 <= 0) {   // no right sibling at this level: carry the block over
        for (int i = threadIdx.x; i < N; i += blockDim.x) b.lamB[s + i] = b.lamA[s + i];
        for (int64_t x = threadIdx.x; x < (int64_t)N * N; x += blockDim.x) {
            const int r = (int)(x % N), cc = (int)(x / N);
            b.QB[(s + r) + (int64_t)(s + cc) * n] = b.QA[(s + r) + (int64_t)(s + cc) * n];
        }
        if (threadIdx.x == 0) {
            b.kcnt[node] = -1;
            b.nrot[node] = 0;
        }
        return;
    }
    double *sd = smem, *sz = smem + N;
    int *sp = reinterpret_cast<int *>(smem + 2 * N);
    const double beta = e[s + n1 - 1];
    const double rho = 2.0 * fabs(beta);
    const double sg = beta < 0.0 ? -1.0 : 1.0;
    auto source = [&](int i, double &dv, double &zv) {   // pole and component of column i, unrotated
        dv = b.lamA[s + i];
        const double q = i < n1 ? b.QA[(s + n1 - 1) + (int64_t)(s + i) * n] : sg * b.QA[(s + n1) + (int64_t)(s + i) * n];
        zv = q * 0.70710678118654752440;
    };
    double mx = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        source(i, sd[i], sz[i]);
        mx = fmax(mx, fmax(fabs(sd[i]), fabs(sz[i])));
    }
    // a valid permutation first: the merge below writes every slot exactly once for ordered
    // inputs, and with unordered ones (NaN) no slot is left holding an index out of range
    for (int i = threadIdx.x; i < N; i += blockDim.x) sp[i] = i;
    const double tol = 8.0 * kUnitRoundoff * eig_block_max(mx, red);   // syncs the block
    // stable merge of the two ascending halves
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const double v = sd[i];
        int lo, hi;
        if (i < n1) {   // count right entries strictly below v
            lo = n1;
            hi = N;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (sd[mid] < v) lo = mid + 1;
                else hi = mid;
            }
            sp[i + (lo - n1)] = i;
        } else {        // count left entries at or below v
            lo = 0;
            hi = n1;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (sd[mid] <= v) lo = mid + 1;
                else hi = mid;
            }
            sp[(i - n1) + lo] = i;
        }
    }
    __syncthreads();
    int *K0 = b.k0 + s, *close = b.flag + s, *hm = b.half + s;
    int *fold = b.ord + s;                    // scratch until the secular stage, as the next two
    double *rC = b.tau + s, *rS = b.lamK + s;
    const int per = (N + (int)blockDim.x - 1) / (int)blockDim.x;
    int k0;   // entries past the z test; the others go to defl at once
    {
        const int t0 = min(N, (int)threadIdx.x * per), t1 = min(N, t0 + per);
        int cnt = 0;
        for (int t = t0; t < t1; t++) cnt += !(rho * fabs(sz[sp[t]]) <= tol);
        int kb = dc_block_excl_scan(cnt, s_wsum, k0);
        for (int t = t0; t < t1; t++) {
            const int nj = sp[t];
            if (!(rho * fabs(sz[nj]) <= tol)) {
                K0[kb] = nj;
                hm[kb] = nj < n1 ? 1 : 2;
                kb++;
            } else {
                b.defl[s + (t - kb)] = nj;
            }
        }
        if (threadIdx.x == 0) s_rot = s_conflict = 0;
        __syncthreads();
    }
    {   // close[m]: the pair (m - 1, m) qualifies for a rotation
        int rot = 0;
        for (int m = threadIdx.x; m < k0; m += blockDim.x) {
            int t = 0;
            if (m > 0) {
                const int pj = K0[m - 1], nj = K0[m];
                t = dc_close(sd[nj] - sd[pj], sz[pj], sz[nj], tol);
            }
            close[m] = t;
            fold[m] = 0;
            rot |= t;
        }
        if (rot) atomicOr(&s_rot, 1);
        __syncthreads();
    }
    const bool any = s_rot != 0;
    if (any) {
        const DeflScan a{K0, close, fold, hm, sd, sz, rC, rS, k0, n1, tol};
        for (int m = 1 + (int)threadIdx.x; m < k0; m += blockDim.x)
            if (close[m] && !close[m - 1])
                if (dc_deflate_scan(a, m, false, source)) atomicOr(&s_conflict, 1);
        __syncthreads();
        if (s_conflict) {
            for (int i = threadIdx.x; i < N; i += blockDim.x) source(i, sd[i], sz[i]);
            for (int m = threadIdx.x; m < k0; m += blockDim.x) {
                fold[m] = 0;
                hm[m] = K0[m] < n1 ? 1 : 2;
            }
            __syncthreads();
            if (threadIdx.x == 0 && k0 > 1) dc_deflate_scan(a, 1, true, source);
            __syncthreads();
        }
    }
    // compaction: the undeflated entries, the folded ones and their rotations, and the entries
    // whose columns reach each half of the node (the others are zero there)
    {
        const int t0 = min(k0, (int)threadIdx.x * per), t1 = min(k0, t0 + per);
        int nf = 0, nt = 0, nbm = 0;
        for (int m = t0; m < t1; m++) {
            const bool gone = any && fold[m];
            nf += gone;
            if (!gone) {
                nt += hm[m] & 1;
                nbm += hm[m] >> 1;
            }
        }
        int tot_f, tot_t, tot_b;
        int fb = dc_block_excl_scan(nf, s_wsum, tot_f);
        int tb = dc_block_excl_scan(nt, s_wsum, tot_t);
        int bb = dc_block_excl_scan(nbm, s_wsum, tot_b);
        for (int m = t0; m < t1; m++) {
            const int j = K0[m];
            if (any && fold[m]) {
                b.rp[s + fb] = j;
                b.rn[s + fb] = K0[m + 1];
                b.rc[s + fb] = rC[m];
                b.rs[s + fb] = rS[m];
                b.defl[s + (N - k0) + fb] = j;
                fb++;
                continue;
            }
            const int q = m - fb;
            b.Kl[s + q] = j;
            b.dK[s + q] = sd[j];
            b.zK[s + q] = sz[j];
            if (hm[m] & 1) b.top[s + tb++] = q;
            if (hm[m] & 2) b.bot[s + bb++] = q;
        }
        __syncthreads();
        const int nd = N - k0 + tot_f;
        for (int m = threadIdx.x; m < nd; m += blockDim.x) b.dv[s + m] = sd[b.defl[s + m]];
        if (threadIdx.x == 0) {
            b.kcnt[node] = k0 - tot_f;
            b.ndef[node] = nd;
            b.nrot[node] = tot_f;
            b.ntop[node] = tot_t;
            b.nbot[node] = tot_b;
            b.rho[node] = rho;
        }
    }
}

// One group of G lanes per secular root (dc_secular_root).
template <int G>
__global__ void dc_secular_kernel(int n, int full, DcBufs b) {
    const int w = (int)((blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G);
    const int node = w < n ? w / full : 0, s = node * full, j = w - s;
    const int k = b.kcnt[node];
    const bool act = w < n && k >= 0 && j < k;
    int o = 0;
    double tau = 0.0, lam = 0.0;
    dc_secular_root<G>(k, j, act, b.dK + s, b.zK + s, act ? b.rho[node] : 1.0, o, tau, lam, b.status);
    if (act && (threadIdx.x & (G - 1)) == 0) {
        b.ord[s + j] = o;
        b.tau[s + j] = tau;
        b.lamK[s + j] = lam;
    }
}

// After the secular stage, one launch for three independent jobs, by block: [0, nz) recompute the
// rank-one vector (one warp per undeflated entry i, zhat_i^2 = prod_j |d_i - lambda_j| /
// prod_{j != i} |d_i - d_j| up to the common factor 1/rho, sign of z_i), [nz, 2 nz) rank the
// node's eigenvalues (one warp per entry: its column in the next level, ties by entry index),
// and [2 nz, ...) apply the deflation's rotations (32 rows per block; the warps take
// contiguous shares of the rotation list cut where a new chain of columns begins).
constexpr int DM_THREADS = 64, DM_ROT_ROWS = 32, DM_ROT_SHARES = DM_THREADS / 32;
__global__ void __launch_bounds__(DM_THREADS) dc_merge_kernel(int n, int full, int nz, DcBufs b) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int role = (int)blockIdx.x < nz ? 0 : (int)blockIdx.x < 2 * nz ? 1 : 2;
    if (role < 2) {
        const int g = ((int)blockIdx.x - role * nz) * (DM_THREADS / 32) + wib;
        if (g >= n) return;
        const int node = g / full, s = node * full, i = g - s;
        const int k = b.kcnt[node];
        if (k < 0) return;
        if (role == 0) {
            if (i >= k) return;
            const double *dk = b.dK + s;
            const double di = dk[i];
            double p = 1.0;
            for (int j = lane; j < k; j += 32) {
                const double dl = fabs((di - dk[b.ord[s + j]]) - b.tau[s + j]);
                p *= (j == i) ? dl : dl * fast_rcp(fabs(dk[j] - di));
            }
            p = eig_warp_prod(p);
            if (lane == 0) b.zh[s + i] = copysign(sqrt(p), b.zK[s + i]);
            return;
        }
        const int N = k + b.ndef[node];
        if (i >= N) return;
        const double v = i < k ? b.lamK[s + i] : b.dv[s + i - k];
        int r = 0;
        for (int m = lane; m < N; m += 32) {
            const double u = m < k ? b.lamK[s + m] : b.dv[s + m - k];
            r += (u < v) || (u == v && m < i);
        }
        r = __reduce_add_sync(0xffffffffu, r);
        if (lane == 0) {
            b.lamB[s + r] = v;
            b.outc[s + i] = s + r;
        }
        return;
    }
    const int row = ((int)blockIdx.x - 2 * nz) * DM_ROT_ROWS + lane;
    const int node = min(row, n - 1) / full, s = node * full;   // full >= 32: the same for the whole warp
    const int nr = b.nrot[node];
    if (nr == 0 || row >= n) return;
    auto cut = [&](int q) {   // first chain start at or after q
        while (q > 0 && q < nr && b.rp[s + q] == b.rn[s + q - 1]) q++;
        return q;
    };
    const int q0 = cut((int)((int64_t)wib * nr / DM_ROT_SHARES)), q1 = cut((int)((int64_t)(wib + 1) * nr / DM_ROT_SHARES));
    double *Q = b.QA + row + (int64_t)s * n;
    for (int q = q0; q < q1; q++) {
        const int64_t op = (int64_t)b.rp[s + q] * n, on = (int64_t)b.rn[s + q] * n;
        const double C = b.rc[s + q], S = b.rs[s + q], x = Q[op], y = Q[on];
        Q[op] = C * x + S * y;
        Q[on] = C * y - S * x;
    }
}

// One block per node entry with an output column in [olo, ohi): column of the merge eigenvector
// matrix (undeflated entries), or the copy of a deflated eigenvector into its output column.
__global__ void dc_vec_kernel(int n, int full, int olo, int ohi, DcBufs b) {
    __shared__ double red[32];
    const int g = blockIdx.x;
    const int node = g / full, s = node * full, i = g - s;
    const int k = b.kcnt[node];
    if (k < 0) return;
    const int N = k + b.ndef[node];
    if (i >= N) return;
    const int oc = b.outc[s + i];
    if (oc < olo || oc >= ohi) return;
    if (i < k) {
        const double *dk = b.dK + s;
        const double dO = dk[b.ord[s + i]], t = b.tau[s + i];
        double *u = b.U + s + (int64_t)(s + i) * n;
        double ss = 0.0;
        for (int m = threadIdx.x; m < k; m += blockDim.x) {
            const double v = b.zh[s + m] * fast_rcp((dk[m] - dO) - t);
            u[m] = v;
            ss = fma(v, v, ss);
        }
        const double inv = 1.0 / sqrt(eig_block_sum(ss, red));
        for (int m = threadIdx.x; m < k; m += blockDim.x) u[m] *= inv;
    } else {
        const int64_t src = (int64_t)(s + b.defl[s + i - k]) * n, dst = (int64_t)oc * n;
        for (int r = threadIdx.x; r < N; r += blockDim.x) b.QB[(s + r) + dst] = b.QA[(s + r) + src];
    }
}

// QB(rows of node, outc[j]) = QA(rows of node, Kl[m]) * U(m, j) for the undeflated entries with
// outc[j] in [olo, ohi), batched over nodes (blockIdx.z).  QA is block diagonal by the two halves of
// the node, so a row of the first half sums over the entries of `top` alone and one of the
// second half over `bot`: half the products.  One 16 x 16 output tile per block, one output per
// thread (row tiles do not cross the halves): the FP64 unit is the limit at any tile, and
// small tiles fill the SMs evenly (n = 791: 13 x 13 tiles of 64 left 152 SMs with one or two each).
constexpr int DG_T = 16, DG_K = 32;
__global__ void __launch_bounds__(256) dc_gemm_kernel(int n, int half, int full, int olo, int ohi, DcBufs b) {
    __shared__ double As[DG_K][DG_T + 1];
    __shared__ double Bs[DG_K][DG_T + 1];
    __shared__ int s_need;
    const int node = blockIdx.z, s = node * full;
    const int k = b.kcnt[node];
    if (k <= 0) return;
    const int N = min(full, n - s);
    const int tt = (half + DG_T - 1) / DG_T;   // row tiles of the first half
    const bool first = (int)blockIdx.x < tt;
    const int r0 = first ? blockIdx.x * DG_T : half + ((int)blockIdx.x - tt) * DG_T, rend = first ? half : N;
    const int c0 = blockIdx.y * DG_T;
    if (r0 >= rend || c0 >= k) return;
    const int *list = (first ? b.top : b.bot) + s;
    const int nl = first ? b.ntop[node] : b.nbot[node];
    const int tid = threadIdx.x, lane = tid & 31, w = ((tid >> 5) + (int)blockIdx.x + (int)blockIdx.y) & 7;
    const int li = 8 * (w & 1) + (lane & 7), lj = 4 * (w >> 1) + (lane >> 3);
    const int gr = r0 + li, gc = c0 + lj;
    const int oc = gc < k ? b.outc[s + gc] : -1;
    const bool want = gc < k && oc >= olo && oc < ohi;
    if (tid == 0) s_need = 0;
    __syncthreads();
    if (want) s_need = 1;
    __syncthreads();
    if (!s_need) return;
    const bool busy = __any_sync(0xffffffffu, want && gr < rend);
    // chunk element loads: A (row fastest) and B (m fastest), two per thread
    double pa[2], pb[2];
    auto fetch = [&](int m0) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int x = tid + 256 * u;
            const int rr = x % DG_T, km = x / DG_T;
            pa[u] = (r0 + rr < rend && m0 + km < nl) ? b.QA[(s + r0 + rr) + (int64_t)(s + b.Kl[s + list[m0 + km]]) * n] : 0.0;
            const int kb = x % DG_K, cc = x / DG_K;
            pb[u] = (m0 + kb < nl && c0 + cc < k) ? b.U[(s + list[m0 + kb]) + (int64_t)(s + c0 + cc) * n] : 0.0;
        }
    };
    double a0 = 0.0, a1 = 0.0;
    fetch(0);
    for (int m0 = 0; m0 < nl; m0 += DG_K) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int x = tid + 256 * u;
            As[x / DG_T][x % DG_T] = pa[u];
            Bs[x % DG_K][x / DG_K] = pb[u];
        }
        __syncthreads();
        if (m0 + DG_K < nl) fetch(m0 + DG_K);
        if (busy) {
            const int kend = min(DG_K, nl - m0);
            if (kend == DG_K) {
#pragma unroll 8
                for (int q = 0; q < DG_K; q += 2) {
                    a0 = fma(As[q][li], Bs[q][lj], a0);
                    a1 = fma(As[q + 1][li], Bs[q + 1][lj], a1);
                }
            } else {
                for (int q = 0; q < kend; q++) a0 = fma(As[q][li], Bs[q][lj], a0);
            }
        }
        __syncthreads();
    }
    if (want && gr < rend) b.QB[(s + gr) + (int64_t)oc * n] = a0 + a1;
}

// Largest divide-and-conquer dimension: the merge scan keeps 20 bytes per column in shared
// memory (227 KB per block).
constexpr int kDcMaxN = 11264;

static std::string slot_name(const char *base, int slot) { return std::string(base) + "#" + std::to_string(slot); }

static DcBufs dc_bufs(Context &c, int n, int slot) {
    DcBufs b;
    const size_t nn = (size_t)n * n;
    auto nm = [&](const char *x) { return slot_name(x, slot); };
    b.QA = wsget<double>(c, nm("dc.QA"), nn);
    b.QB = wsget<double>(c, nm("dc.QB"), nn);
    b.U = wsget<double>(c, nm("dc.U"), nn);
    // the vectors of one slot in two allocations: 11 of doubles, 16 of integers
    const size_t m = (size_t)n + 8;
    double *f = wsget<double>(c, nm("dc.f"), 11 * m);
    b.lamA = f, b.lamB = f + m, b.dK = f + 2 * m, b.zK = f + 3 * m, b.dv = f + 4 * m, b.rc = f + 5 * m;
    b.rs = f + 6 * m, b.tau = f + 7 * m, b.lamK = f + 8 * m, b.zh = f + 9 * m, b.rho = f + 10 * m;
    int *q = wsget<int>(c, nm("dc.i"), 16 * m);
    b.Kl = q, b.defl = q + m, b.rp = q + 2 * m, b.rn = q + 3 * m, b.ord = q + 4 * m, b.outc = q + 5 * m;
    b.top = q + 6 * m, b.bot = q + 7 * m, b.k0 = q + 8 * m, b.flag = q + 9 * m, b.half = q + 10 * m;
    b.kcnt = q + 11 * m, b.ndef = q + 12 * m, b.nrot = q + 13 * m, b.ntop = q + 14 * m, b.nbot = q + 15 * m;
    b.status = b.nbot + n + 4;
    return b;
}

// The merge eigenvectors of one level and their product with the children's, for output columns
// [olo, ohi) of the whole matrix.
static void dc_level_vectors(Context &c, int n, int half, int olo, int ohi, const DcBufs &b) {
    const int full = 2 * half, nodes = (n + full - 1) / full;
    dc_vec_kernel<<<n, 128, 0, c.stream>>>(n, full, olo, ohi, b);
    DCG_LAUNCHED(c);
    const int tt = (half + DG_T - 1) / DG_T, tb = (std::min(full, n) - half + DG_T - 1) / DG_T;
    dim3 gg(tt + std::max(tb, 1), grid1d(std::min(full, n), DG_T), nodes);
    dc_gemm_kernel<<<gg, 256, 0, c.stream>>>(n, half, full, olo, ohi, b);
    DCG_LAUNCHED(c);
}

// Bound by latency (launches, serial FP64 chains) below a few hundred columns and by the FP64
// pipe above.  Order 791, values: 2.4 ms with the base kernel, four launches a level, the short
// secular steps and the merge products by halves; 6 ms with six launches a level from 1 x 1
// leaves and divisions.
// Eigenvalues (ascending, into w) of the symmetric tridiagonal (d, e), and its eigenvectors up to
// the last merge, whose own vectors dc_vectors forms for the columns that are asked for (most
// of the merge products of a decomposition are the last one's).  d and e are device arrays;
// e has n-1 entries.
static void tridiag_dc(Context &c, int n, const double *d, const double *e, double *w, int slot) {
    if (n > kDcMaxN)
        throw Error{DCG_E_ARG, "eigensolver dimension " + std::to_string(n) + " exceeds " + std::to_string(kDcMaxN)};
    DcBufs b = dc_bufs(c, n, slot);
    // Both buffers start at zero: rotations and deflated copies touch whole columns of a node
    // block, including the cross blocks between its two children, which no earlier level writes.
    DCG_CUDA(cudaMemsetAsync(b.QA, 0, sizeof(double) * (size_t)n * n, c.stream));
    if (n > kDcBase) DCG_CUDA(cudaMemsetAsync(b.QB, 0, sizeof(double) * (size_t)n * n, c.stream));
    DCG_CUDA(cudaMemsetAsync(b.status, 0, sizeof(int), c.stream));
    dc_base_kernel<<<grid1d(n, kDcBase), 128, 0, c.stream>>>(n, d, e, b);
    DCG_LAUNCHED(c);
    c.eig_n[slot] = n;
    c.eig_status[slot] = b.status;
    c.eig_Q[slot] = b.QA;
    c.eig_last[slot] = 0;
    DCG_CUDA(cudaFuncSetAttribute(dc_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 20 * kDcMaxN));
    for (int half = kDcBase; half < n; half *= 2) {
        const int full = 2 * half;
        const int nodes = (n + full - 1) / full;
        const int nmax = std::min(full, n);
        dc_prep_kernel<<<nodes, 256, 20 * (size_t)nmax, c.stream>>>(n, half, full, e, b);
        DCG_LAUNCHED(c);
        // a warp per root while that is about one warp per quarter SM, half a warp for more
        // roots (a root's scalar steps cost as much as eight poles a lane); blocks of two
        // warps reach every SM
        if (n <= 4 * std::max(1, c.num_sms)) dc_secular_kernel<32><<<grid1d((int64_t)n * 32, 64), 64, 0, c.stream>>>(n, full, b);
        else dc_secular_kernel<16><<<grid1d((int64_t)n * 16, 64), 64, 0, c.stream>>>(n, full, b);
        DCG_LAUNCHED(c);
        const int nz = (int)grid1d((int64_t)n * 32, DM_THREADS);
        dc_merge_kernel<<<2 * nz + grid1d(n, DM_ROT_ROWS), DM_THREADS, 0, c.stream>>>(n, full, nz, b);
        DCG_LAUNCHED(c);
        std::swap(b.lamA, b.lamB);
        if (full >= n) {
            c.eig_last[slot] = half;
            c.eig_Q[slot] = nullptr;   // formed on request
            break;
        }
        dc_level_vectors(c, n, half, 0, n, b);
        std::swap(b.QA, b.QB);
    }
    DCG_CUDA(cudaMemcpyAsync(w, b.lamA, sizeof(double) * n, cudaMemcpyDeviceToDevice, c.stream));
}

// Columns [vlo, vhi) of the tridiagonal's eigenvectors of the slot's last tridiag_dc (n x n,
// ld n; other columns are undefined).
static const double *dc_vectors(Context &c, int slot, int n, int vlo, int vhi) {
    const int half = c.eig_last[slot];
    if (half == 0) return c.eig_Q[slot];
    DcBufs b = dc_bufs(c, n, slot);
    int swaps = 0;
    for (int h = kDcBase; h < half; h *= 2) swaps++;
    if (swaps & 1) std::swap(b.QA, b.QB);
    dc_level_vectors(c, n, half, vlo, vhi, b);
    return b.QB;
}

// ===================================================================== 3. back-transformation
// Z = H_0 H_1 ... H_{n-2} Qt(:, vlo:vhi), applied in panels of WY_NB reflectors: the product
// of a panel H_k0 ... H_{k0+nb-1} is I - V T V^H with T upper triangular (the compact WY form
// of Schreiber & Van Loan, SIAM J. Sci. Stat. Comput. 10 (1989) 53), built by the forward
// recurrence T(0:i, i) = -tau_i T(0:i, 0:i) (V(:, 0:i)^H v_i).  Each panel costs three GEMMs.
constexpr int WY_NB = 64;

__global__ void z_from_real_kernel(int n, const double *__restrict__ Qt, int vlo, int nvec, cplx *Z, int64_t ldz) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n * nvec) return;
    const int i = (int)(idx % n), c = (int)(idx / n);
    Z[i + (int64_t)c * ldz] = mk(Qt[i + (int64_t)(vlo + c) * n], 0.0);
}

// Panel p starts at this element of the packed reflectors (all panels before are full).
__host__ __device__ __forceinline__ int64_t wy_offset(int n, int p) {
    return (int64_t)WY_NB * ((int64_t)p * (n - 1) - (int64_t)WY_NB * p * (p - 1) / 2);
}

// Panel reflectors k0..k0+nbp-1 as a dense (m0 x nbp) matrix, m0 = n-k0-1, row r = global
// row k0+1+r: zero above each reflector's unit entry.  blockIdx.y is the panel.
__global__ void wy_extract_kernel(int n, const cplx *__restrict__ A, int64_t lda, cplx *Vp) {
    const int k0 = blockIdx.y * WY_NB, nbp = min(WY_NB, n - 1 - k0), m0 = n - k0 - 1;
    Vp += wy_offset(n, blockIdx.y);
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (idx >= (int64_t)m0 * nbp) return;
    const int r = (int)(idx % m0), jj = (int)(idx / m0);
    cplx v = mk(0.0, 0.0);
    if (r == jj) v = mk(1.0, 0.0);
    else if (r > jj) v = A[(k0 + 1 + r) + (int64_t)(k0 + jj) * lda];
    Vp[r + (int64_t)jj * m0] = v;
}

// T (nbp x nbp, ld WY_NB) from G = Vp^H Vp and tau[k0..]; one block of WY_NB threads a panel
// with G and T staged in shared memory.  The recurrence is sequential in i and takes 0.36 ms
// however few SMs work, so all panels go in one launch before the first is applied
// (40/14/800: 84 launches, 30.7 ms -> 3 launches, 1 ms).
__global__ void wy_tfactor_kernel(int n, const cplx *__restrict__ G, const cplx *__restrict__ tau, cplx *T) {
    extern __shared__ cplx wy_sm[];
    const int k0 = blockIdx.x * WY_NB, nbp = min(WY_NB, n - 1 - k0);
    G += (int64_t)blockIdx.x * WY_NB * WY_NB;
    T += (int64_t)blockIdx.x * WY_NB * WY_NB;
    cplx *Gs = wy_sm, *Ts = wy_sm + WY_NB * WY_NB;
    const int j = threadIdx.x;
    for (int x = j; x < WY_NB * WY_NB; x += blockDim.x) {
        Ts[x] = mk(0.0, 0.0);
        const int r = x % WY_NB, cc = x / WY_NB;
        Gs[x] = (r < nbp && cc < nbp) ? G[r + cc * nbp] : mk(0.0, 0.0);
    }
    __syncthreads();
    for (int i = 0; i < nbp; i++) {
        const cplx ti = tau[k0 + i];
        cplx acc = mk(0.0, 0.0);
        if (j < i)
            for (int l = j; l < i; l++) cfma(acc, Ts[j + l * WY_NB], Gs[l + i * WY_NB]);
        __syncthreads();
        if (j < i) Ts[j + i * WY_NB] = cmul(mk(-ti.x, -ti.y), acc);
        if (j == i) Ts[i + i * WY_NB] = ti;
        __syncthreads();
    }
    for (int x = j; x < WY_NB * WY_NB; x += blockDim.x) T[x] = Ts[x];
}

// f = t (sum of s over the column's WPC warps), the same in every lane.  The lower half of a
// warp sums the real part and the upper half the imaginary part, and each forms its part of f:
// 8 FP64 instructions where both in every lane take 16 of the 72 of a 791-row reflector in
// two warps (two times 791 vectors of order 791: 9.8 -> 9.3 ms).  The caller alternates `part`
// between two buffers from one applied reflector to the next, so one barrier each is enough: a
// buffer is written again only after the barrier of the reflector between, which the other warp
// reaches when it has read the old sums.  Reflectors with tau = 0 are skipped and have no
// barrier, so they do not count (by the reflector's number, two applied ones around a skipped
// one would share a buffer with nothing between them).
template <int WPC, bool REAL>
__device__ __forceinline__ void bt_scale(double sr, double si, cplx t, int wsub, double (&part)[2][2], double &fr,
                                         double &fi) {
    const int lane = threadIdx.x & 31;
    if (REAL) {
        for (int o = 16; o > 0; o >>= 1) sr += __shfl_xor_sync(0xffffffffu, sr, o);
        if (WPC == 2) {
            if (lane == 0) part[wsub][0] = sr;
            __syncthreads();
            sr = part[0][0] + part[1][0];
        }
        fr = t.x * sr;
        fi = 0.0;
        return;
    }
    const int h = lane >> 4;
    double s = h ? si : sr;
    s += __shfl_xor_sync(0xffffffffu, h ? sr : si, 16);
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (WPC == 2) {   // the two warps' sums, in a fixed order
        if ((lane & 15) == 0) part[wsub][h] = s;
        __syncthreads();
        s = part[0][h] + part[1][h];
    }
    const double other = __shfl_xor_sync(0xffffffffu, s, 16);
    // Re f = t.x Re s - t.y Im s, Im f = t.x Im s + t.y Re s
    const double ty = __hiloint2double(__double2hiint(t.y) ^ (h ? 0 : (int)0x80000000), __double2loint(t.y));
    const double f = fma(t.x, s, ty * other);
    fr = __shfl_sync(0xffffffffu, f, 0);
    fi = __shfl_sync(0xffffffffu, f, 16);
}

// Register-resident back-transformation (n <= 32 R WPC): WPC warps per eigenvector column,
// the column held in registers (warp w, lane l owns rows l + 32 (WPC i + w)), the reflectors
// applied from the last to the first.  Reflector k-1 is loaded into registers while reflector
// k is applied, so the per-reflector chain is FMAs and shuffles only; this matters most for a
// single column (a CASCI root: n-1 strictly sequential reflections).  With two warps per
// column their partial dot products meet in double-buffered shared memory, summed in a fixed
// order.  Columns are independent, and the FP64 work (8 FMAs per row and reflector) spreads
// over every SM.
template <int R, int WPC, bool PF, bool REAL>
__global__ void __launch_bounds__(64) backtransform_reg_kernel(int n, const cplx *__restrict__ A, int64_t lda,
                                                                const cplx *__restrict__ tau,
                                                                const double *__restrict__ Qt, int vlo, int nvec,
                                                                cplx *Z, int64_t ldz) {
    __shared__ double part[2][2][2];   // [buffer][warp][re, im]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wsub = warp % WPC;                               // warp within its column
    const int col = blockIdx.x * (2 / WPC) + warp / WPC;       // 64 threads: 2 / WPC columns
    const bool have = col < nvec;
    cplx z[R], vc[PF ? R : 1], vn[PF ? R : 1];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int r = lane + 32 * (WPC * i + wsub);
        z[i] = (have && r < n) ? mk(Qt[r + (int64_t)(vlo + col) * n], 0.0) : mk(0.0, 0.0);
    }
#define BT_LOAD(kk, dst)                                                                     \
    {                                                                                        \
        const cplx *v_ = A + (int64_t)(kk) * lda;                                            \
        _Pragma("unroll") for (int i = 0; i < R; i++) {                                      \
            const int r = lane + 32 * (WPC * i + wsub);                                      \
            dst[i] = (have && r > (kk) && r < n) ? __ldg(v_ + r) : mk(0.0, 0.0);             \
        }                                                                                    \
    }
    if (PF && n >= 2) BT_LOAD(n - 2, vc);
    int applied = 0;   // reflectors that were not skipped
    for (int k = n - 2; k >= 0; k--) {
        if (PF && k >= 1) BT_LOAD(k - 1, vn);
        const cplx t = __ldg(tau + k);
        if (t.x != 0.0 || t.y != 0.0) {   // uniform over the block
            const int i0 = (k + 1) / (32 * WPC);   // row chunks below k+1 hold v = 0 in every lane
            double s0r = 0.0, s0i = 0.0, s1r = 0.0, s1i = 0.0;
            const cplx *vk = A + (int64_t)k * lda;
#pragma unroll
            for (int i = 0; i < R; i++) {
                if (i < i0) continue;
                cplx vv;
                if (PF) {
                    vv = vc[i];
                } else {   // read from L1/L2 (shared by the SM's warps) instead of holding it
                    const int r = lane + 32 * (WPC * i + wsub);
                    vv = (have && r > k && r < n) ? __ldg(vk + r) : mk(0.0, 0.0);
                }
                if (i & 1) {   // conj(v) z, two accumulator chains
                    s1r = fma(vv.x, z[i].x, s1r);
                    if (!REAL) {
                        s1r = fma(vv.y, z[i].y, s1r);
                        s1i = fma(vv.x, z[i].y, s1i);
                        s1i = fma(-vv.y, z[i].x, s1i);
                    }
                } else {
                    s0r = fma(vv.x, z[i].x, s0r);
                    if (!REAL) {
                        s0r = fma(vv.y, z[i].y, s0r);
                        s0i = fma(vv.x, z[i].y, s0i);
                        s0i = fma(-vv.y, z[i].x, s0i);
                    }
                }
            }
            double fr, fi;   // f = tau (v^H z)
            bt_scale<WPC, REAL>(s0r + s1r, REAL ? 0.0 : s0i + s1i, t, wsub, part[applied++ & 1], fr, fi);
#pragma unroll
            for (int i = 0; i < R; i++) {
                if (i < i0) continue;
                cplx vv;
                if (PF) {
                    vv = vc[i];
                } else {
                    const int r = lane + 32 * (WPC * i + wsub);
                    vv = (have && r > k && r < n) ? __ldg(vk + r) : mk(0.0, 0.0);
                }
                z[i].x = fma(-vv.x, fr, z[i].x);   // z -= v f
                if (!REAL) {
                    z[i].x = fma(vv.y, fi, z[i].x);
                    z[i].y = fma(-vv.x, fi, z[i].y);
                    z[i].y = fma(-vv.y, fr, z[i].y);
                }
            }
        }
        if (PF) {
#pragma unroll
            for (int i = 0; i < R; i++) vc[i] = vn[i];
        }
    }
#undef BT_LOAD
    if (have) {
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int r = lane + 32 * (WPC * i + wsub);
            if (r < n) Z[r + (int64_t)col * ldz] = z[i];
        }
    }
}

template <int R, int WPC, bool PF>
static void launch_bt_reg(Context &c, int n, const cplx *A, int64_t lda, const cplx *tau, const double *Qt, int vlo,
                          int nvec, cplx *Z, int64_t ldz) {
    auto *kern = c.real_now ? backtransform_reg_kernel<R, WPC, PF, true> : backtransform_reg_kernel<R, WPC, PF, false>;
    kern<<<grid1d(nvec, 2 / WPC), 64, 0, c.stream>>>(n, A, lda, tau, Qt, vlo, nvec, Z, ldz);
    DCG_LAUNCHED(c);
}

// ===================================================================== driver
struct HeevWork {
    double *d, *e;
    cplx *tau, *ppart, *w;
};

static HeevWork heev_work(Context &c, int n, int slot) {
    HeevWork h;
    h.d = wsget<double>(c, slot_name("heev.d", slot), n + 1);
    h.e = wsget<double>(c, slot_name("heev.e", slot), n + 1);
    h.tau = wsget<cplx>(c, slot_name("heev.tau", slot), n + 1);
    int nchunk = (n + HH_CHUNK - 1) / HH_CHUNK;
    h.ppart = wsget<cplx>(c, slot_name("heev.ppart", slot), (size_t)nchunk * (n + 1));
    h.w = wsget<cplx>(c, slot_name("heev.w", slot), n + 1);
    return h;
}

// Cooperative launches from different contexts (a serving process runs one context per
// slot, each on its own stream) are serialised from launch to completion: two grid-synchronised
// kernels must never wait for each other's SMs.
static std::mutex g_coop_mutex;

static uint64_t trd_wait_limit(const Context &c) { return c.wait_limit_ns ? c.wait_limit_ns : kBarrierLimitNs; }

// A fresh barrier (counters and error flag zero) with the context's wait limit, written in
// stream order (a copy from pageable host memory is staged before the call returns).
static void gridbar_reset(Context &c, GridBar *gb) {
    GridBar x{};
    x.limit_ns = trd_wait_limit(c);
    DCG_CUDA(cudaMemcpyAsync(gb, &x, sizeof(GridBar), cudaMemcpyHostToDevice, c.stream));
}

static void tridiag_persistent(Context &c, int n, cplx *A, int64_t lda, HeevWork &h) {
    std::lock_guard<std::mutex> coop(g_coop_mutex);
    const size_t smem = 2 * sizeof(cplx) * (size_t)std::max(n - 1, 1);
    DCG_CUDA(cudaFuncSetAttribute(tridiag_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    DCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tridiag_persistent_kernel, TRD_THREADS, smem));
    if (per_sm < 1) throw Error{DCG_E_CUDA, "tridiagonalisation kernel does not fit on an SM"};
    // one warp per trailing column at most; never more blocks than can be co-resident
    const int want = std::max(1, (n + (TRD_THREADS / 32) - 1) / (TRD_THREADS / 32));
    const int nblocks = std::min({want, per_sm * std::max(1, c.num_sms), 2 * std::max(1, c.num_sms)});
    cplx *pbuf = wsget<cplx>(c, "trd.p", (size_t)n + 1);
    double2 *part = wsget<double2>(c, "trd.part", (size_t)nblocks + 1);
    GridBar *gb = wsget<GridBar>(c, "trd.bar", 1);
    gridbar_reset(c, gb);
    void *args[] = {&n, &A, &lda, &h.d, &h.e, &h.tau, &pbuf, &part, &gb};
    DCG_CUDA(cudaLaunchCooperativeKernel((const void *)tridiag_persistent_kernel, dim3(nblocks), dim3(TRD_THREADS),
                                         args, smem, c.stream));
    DCG_LAUNCHED(c);
    GridBar hb;
    DCG_CUDA(cudaMemcpyAsync(&hb, gb, sizeof(GridBar), cudaMemcpyDeviceToHost, c.stream));
    DCG_CUDA(cudaStreamSynchronize(c.stream));
    if (hb.err) throw Error{DCG_E_NUMERIC, "tridiagonalisation: a grid barrier wait timed out"};
}

// Shared-memory tridiagonalisation of several matrices in one cooperative launch (one job = one
// block group).  Block counts come from a cost model: a job's FP64 work (12 FMAs per trailing
// element and column, whole columns per block, on a unit of 1.66 FMAs per clock and SM) spreads
// over its blocks, while every block of a column reads all of its exchanged words; the jobs
// share the SMs, and blocks go to the job that is currently the slowest.  False (nothing
// launched) when the jobs do not fit.
static double trd_cost(const TrdJob &j, int nb) {
    const double n = j.n, fma = (j.real ? 3.0 : 12.0) / 3.8e9;
    const double own = std::ceil(n / nb);   // a block's columns also follow one another in its reductions
    return fma * (n * n * n / (3.0 * nb) + n * n / 4.0) +
           n * ((nb > 1 ? 4.3e-6 : 3.2e-6) + 0.3e-6 * own + 0.002e-6 * nb);
}

// v and w, the owned columns and their partial sums
static size_t trd_bytes_for(int n, int nbk) {
    const size_t nown = (size_t)(n + nbk - 1) / nbk;
    return (nown + 2) * n * sizeof(cplx) + nown * 8 * sizeof(double);
}

// Shared-memory limit of one block of the batched kernel (its static shared memory aside).
static size_t trd_smem_limit(const Context &c) {
    int optin = 0;
    DCG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c.device));
    return (size_t)std::max(0, optin - 1024);
}

// Block groups of one batched launch: every job gets the fewest blocks whose shared memory holds
// its columns, then the remaining SMs go one by one to the job that is currently the slowest
// and that they help (trd_cost); b0 and the largest block's shared memory follow.  False when
// the jobs do not fit one launch.
static bool trd_plan(const Context &c, std::vector<TrdJob> &jobs, int &total, size_t &smem) {
    const int sms = std::max(1, c.num_sms);
    const size_t limit = trd_smem_limit(c);
    total = 0;
    if (jobs.size() > (size_t)kTrdMaxJobs) return false;
    for (TrdJob &j : jobs) {
        if (j.n > kTridiagSmemMaxN) return false;
        int nb = 1;
        while (nb < std::min(sms, j.n) && trd_bytes_for(j.n, nb) > limit) nb++;
        if (trd_bytes_for(j.n, nb) > limit) return false;
        j.nb = nb;
        total += nb;
    }
    if (total > sms) return false;
    while (total < sms) {   // give the next blocks to the slowest job that they help
        int best = -1, add = 1;
        double worst = -1.0;
        for (size_t q = 0; q < jobs.size(); q++) {
            const TrdJob &j = jobs[q];
            // one block pays no exchange, so the second may only pay together with more
            int up = 0;
            for (int t : {1, 2, 4, 8, 16})
                if (up == 0 && j.nb + t <= j.n && total + t <= sms && trd_cost(j, j.nb + t) < trd_cost(j, j.nb)) up = t;
            if (up == 0) continue;
            const double cst = trd_cost(j, j.nb);
            if (cst > worst) {
                worst = cst;
                best = (int)q;
                add = up;
            }
        }
        if (best < 0) break;
        jobs[best].nb += add;
        total += add;
    }
    smem = 0;
    int b0 = 0;
    for (TrdJob &j : jobs) {
        smem = std::max(smem, trd_bytes_for(j.n, j.nb));
        j.b0 = b0;
        b0 += j.nb;
    }
    DCG_CUDA(cudaFuncSetAttribute(tridiag_smem_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    int per_sm = 0;
    DCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tridiag_smem_batched_kernel, TRS_THREADS, smem));
    return per_sm >= 1 && total <= per_sm * sms;
}

// The exchange words of a context's jobs start at zero, in stream order.
static void trd_clear(Context &c, const std::vector<TrdJob> &jobs) {
    for (const TrdJob &j : jobs)
        if (j.nb != 1) DCG_CUDA(cudaMemsetAsync(j.ll, 0, trd_ll_words(j.n) * sizeof(ulonglong2), c.stream));
}

// The launch of planned jobs on `stream` (their exchange words already cleared in stream order):
// cooperative, or with ncta > 0 one cluster of ncta blocks per job.  Returns each job's error
// flag, read back after the launch completes.
static std::vector<int> trd_launch(Context &c, const std::vector<TrdJob> &jobs, int total, size_t smem,
                                   cudaStream_t stream, const char *table, int ncta = 0, bool global = false) {
    const size_t nj = jobs.size();
    TrdTable T{};
    for (size_t q = 0; q < nj; q++) T.j[q] = jobs[q];
    T.njobs = (int)nj;
    T.err = wsget<int>(c, table, kTrdMaxJobs);
    int *herr = (int *)c.ws.host(table, kTrdMaxJobs * sizeof(int));
    DCG_CUDA(cudaMemsetAsync(T.err, 0, nj * sizeof(int), stream));
    if (ncta > 0) {
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)ncta;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)total);
        cfg.blockDim = dim3(TRS_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        DCG_CUDA(cudaLaunchKernelEx(&cfg, tridiag_smem_batched_kernel, T));
    } else {
        void *args[] = {&T};
        const void *kern = global ? (const void *)tridiag_global_kernel : (const void *)tridiag_smem_batched_kernel;
        DCG_CUDA(cudaLaunchCooperativeKernel(kern, dim3(total), dim3(TRS_THREADS), args, smem, stream));
    }
    DCG_CUDA(cudaGetLastError());
    DCG_CUDA(cudaMemcpyAsync(herr, T.err, nj * sizeof(int), cudaMemcpyDeviceToHost, stream));
    DCG_CUDA(cudaStreamSynchronize(stream));
    return std::vector<int>(herr, herr + nj);
}

// ---- merging the reductions of several contexts (the serving loop's slots)
// A context with merge_reductions set hands its batched reduction to a per-device batcher
// instead of launching it.  The first waiting thread that finds the batcher idle becomes the
// leader: it takes, in arrival order, the submissions whose jobs fit one launch together, makes
// a batcher stream wait for each submission's ready event, launches them as one cooperative
// kernel (each job its own block group and words) and hands every submission its result.
// Requests that run concurrently then overlap their exchange-bound column loops inside one kernel
// instead of queueing on the cooperative-launch lock.  The block-group sizes change with the
// company, the arithmetic of a job does not: its partial sums do not depend on the number of
// blocks reducing it, so a matrix gets the same bits alone and merged.
struct CoopSub {
    Context *c = nullptr;
    std::vector<TrdJob> jobs;
    cudaEvent_t ready = nullptr;
    int state = 0;   // 0 waiting, 1 reduced, 2 does not fit a launch, 3 a wait timed out, 4 CUDA error
    std::string msg;
};

struct CoopBatcher {
    std::mutex mu;
    std::condition_variable cv;
    std::deque<CoopSub *> pending;
    bool busy = false;
    cudaStream_t stream = nullptr;
    int64_t launches = 0, joint = 0, carried = 0;
};

static std::mutex g_batchers_mu;
static std::map<int, CoopBatcher *> g_batchers;   // per device, for the life of the process

static CoopBatcher &coop_batcher(int device) {
    std::lock_guard<std::mutex> lk(g_batchers_mu);
    CoopBatcher *&b = g_batchers[device];
    if (!b) {
        b = new CoopBatcher;
        DCG_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    }
    return *b;
}

// One joint launch of the taken submissions (leader thread, leader context's workspace).
static void coop_run(Context &leader, CoopBatcher &B, std::vector<CoopSub *> &take) {
    std::vector<TrdJob> all;
    for (CoopSub *s : take) all.insert(all.end(), s->jobs.begin(), s->jobs.end());
    try {
        std::lock_guard<std::mutex> coop(g_coop_mutex);
        int total = 0;
        size_t smem = 0;
        if (!trd_plan(leader, all, total, smem)) throw Error{DCG_E_CUDA, "merged reduction does not fit"};
        for (CoopSub *s : take) DCG_CUDA(cudaStreamWaitEvent(B.stream, s->ready, 0));
        const std::vector<int> he = trd_launch(leader, all, total, smem, B.stream, "trd.err.joint");
        size_t q = 0;
        for (CoopSub *s : take) {
            bool err = false;
            for (size_t k = 0; k < s->jobs.size(); k++, q++) err = err || he[q] != 0;
            s->state = err ? 3 : 1;
            s->c->launches++;
        }
        B.launches++;
        if (take.size() > 1) B.joint++;
        B.carried += (int64_t)take.size();
    } catch (const Error &e) {
        for (CoopSub *s : take) {
            s->state = 4;
            s->msg = e.msg;
        }
    }
}

static bool tridiag_smem_merged(Context &c, std::vector<TrdJob> &jobs) {
    {   // a submission that cannot run even alone goes the unbatched way
        std::vector<TrdJob> alone = jobs;
        int total = 0;
        size_t smem = 0;
        if (!trd_plan(c, alone, total, smem)) return false;
    }
    for (TrdJob &j : jobs) j.nb = 0;   // not planned yet: any block count
    trd_clear(c, jobs);
    CoopSub me;
    me.c = &c;
    me.jobs = jobs;
    DCG_CUDA(cudaEventCreateWithFlags(&me.ready, cudaEventDisableTiming));
    const cudaError_t er = cudaEventRecord(me.ready, c.stream);
    if (er != cudaSuccess) {
        cudaEventDestroy(me.ready);
        throw Error{DCG_E_CUDA, std::string("cudaEventRecord: ") + cudaGetErrorString(er)};
    }
    CoopBatcher &B = coop_batcher(c.device);
    // merge window: a leader that finds no other submission waits this long for one
    // (DCG_MERGE_WINDOW_US, default 0: launch at once)
    const char *wenv = getenv("DCG_MERGE_WINDOW_US");
    const long window_us = wenv ? std::max(0L, std::min(5000000L, atol(wenv))) : 0L;
    {
        std::unique_lock<std::mutex> lk(B.mu);
        B.pending.push_back(&me);
        B.cv.notify_all();
        while (me.state == 0) {
            if (B.busy) {
                B.cv.wait(lk);
                continue;
            }
            B.busy = true;
            if (window_us > 0 && B.pending.size() < 2)
                B.cv.wait_for(lk, std::chrono::microseconds(window_us), [&] { return B.pending.size() >= 2; });
            std::vector<CoopSub *> take;
            std::vector<TrdJob> trial;
            while (!B.pending.empty()) {
                CoopSub *s = B.pending.front();
                std::vector<TrdJob> t2 = trial;
                t2.insert(t2.end(), s->jobs.begin(), s->jobs.end());
                int total = 0;
                size_t smem = 0;
                bool fits = false;
                try {
                    fits = trd_plan(c, t2, total, smem);
                } catch (const Error &) {
                    fits = false;
                }
                if (!fits && !take.empty()) break;   // the rest waits for the next launch
                B.pending.pop_front();
                if (!fits) {                            // cannot run merged at all
                    s->state = 2;
                    continue;
                }
                take.push_back(s);
                trial.swap(t2);
            }
            lk.unlock();
            if (!take.empty()) coop_run(c, B, take);
            lk.lock();
            B.busy = false;
            B.cv.notify_all();
        }
    }
    cudaEventDestroy(me.ready);
    if (me.state == 2) return false;
    if (me.state == 3) throw Error{DCG_E_NUMERIC, "tridiagonalisation: a wait for another block's words timed out"};
    if (me.state == 4) throw Error{DCG_E_CUDA, "merged tridiagonalisation: " + me.msg};
    return true;
}

// Cluster form (an option, orders up to kTridiagClusterMaxN): the same kernel with one cluster of
// ncta blocks per matrix instead of a cooperative launch: a cluster's blocks are resident
// together by definition, so nothing is serialised against other contexts, and a matrix reduces
// on the same few SMs whatever its company.
constexpr int kTridiagClusterMaxN = 400;

// Blocks per cluster for an order-n matrix (a function of n alone): more blocks share the FP64
// work of larger matrices, fewer keep the exchange short for small ones.
static int trd_cluster_ctas(int n) {
    if (n <= 32) return 1;
    if (n <= 64) return 4;
    return 16;   // a GB300 SM retires 1.66 FP64 FMAs per clock: the column work needs the blocks
}

// Jobs of one cluster shape.  False when no cluster of this shape can be resident (the caller then
// uses the cooperative form).
static bool tridiag_cluster_group(Context &c, std::vector<TrdJob> &jobs, int ncta) {
    size_t smem = 0;
    for (size_t q = 0; q < jobs.size(); q++) {
        smem = std::max(smem, trd_bytes_for(jobs[q].n, ncta));
        jobs[q].nb = ncta;
        jobs[q].b0 = ncta * (int)q;
    }
    const size_t limit = trd_smem_limit(c);
    if (smem > limit || jobs.size() > (size_t)kTrdMaxJobs) return false;
    // the same values from every context and thread (serving slots launch concurrently), so
    // no launch can see another's smaller limit
    DCG_CUDA(cudaFuncSetAttribute(tridiag_smem_batched_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit));
    DCG_CUDA(cudaFuncSetAttribute(tridiag_smem_batched_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ncta;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    const int total = ncta * (int)jobs.size();
    cfg.gridDim = dim3((unsigned)total);
    cfg.blockDim = dim3(TRS_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int resident = 0;
    if (cudaOccupancyMaxActiveClusters(&resident, (const void *)tridiag_smem_batched_kernel, &cfg) != cudaSuccess ||
        resident < 1) {
        cudaGetLastError();
        return false;
    }
    trd_clear(c, jobs);
    const std::vector<int> he = trd_launch(c, jobs, total, smem, c.stream, "trd.err.cluster", ncta);
    c.launches++;
    for (int e : he)
        if (e) throw Error{DCG_E_NUMERIC, "tridiagonalisation: a wait for another block's words timed out"};
    return true;
}

// Whether the cluster form takes the matrices it fits (DCG_TRD_CLUSTER=1).  Off by default: a
// 16-block cluster carries several times the per-block FP64 work of a column of the
// cooperative form's larger block groups.
static bool trd_cluster_enabled() {
    static const bool on = [] {
        const char *e = getenv("DCG_TRD_CLUSTER");
        return e && e[0] == '1';
    }();
    return on;
}

static bool tridiag_smem_batched(Context &c, std::vector<TrdJob> &jobs) {
    if (c.merge_reductions) return tridiag_smem_merged(c, jobs);
    std::lock_guard<std::mutex> coop(g_coop_mutex);
    int total = 0;
    size_t smem = 0;
    if (!trd_plan(c, jobs, total, smem)) return false;
    trd_clear(c, jobs);
    const std::vector<int> he = trd_launch(c, jobs, total, smem, c.stream, "trd.err");
    c.launches++;
    for (int e : he)
        if (e) throw Error{DCG_E_NUMERIC, "tridiagonalisation: a wait for another block's words timed out"};
    return true;
}

// One matrix on columns in global memory (tridiag_global_kernel); false when v, x and u do not fit
// a block's shared memory (n above about 4800).
static bool tridiag_global(Context &c, int n, cplx *A, int64_t lda, HeevWork &h) {
    const int nb = std::min(std::max(1, c.num_sms), n);
    const size_t smem = 3 * sizeof(cplx) * (size_t)n + ((size_t)(n + nb - 1) / nb) * 8 * sizeof(double);
    if (smem > trd_smem_limit(c)) return false;
    std::lock_guard<std::mutex> coop(g_coop_mutex);
    DCG_CUDA(cudaFuncSetAttribute(tridiag_global_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)trd_smem_limit(c)));
    int per_sm = 0;
    DCG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tridiag_global_kernel, TRS_THREADS, smem));
    if (per_sm < 1) return false;
    TrdJob j{};
    j.A = A;
    j.lda = lda;
    j.d = h.d;
    j.e = h.e;
    j.tau = h.tau;
    j.ll = wsget<ulonglong2>(c, "trd.ll.global", trd_ll_words(n));
    j.limit_ns = trd_wait_limit(c);
    j.n = n;
    j.nb = nb;
    j.real = c.real_now;
    std::vector<TrdJob> jobs(1, j);
    trd_clear(c, jobs);
    const std::vector<int> he = trd_launch(c, jobs, nb, smem, c.stream, "trd.err.global", 0, true);
    c.launches++;
    if (he[0]) throw Error{DCG_E_NUMERIC, "tridiagonalisation: a wait for another block's words timed out"};
    return true;
}

// One matrix: columns in global memory, the L2-resident persistent kernel, or one kernel launch per
// column beyond it.
static void tridiag_single(Context &c, int n, cplx *A, int64_t lda, HeevWork &h) {
    if (tridiag_global(c, n, A, lda, h)) return;
    if (n <= kTridiagPersistentMaxN) {
        tridiag_persistent(c, n, A, lda, h);
        return;
    }
    for (int k = 0; k + 1 < n; k++) {
        const int m = n - k - 1;
        hh_gen_kernel<<<1, 256, 0, c.stream>>>(n, k, A, lda, h.d, h.e, h.tau);
        DCG_LAUNCHED(c);
        const int nchunk = (m + HH_CHUNK - 1) / HH_CHUNK;
        dim3 g1(grid1d(m, 128), nchunk);
        hh_matvec_kernel<<<g1, 128, 0, c.stream>>>(n, k, A, lda, h.tau, h.ppart);
        DCG_LAUNCHED(c);
        hh_w_kernel<<<1, 512, 0, c.stream>>>(n, k, A, lda, h.tau, h.ppart, nchunk, h.w);
        DCG_LAUNCHED(c);
        dim3 g2(grid1d(m, 128), m);
        hh_update_kernel<<<g2, 128, 0, c.stream>>>(n, k, A, lda, h.w);
        DCG_LAUNCHED(c);
    }
    hh_last_kernel<<<1, 1, 0, c.stream>>>(n, A, lda, h.d);
    DCG_LAUNCHED(c);
}

static void check_dc_status(Context &c, int slot) {
    if (!c.eig_status[slot]) return;
    int st = 0;
    DCG_CUDA(cudaMemcpyAsync(&st, c.eig_status[slot], sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    DCG_CUDA(cudaStreamSynchronize(c.stream));
    if (st) throw Error{DCG_E_NUMERIC, "divide-and-conquer merge met coincident undeflated poles"};
}

// Eigenvalues of every job's matrix (ascending, into job.w); the reflectors stay in job.A and
// the tridiagonal eigenvectors in the job's slot for heev_vectors_slot.  Jobs that fit the
// shared-memory tridiagonalisation are reduced together in one launch.
void heev_values_batched(Context &c, const std::vector<EigJob> &jobs) {
    if (jobs.empty()) return;
    double work = 0.0;
    for (const EigJob &j : jobs) {
        if (j.slot < 0 || j.slot >= kEigSlots) throw Error{DCG_E_ARG, "eigensolver slot out of range"};
        work += (16.0 / 3.0) * (double)j.n * j.n * j.n;
    }
    std::vector<HeevWork> hw;
    for (const EigJob &j : jobs) hw.push_back(heev_work(c, std::max(j.n, 1), j.slot));
    FamScope fs(c, DCG_FAM_EIG, work);
    {
        FamScope f1(c, DCG_FAM_EIG_TRI, work);
        std::vector<TrdJob> tj;
        std::vector<size_t> who;
        for (size_t q = 0; q < jobs.size(); q++) {
            const EigJob &j = jobs[q];
            if (j.n <= 0 || j.n > kTridiagSmemMaxN) continue;
            TrdJob t;
            t.A = j.A;
            t.lda = j.lda;
            t.d = hw[q].d;
            t.e = hw[q].e;
            t.tau = hw[q].tau;
            t.ll = wsget<ulonglong2>(c, slot_name("trd.ll", j.slot), trd_ll_words(j.n));
            t.limit_ns = trd_wait_limit(c);
            t.n = j.n;
            t.real = c.real_now;
            t.b0 = t.nb = 0;
            tj.push_back(t);
            who.push_back(q);
        }
        std::vector<bool> done(jobs.size(), false);
        if (!tj.empty() && trd_cluster_enabled()) {   // small matrices: one cluster each
            std::map<int, std::vector<size_t>> groups;   // blocks per cluster -> indices into tj
            for (size_t k = 0; k < tj.size(); k++)
                if (tj[k].n <= kTridiagClusterMaxN) groups[trd_cluster_ctas(tj[k].n)].push_back(k);
            std::vector<bool> taken(tj.size(), false);
            for (auto &g : groups) {
                std::vector<TrdJob> gj;
                for (size_t k : g.second) gj.push_back(tj[k]);
                if (!tridiag_cluster_group(c, gj, g.first)) continue;
                for (size_t k : g.second) {
                    taken[k] = true;
                    done[who[k]] = true;
                }
            }
            std::vector<TrdJob> rest;
            std::vector<size_t> rwho;
            for (size_t k = 0; k < tj.size(); k++)
                if (!taken[k]) {
                    rest.push_back(tj[k]);
                    rwho.push_back(who[k]);
                }
            tj.swap(rest);
            who.swap(rwho);
        }
        if (!tj.empty()) {
            if (tridiag_smem_batched(c, tj)) {
                for (size_t q : who) done[q] = true;
            } else if (tj.size() > 1) {   // too many for one launch: each on its own
                for (size_t k = 0; k < tj.size(); k++) {
                    std::vector<TrdJob> one(1, tj[k]);
                    if (tridiag_smem_batched(c, one)) done[who[k]] = true;
                }
            }
        }
        for (size_t q = 0; q < jobs.size(); q++)
            if (!done[q] && jobs[q].n > 0) tridiag_single(c, jobs[q].n, jobs[q].A, jobs[q].lda, hw[q]);
    }
    {
        FamScope f2(c, DCG_FAM_EIG_VAL, work / 4.0);
        std::vector<size_t> dq;   // largest first, so the long chains start first
        for (size_t q = 0; q < jobs.size(); q++)
            if (jobs[q].n > 0 && !jobs[q].tridiag_only) dq.push_back(q);
        std::stable_sort(dq.begin(), dq.end(), [&](size_t x, size_t y) { return jobs[x].n > jobs[y].n; });
        on_aux_streams(c, (int)dq.size(), [&](int k) {
            const size_t q = dq[k];
            tridiag_dc(c, jobs[q].n, hw[q].d, hw[q].e, jobs[q].w, jobs[q].slot);
        });
    }
    for (const EigJob &j : jobs)
        if (j.n > 0 && !j.tridiag_only) check_dc_status(c, j.slot);
}

// y <- Q^H y for the columns of Y0 (written to Y), Q = H_0 H_1 ... H_{n-2} the reflectors of a
// tridiagonal reduction (H_k = I - tau_k v_k v_k^H, v_k in column k of A below the diagonal):
// H_0^H first.  One warp per column, the column in registers (R = ceil(n / 32)).
template <int R, int WPC, bool REAL>
__global__ void __launch_bounds__(64) apply_qh_kernel(int n, const cplx *__restrict__ A, int64_t lda,
                                                     const cplx *__restrict__ tau, const cplx *__restrict__ Y0,
                                                     int64_t ldy0, int ncol, cplx *Y, int64_t ldy) {
    __shared__ double part[2][2][2];   // [buffer][warp][re, im]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wsub = warp % WPC;                              // warp within its column
    const int col = blockIdx.x * (2 / WPC) + warp / WPC;      // 64 threads: 2 / WPC columns
    const bool have = col < ncol;
    if (WPC == 1 && !have) return;   // whole warp; with two warps per column both stay for the barriers
    cplx z[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int r = lane + 32 * (WPC * i + wsub);
        z[i] = (have && r < n) ? Y0[r + (int64_t)col * ldy0] : mk(0.0, 0.0);
    }
    int applied = 0;   // reflectors that were not skipped
    for (int k = 0; k + 1 < n; k++) {
        const cplx t = __ldg(tau + k);
        if (t.x == 0.0 && t.y == 0.0) continue;   // uniform over the block
        const int i0 = (k + 1) / (32 * WPC);      // row chunks below k+1 hold v = 0 in every lane
        const cplx *vk = A + (int64_t)k * lda;
        double sr = 0.0, si = 0.0;
#pragma unroll
        for (int i = 0; i < R; i++) {
            if (i < i0) continue;
            const int r = lane + 32 * (WPC * i + wsub);
            const cplx vv = (have && r > k && r < n) ? __ldg(vk + r) : mk(0.0, 0.0);
            sr = fma(vv.x, z[i].x, REAL ? sr : fma(vv.y, z[i].y, sr));    // conj(v) z
            if (!REAL) si = fma(vv.x, z[i].y, fma(-vv.y, z[i].x, si));
        }
        double fr, fi;   // f = conj(tau) (v^H z)
        bt_scale<WPC, REAL>(sr, si, mk(t.x, -t.y), wsub, part[applied++ & 1], fr, fi);
#pragma unroll
        for (int i = 0; i < R; i++) {
            if (i < i0) continue;
            const int r = lane + 32 * (WPC * i + wsub);
            const cplx vv = (have && r > k && r < n) ? __ldg(vk + r) : mk(0.0, 0.0);
            z[i].x = fma(-vv.x, fr, REAL ? z[i].x : fma(vv.y, fi, z[i].x));   // z -= v f
            if (!REAL) z[i].y = fma(-vv.x, fi, fma(-vv.y, fr, z[i].y));
        }
    }
    if (!have) return;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int r = lane + 32 * (WPC * i + wsub);
        if (r < n) Y[r + (int64_t)col * ldy] = z[i];
    }
}

// Per outer index o (one thread): solve (T + alpha_o) z = y_o by Gaussian elimination with
// partial pivoting on the tridiagonal (Golub & Van Loan, Matrix Computations, 4th ed., 4.3:
// row interchanges add one superdiagonal of fill-in), then e2o = -Re y^H z, sco = |z|^2.
// T: diagonal d (n), off-diagonal e (n-1), real.  The eliminated rows go to per-thread scratch
// laid out [row * nouter + o] (coalesced across threads), the pivots as reciprocals.  A serial
// chain a thread: one reciprocal a row instead of a division in each of two branches that both
// run, none in the back substitution, rows read ahead (20/12/300, two of 792 rows: 0.91 -> 0.55 ms each).
__global__ void tridiag_solve_e2_kernel(int n, const double *__restrict__ d, const double *__restrict__ e,
                                        const cplx *__restrict__ Y, int64_t ldy, int nouter,
                                        const double *__restrict__ alpha, double *D, double *U, double *U2, cplx *B,
                                        double *e2o, double *sco) {
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= nouter) return;
    const double al = alpha[o];
    const cplx *y = Y + (int64_t)o * ldy;
#define IX(k) ((int64_t)(k) * nouter + o)
    double dcur = d[0] + al, ucur = n > 1 ? e[0] : 0.0;
    cplx bcur = y[0], bnext = n > 1 ? y[1] : mk(0.0, 0.0);
    double dnext = n > 1 ? d[1] : 0.0, dl = n > 1 ? e[0] : 0.0;
    for (int i = 0; i + 1 < n; i++) {
        const double dn = dnext + al, un = i + 2 < n ? e[i + 1] : 0.0;
        const cplx bn = bnext;
        if (i + 2 < n) {   // the next row, while this one is eliminated
            dnext = d[i + 2];
            bnext = y[i + 2];
        }
        // the pivot row p and the other, q: rows i + 1 and i exchanged when i + 1 has the larger
        // entry (on the bits; no branch, the lanes differ)
        const bool ex = __double_as_longlong(fabs(dcur)) < __double_as_longlong(fabs(dl));
        const double pd = ex ? dl : dcur, qd = ex ? dcur : dl;
        const double pu = ex ? dn : ucur, qu = ex ? ucur : dn;
        const double pu2 = ex ? un : 0.0, qu2 = ex ? 0.0 : un;
        const cplx pb = ex ? bn : bcur, qb = ex ? bcur : bn;
        const double r = safe_rcp(pd), f = qd * r;
        D[IX(i)] = r;
        U[IX(i)] = pu;
        U2[IX(i)] = pu2;
        B[IX(i)] = pb;
        dcur = fma(-f, pu, qu);
        ucur = fma(-f, pu2, qu2);
        bcur = mk(fma(-f, pb.x, qb.x), fma(-f, pb.y, qb.y));
        dl = un;
    }
    // back substitution, with the two sums; the rows are read one ahead
    const double rn = safe_rcp(dcur);
    cplx z1 = mk(bcur.x * rn, bcur.y * rn), z2 = mk(0.0, 0.0), yi = y[n - 1];
    double er = fma(yi.x, z1.x, yi.y * z1.y), s = fma(z1.x, z1.x, z1.y * z1.y);
    double ri = 0.0, ui = 0.0, u2i = 0.0;
    cplx bi = mk(0.0, 0.0);
    if (n > 1) {
        const int64_t x = IX(n - 2);
        ri = D[x], ui = U[x], u2i = U2[x], bi = B[x], yi = y[n - 2];
    }
    for (int i = n - 2; i >= 0; i--) {
        const double r0 = ri, u0 = ui, v0 = u2i;
        const cplx b0 = bi, y0 = yi;
        if (i > 0) {
            const int64_t x = IX(i - 1);
            ri = D[x], ui = U[x], u2i = U2[x], bi = B[x], yi = y[i - 1];
        }
        const cplx zi = mk(fma(-u0, z1.x, fma(-v0, z2.x, b0.x)) * r0, fma(-u0, z1.y, fma(-v0, z2.y, b0.y)) * r0);
        er = fma(y0.x, zi.x, fma(y0.y, zi.y, er));
        s = fma(zi.x, zi.x, fma(zi.y, zi.y, s));
        z2 = z1;
        z1 = zi;
    }
#undef IX
    e2o[o] = -er;
    sco[o] = s;
}

void tridiag_e2(Context &c, int slot, int n, const cplx *A, int64_t lda, const cplx *VC, int64_t ldvc, int nouter,
                const double *alpha, double *e2o, double *sco) {
    if (n <= 0 || nouter <= 0) return;
    if (n > kTridiagE2MaxN) throw Error{DCG_E_ARG, "tridiag_e2: dimension above the register limit"};
    HeevWork h = heev_work(c, n, slot);
    cplx *Y = wsget<cplx>(c, slot_name("te2.Y", slot), (size_t)n * nouter);
    FamScope fs(c, DCG_FAM_EIG, 8.0 * (double)n * n * nouter);
    // one warp per vector up to 256 rows; above, two warps per vector (twice the warps to hide
    // the per-reflector reduction latency) and the register chunks sized to the rows
#define DCG_QH(r, w, g)                                                                                              \
    {                                                                                                                \
        auto *kern = c.real_now ? apply_qh_kernel<r, w, true> : apply_qh_kernel<r, w, false>;                        \
        kern<<<(g), 64, 0, c.stream>>>(n, A, lda, h.tau, VC, ldvc, nouter, Y, n);                                    \
    }
    if (n <= 256) DCG_QH(8, 1, grid1d(nouter, 2))
    else if (n <= 512) DCG_QH(8, 2, (unsigned)nouter)
    else if (n <= 768) DCG_QH(12, 2, (unsigned)nouter)
    else if (n <= 896) DCG_QH(14, 2, (unsigned)nouter)
    else DCG_QH(16, 2, (unsigned)nouter)
#undef DCG_QH
    DCG_LAUNCHED(c);
    const size_t sz = (size_t)n * nouter;
    double *D = wsget<double>(c, slot_name("te2.D", slot), sz);
    double *U = wsget<double>(c, slot_name("te2.U", slot), sz);
    double *U2 = wsget<double>(c, slot_name("te2.U2", slot), sz);
    cplx *B = wsget<cplx>(c, slot_name("te2.B", slot), sz);
    // one thread per outer index, its tridiagonal solve a serial FP64 chain: blocks of one warp
    // spread the indices over as many SMs as there are warps
    tridiag_solve_e2_kernel<<<grid1d(nouter, 32), 32, 0, c.stream>>>(n, h.d, h.e, Y, n, nouter, alpha, D, U, U2, B,
                                                                      e2o, sco);
    DCG_LAUNCHED(c);
}

// Eigenvectors [vlo, vhi) of the matrix reduced in slot `slot` by heev_values_batched (its
// reflectors still in A, its tridiagonal eigenvectors in the slot).
void heev_vectors_slot(Context &c, int slot, int n, cplx *A, int64_t lda, int vlo, int vhi, cplx *Z, int64_t ldz) {
    const int nvec = vhi - vlo;
    if (nvec <= 0 || n <= 0 || Z == nullptr) return;
    if (slot < 0 || slot >= kEigSlots || (c.eig_Q[slot] == nullptr && c.eig_last[slot] == 0) || c.eig_n[slot] != n)
        throw Error{DCG_E_STATE, "eigenvectors requested without a matching eigenvalue stage"};
    HeevWork h = heev_work(c, n, slot);
    FamScope fs(c, DCG_FAM_EIG, 8.0 * (double)n * n * nvec);
    const double *Qt = dc_vectors(c, slot, n, vlo, vhi);
    FamScope f4(c, DCG_FAM_EIG_BACK, 8.0 * (double)n * n * nvec);
    // Many columns: the FP64 pipe is the limit, one warp per column without prefetch (fewest
    // registers).  Few columns: the n-1 sequential reflections are the limit, prefetch the next
    // reflector (two warps per column above 512 rows to keep it in registers).
    if (n <= 1024) {
        const bool many = nvec >= 64;
        if (n <= 256) {
            if (many) launch_bt_reg<8, 1, false>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
            else launch_bt_reg<8, 1, true>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
        } else if (n <= 512) {
            if (many) launch_bt_reg<8, 2, false>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
            else launch_bt_reg<16, 1, true>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
        } else {
            // many columns: two warps per column, register chunks sized to the rows (a 792-row
            // column in 14 chunks instead of 32 one-warp chunks of which 7 are empty)
            if (many) {
                if (n <= 768) launch_bt_reg<12, 2, false>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
                else if (n <= 896) launch_bt_reg<14, 2, false>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
                else launch_bt_reg<16, 2, false>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
            } else {
                launch_bt_reg<16, 2, true>(c, n, A, lda, h.tau, Qt, vlo, nvec, Z, ldz);
            }
        }
        return;
    }
    z_from_real_kernel<<<grid1d((int64_t)n * nvec, 256), 256, 0, c.stream>>>(n, Qt, vlo, nvec, Z, ldz);
    DCG_LAUNCHED(c);
    const cplx one = mk(1.0, 0.0), zero = mk(0.0, 0.0), mone = mk(-1.0, 0.0);
    const int nref = n - 1;
    const int npanel = (nref + WY_NB - 1) / WY_NB;
    cplx *Vall = wsget<cplx>(c, "wy.V", (size_t)wy_offset(n, npanel - 1) + (size_t)(n - (npanel - 1) * WY_NB) * WY_NB);
    cplx *G = wsget<cplx>(c, "wy.G", (size_t)npanel * WY_NB * WY_NB);
    cplx *T = wsget<cplx>(c, "wy.T", (size_t)npanel * WY_NB * WY_NB);
    cplx *W1 = wsget<cplx>(c, "wy.W1", (size_t)WY_NB * nvec);
    cplx *W2 = wsget<cplx>(c, "wy.W2", (size_t)WY_NB * nvec);
    DCG_CUDA(cudaFuncSetAttribute(wy_tfactor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  2 * WY_NB * WY_NB * (int)sizeof(cplx)));
    wy_extract_kernel<<<dim3(grid1d((int64_t)nref * WY_NB, 256), npanel), 256, 0, c.stream>>>(n, A, lda, Vall);
    DCG_LAUNCHED(c);
    for (int p = 0; p < npanel; p++) {
        const int nbp = std::min(WY_NB, nref - p * WY_NB), m0 = nref - p * WY_NB;
        const cplx *Vp = Vall + wy_offset(n, p);
        zgemm(c, OP_C, OP_N, nbp, nbp, m0, one, Vp, m0, 0, Vp, m0, 0, zero, G + (int64_t)p * WY_NB * WY_NB, nbp, 0, 1);
    }
    wy_tfactor_kernel<<<npanel, WY_NB, 2 * WY_NB * WY_NB * sizeof(cplx), c.stream>>>(n, G, h.tau, T);
    DCG_LAUNCHED(c);
    for (int p = npanel - 1; p >= 0; p--) {
        const int k0 = p * WY_NB;
        const int nbp = std::min(WY_NB, nref - k0);
        const int m0 = n - k0 - 1;
        const cplx *Vp = Vall + wy_offset(n, p), *Tp = T + (int64_t)p * WY_NB * WY_NB;
        cplx *Zs = Z + (k0 + 1);
        zgemm(c, OP_C, OP_N, nbp, nvec, m0, one, Vp, m0, 0, Zs, ldz, 0, zero, W1, nbp, 0, 1);
        zgemm(c, OP_N, OP_N, nbp, nvec, nbp, one, Tp, WY_NB, 0, W1, nbp, 0, zero, W2, nbp, 0, 1);
        zgemm(c, OP_N, OP_N, m0, nvec, nbp, mone, Vp, m0, 0, W2, nbp, 0, one, Zs, ldz, 0, 1);
    }
}

void eig_slot_jobs(Context &c, const std::vector<VecJob> &vj, const std::vector<TE2Job> &tj) {
    struct Item {
        const VecJob *v;
        const TE2Job *t;
        double work;
    };
    std::vector<Item> items;
    double wv = 0.0, wt = 0.0;
    for (const VecJob &v : vj) {
        if (v.n <= 0 || v.vhi <= v.vlo || v.Z == nullptr) continue;
        if (v.n > 1024) {
            heev_vectors_slot(c, v.slot, v.n, v.A, v.lda, v.vlo, v.vhi, v.Z, v.ldz);
            continue;
        }
        const double w = 8.0 * (double)v.n * v.n * (v.vhi - v.vlo);
        items.push_back({&v, nullptr, w});
        wv += w;
    }
    for (const TE2Job &t : tj) {
        if (t.n <= 0 || t.nouter <= 0) continue;
        const double w = 8.0 * (double)t.n * t.n * t.nouter;
        items.push_back({nullptr, &t, w});
        wt += w;
    }
    if (items.empty()) return;
    std::stable_sort(items.begin(), items.end(), [](const Item &x, const Item &y) { return x.work > y.work; });
    FamScope fs(c, DCG_FAM_EIG, wv + wt);
    FamScope fb(c, DCG_FAM_EIG_BACK, wv);
    const int fam = c.fam;
    c.fam = 0;   // the two scopes above time the overlapped group once, on the context stream
    try {
        on_aux_streams(c, (int)items.size(), [&](int k) {
            const Item &it = items[k];
            if (it.v) heev_vectors_slot(c, it.v->slot, it.v->n, it.v->A, it.v->lda, it.v->vlo, it.v->vhi, it.v->Z, it.v->ldz);
            else tridiag_e2(c, it.t->slot, it.t->n, it.t->A, it.t->lda, it.t->VC, it.t->ldvc, it.t->nouter, it.t->alpha,
                            it.t->e2o, it.t->sco);
        });
    } catch (...) {
        c.fam = fam;
        throw;
    }
    c.fam = fam;
}

void heev(Context &c, int n, cplx *A, int64_t lda, double *w, int vlo, int vhi, cplx *Z, int64_t ldz) {
    if (n <= 0) return;
    EigJob j;
    j.n = n;
    j.A = A;
    j.lda = lda;
    j.w = w;
    j.slot = 0;
    heev_values_batched(c, std::vector<EigJob>(1, j));
    heev_vectors_slot(c, 0, n, A, lda, vlo, vhi, Z, ldz);
}

// Eigenvectors [vlo, vhi) of the matrix most recently passed to heev() (slot 0).
void heev_vectors_only(Context &c, int n, cplx *A, int64_t lda, const double *w, int vlo, int vhi, cplx *Z,
                       int64_t ldz) {
    (void)w;
    heev_vectors_slot(c, 0, n, A, lda, vlo, vhi, Z, ldz);
}

// Symmetric tridiagonal eigendecomposition (the divide-and-conquer stage alone): d (n),
// e (n-1) device arrays; ascending eigenvalues into w (device) and eigenvectors returned
// (device, n x n, ld n; valid until the next eigensolver call).
const double *stedc(Context &c, int n, const double *d, const double *e, double *w) {
    if (n <= 0) return nullptr;
    tridiag_dc(c, n, d, e, w, 0);
    check_dc_status(c, 0);
    return dc_vectors(c, 0, n, 0, n);
}

}  // namespace dcg

namespace dcg {
// Joint-launch counters of the merged reductions on a device: launches, launches that carried
// more than one context's submission, and submissions carried.
void coop_merge_stats(int device, int64_t out[3]) {
    out[0] = out[1] = out[2] = 0;
    std::lock_guard<std::mutex> lk(g_batchers_mu);
    auto it = g_batchers.find(device);
    if (it == g_batchers.end()) return;
    std::lock_guard<std::mutex> lb(it->second->mu);
    out[0] = it->second->launches;
    out[1] = it->second->joint;
    out[2] = it->second->carried;
}
}  // namespace dcg
