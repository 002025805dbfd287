// Dense FP64 complex linear algebra on the device: workspace, GEMM, Hermitian fill,
// deterministic sums and the LU solve (Golub & Van Loan, Matrix Computations, 4th ed.,
// 3.4: partial pivoting).  The Hermitian eigensolver lives in dcg_eig.cu.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "dcg_common.cuh"

namespace dcg {

// ===================================================================== workspace
void *Workspace::get(const std::string &name, size_t bytes) {
    Buf &b = bufs_[name];
    if (b.bytes >= bytes && b.p) return b.p;
    if (b.p) {
        cudaFree(b.p);
        total_ -= b.bytes;
        b.p = nullptr;
        b.bytes = 0;
    }
    size_t alloc = bytes < 256 ? 256 : bytes;
    cudaError_t e = cudaMalloc(&b.p, alloc);
    if (e != cudaSuccess) {
        b.p = nullptr;
        cudaGetLastError();
        throw Error{DCG_E_NOMEM, "device allocation of " + std::to_string(alloc) + " bytes for " + name +
                                     " failed: " + cudaGetErrorString(e)};
    }
    b.bytes = alloc;
    total_ += alloc;
    return b.p;
}

void *Workspace::host(const std::string &name, size_t bytes) {
    Buf &b = host_[name];
    if (b.bytes >= bytes && b.p) return b.p;
    if (b.p) {
        cudaFreeHost(b.p);
        b.p = nullptr;
        b.bytes = 0;
    }
    const size_t alloc = bytes < 256 ? 256 : bytes;
    const cudaError_t e = cudaHostAlloc(&b.p, alloc, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        b.p = nullptr;
        cudaGetLastError();
        throw Error{DCG_E_NOMEM, "page-locked allocation for " + name + " failed: " + cudaGetErrorString(e)};
    }
    b.bytes = alloc;
    return b.p;
}

void Workspace::release_all() {
    for (auto &kv : bufs_)
        if (kv.second.p) cudaFree(kv.second.p);
    bufs_.clear();
    for (auto &kv : host_)
        if (kv.second.p) cudaFreeHost(kv.second.p);
    host_.clear();
    total_ = 0;
}

// ===================================================================== block reductions
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic block sum (fixed reduction tree); result valid in every thread.
__device__ double block_sum(double v, double *sh) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    int nw = (blockDim.x + 31) >> 5;
    double t = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
    if (wid == 0) t = warp_sum(t);
    if (threadIdx.x == 0) sh[0] = t;
    __syncthreads();
    double r = sh[0];
    __syncthreads();
    return r;
}

// ===================================================================== ZGEMM
// 256 threads as TYN x (256 / TYN), each owning a 4 x 4 block of outputs spaced TYN rows and
// 256/TYN columns apart: tiles of 64 x 64 (TYN 16), 32 x 128 (TYN 8) or 128 x 32 (TYN 32).
// A GB300 SM retires 1.66 FP64 FMAs per clock, so the useful fraction of a tile is the
// fraction of the GPU's FP64 rate a skinny product gets: the autotuner picks the tile.
constexpr int kZgTiles = 3;
// Rows and columns of all tile shapes: these three, then the fine-grained ones (zgemm_fine_kernel).
constexpr int kZgShapes = 7;
constexpr int kZgBm[kZgShapes] = {64, 32, 128, 32, 16, 8, 8};
constexpr int kZgBn[kZgShapes] = {64, 128, 32, 32, 16, 8, 4};

template <int OPA, int OPB, int TYN>
__global__ void __launch_bounds__(256) zgemm_kernel(int m, int n, int k, cplx alpha, const cplx *__restrict__ A,
                                                    int64_t lda, int64_t sa, const cplx *__restrict__ B,
                                                    int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc,
                                                    int64_t sc, int zoff, int upper) {
    constexpr int TXN = 256 / TYN, BM = 4 * TYN, BN = 4 * TXN, BK = 16;
    __shared__ cplx As[BK][BM + 1];
    __shared__ cplx Bs[BK][BN + 1];
    const int64_t bz = (int64_t)blockIdx.z + zoff;
    A += bz * sa;
    B += bz * sb;
    C += bz * sc;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    if (upper && m0 >= n0 + BN) return;   // tile strictly below the diagonal (Hermitian product, upper half)
    const int tx = threadIdx.x % TXN, ty = threadIdx.x / TXN;
    cplx acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = mk(0.0, 0.0);
    for (int k0 = 0; k0 < k; k0 += BK) {
        for (int e = threadIdx.x; e < BM * BK; e += 256) {
            int i, kk;
            if (OPA == OP_N || OPA == OP_R) {
                i = e % BM;
                kk = e / BM;
            } else {
                kk = e % BK;
                i = e / BK;
            }
            int gi = m0 + i, gk = k0 + kk;
            cplx v = mk(0.0, 0.0);
            if (gi < m && gk < k) {
                v = (OPA == OP_N || OPA == OP_R) ? A[gi + (int64_t)gk * lda] : A[gk + (int64_t)gi * lda];
                if (OPA == OP_C || OPA == OP_R) v = cconj(v);
            }
            As[kk][i] = v;
        }
        for (int e = threadIdx.x; e < BN * BK; e += 256) {
            int j, kk;
            if (OPB == OP_N || OPB == OP_R) {
                kk = e % BK;
                j = e / BK;
            } else {
                j = e % BN;
                kk = e / BN;
            }
            int gj = n0 + j, gk = k0 + kk;
            cplx v = mk(0.0, 0.0);
            if (gj < n && gk < k) {
                v = (OPB == OP_N || OPB == OP_R) ? B[gk + (int64_t)gj * ldb] : B[gj + (int64_t)gk * ldb];
                if (OPB == OP_C || OPB == OP_R) v = cconj(v);
            }
            Bs[kk][j] = v;
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < BK; kk++) {
            cplx a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                a[q] = As[kk][ty + TYN * q];
                b[q] = Bs[kk][tx + TXN * q];
            }
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int q = 0; q < 4; q++) cfma(acc[p][q], a[p], b[q]);
        }
        __syncthreads();
    }
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int p = 0; p < 4; p++) {
        int gi = m0 + ty + TYN * p;
        if (gi >= m) continue;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int gj = n0 + tx + TXN * q;
            if (gj >= n) continue;
            cplx r = cmul(alpha, acc[p][q]);
            int64_t o = gi + (int64_t)gj * ldc;
            if (use_beta) r = cadd(r, cmul(beta, C[o]));
            C[o] = r;
        }
    }
}

// Element arithmetic of the products below: complex, or real when every imaginary part of the
// operands is zero (Context::real_now; one FMA a multiply-add instead of four).
template <bool REAL>
struct ZArith {
    using T = cplx;
    static __device__ __forceinline__ T get(cplx v) { return v; }
    static __device__ __forceinline__ T zero() { return mk(0.0, 0.0); }
    static __device__ __forceinline__ void mac(T &acc, T a, T b) { cfma(acc, a, b); }
    static __device__ __forceinline__ T add(T a, T b) { return cadd(a, b); }
    // alpha acc (+ beta c)
    static __device__ __forceinline__ void put(cplx *c, cplx alpha, T acc, cplx beta, bool use_beta) {
        cplx r = cmul(alpha, acc);
        if (use_beta) r = cadd(r, cmul(beta, *c));
        *c = r;
    }
};
template <>
struct ZArith<true> {
    using T = double;
    static __device__ __forceinline__ T get(cplx v) { return v.x; }
    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ void mac(T &acc, T a, T b) { acc = fma(a, b, acc); }
    static __device__ __forceinline__ T add(T a, T b) { return a + b; }
    static __device__ __forceinline__ void put(cplx *c, cplx alpha, T acc, cplx beta, bool use_beta) {
        double r = alpha.x * acc;
        if (use_beta) r = fma(beta.x, c->x, r);
        *c = mk(r, 0.0);
    }
};

// ---- fine-grained products.  A warp's FP64 instruction holds its quarter of a GB300 SM for 77
// clocks (measured with all four busy, 1.66 FMAs per clock and SM) and one complex multiply-add
// of 32 outputs for 308: shared-memory and L2 bandwidth are never the limit, padding is.  Here a warp
// owns 8 x 4 outputs (one per lane, QN of such pieces along n), pieces outside the matrix are
// skipped, and the chunks of K end at k, so a 14 x 14 x 14 product costs 16 x 16 x 14 instead of
// 64 x 64 x 16.  A block is 8 warps as RM x RN pieces x KG groups of K: small outputs use
// all four quarters of an SM on one piece by splitting K between warps (summed in a fixed
// order through shared memory).  The next chunk is loaded into registers while the current
// one is multiplied.  Pieces go to warps rotated by the block index, so a ragged edge does
// not idle the same quarter of every SM.
// Measured: the small products of a solve take under 10 us a launch where tiles of 64 x 64 and up
// took 70 to 274 us.
template <int RM, int RN, int KG, int QN>
struct ZfShape {
    static constexpr int BM = 8 * RM, BN = 4 * RN * QN, BK = KG > 1 ? 32 : 16;
    static constexpr int NA = (BM * BK + 255) / 256, NB = (BN * BK + 255) / 256;
    static_assert(RM * RN * KG == 8, "eight warps");
};

// element (i, kk) of op(X) stored with leading dimension ld, (row, col) = (i, kk) for N and R
__device__ __forceinline__ cplx zf_load(const cplx *__restrict__ X, int64_t ld, int i, int kk, int op, bool trans) {
    cplx v = trans ? X[kk + (int64_t)i * ld] : X[i + (int64_t)kk * ld];
    if (op == OP_C || op == OP_R) v.y = -v.y;
    return v;
}

template <int RM, int RN, int KG, int QN, bool REAL>
__global__ void __launch_bounds__(256) zgemm_fine_kernel(int m, int n, int k, int opa, int opb, cplx alpha,
                                                         const cplx *__restrict__ A, int64_t lda, int64_t sa,
                                                         const cplx *__restrict__ B, int64_t ldb, int64_t sb, cplx beta,
                                                         cplx *C, int64_t ldc, int64_t sc, int zoff, int upper) {
    using S = ZfShape<RM, RN, KG, QN>;
    using Z = ZArith<REAL>;
    using T = typename Z::T;
    constexpr int BM = S::BM, BN = S::BN, BK = S::BK, NA = S::NA, NB = S::NB;
    __shared__ T As[BK][BM + 1];
    __shared__ T Bs[BK][BN + 1];
    __shared__ T red[KG > 1 ? 8 * 32 * QN : 1];
    const int64_t bz = (int64_t)blockIdx.z + zoff;
    A += bz * sa;
    B += bz * sb;
    C += bz * sc;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    if (upper && m0 >= n0 + BN) return;   // tile strictly below the diagonal (Hermitian product, upper half)
    const int tid = threadIdx.x, lane = tid & 31;
    const int w = ((tid >> 5) + (KG > 1 ? 0 : (int)(blockIdx.x + blockIdx.y + blockIdx.z))) & 7;
    const int kg = w % KG, sub = w / KG, rm = sub % RM, rn = sub / RM;
    const int li = 8 * rm + (lane & 7), lj = 4 * rn + (lane >> 3);   // this lane's row and first column in the tile
    const bool ta = opa == OP_T || opa == OP_C, tb = opb == OP_T || opb == OP_C;   // A stored k x m; B stored n x k
    const bool rows = m0 + 8 * rm < m;
    int nq = 0;   // pieces of this warp inside the matrix (uniform over the warp)
#pragma unroll
    for (int q = 0; q < QN; q++)
        if (rows && n0 + 4 * (rn + RN * q) < n) nq = q + 1;
    T acc[QN];
#pragma unroll
    for (int q = 0; q < QN; q++) acc[q] = Z::zero();
    T pa[NA], pb[NB];
    // element e of a chunk: A by rows fastest (N, R) or k fastest (T, C), B the other way round
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < NA; u++) {
            const int e = tid + 256 * u;
            const int i = ta ? e / BK : e % BM, kk = ta ? e % BK : e / BM;
            pa[u] = (e < BM * BK && m0 + i < m && k0 + kk < k) ? Z::get(zf_load(A, lda, m0 + i, k0 + kk, opa, ta)) : Z::zero();
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int e = tid + 256 * u;
            const int j = tb ? e % BN : e / BK, kk = tb ? e / BN : e % BK;
            pb[u] = (e < BN * BK && n0 + j < n && k0 + kk < k) ? Z::get(zf_load(B, ldb, n0 + j, k0 + kk, opb, !tb)) : Z::zero();
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < k; k0 += BK) {
#pragma unroll
        for (int u = 0; u < NA; u++) {
            const int e = tid + 256 * u;
            if (e < BM * BK) As[ta ? e % BK : e / BM][ta ? e / BK : e % BM] = pa[u];
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int e = tid + 256 * u;
            if (e < BN * BK) Bs[tb ? e / BN : e % BK][tb ? e % BN : e / BK] = pb[u];
        }
        __syncthreads();
        if (k0 + BK < k) fetch(k0 + BK);
        const int kend = min(BK, k - k0);
        if (nq == QN) {
#pragma unroll 4
            for (int kk = kg; kk < kend; kk += KG) {
                const T a = As[kk][li];
#pragma unroll
                for (int q = 0; q < QN; q++) Z::mac(acc[q], a, Bs[kk][lj + 4 * RN * q]);
            }
        } else if (nq > 0) {
            for (int kk = kg; kk < kend; kk += KG) {
                const T a = As[kk][li];
#pragma unroll
                for (int q = 0; q < QN; q++)
                    if (q < nq) Z::mac(acc[q], a, Bs[kk][lj + 4 * RN * q]);
            }
        }
        __syncthreads();
    }
    if (KG > 1) {   // the K groups' sums, added in group order by group 0
#pragma unroll
        for (int q = 0; q < QN; q++) red[(w * QN + q) * 32 + lane] = acc[q];
        __syncthreads();
        if (kg != 0) return;
        for (int g = 1; g < KG; g++)
#pragma unroll
            for (int q = 0; q < QN; q++) acc[q] = Z::add(acc[q], red[((w + g) * QN + q) * 32 + lane]);
    }
    const int gi = m0 + li;
    if (gi >= m) return;
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int q = 0; q < QN; q++) {
        const int gj = n0 + lj + 4 * RN * q;
        if (gj < n) Z::put(C + gi + (int64_t)gj * ldc, alpha, acc[q], beta, use_beta);
    }
}

// ---- small-dimension GEMMs of the 4-index transformation.  When the contracted index
// and the small output index are at most SMALL_D (an active or inactive orbital dimension),
// the GEMM is memory-bound: the small matrix is staged in shared memory and the large
// operand is streamed once.  Each thread owns one row (right-small) or one column
// (left-small) and SMALL_G consecutive outputs of it.
constexpr int SMALL_D = 32, SMALL_G = 8;

// C(m x n) = alpha * A(m x k) * op(B)(k x n) + beta * C, op(B) = B or conj(B); k, n <= SMALL_D.
template <int OPB, bool REAL>
__global__ void __launch_bounds__(256) zgemm_rsmall_kernel(int m, int n, int k, cplx alpha, const cplx *__restrict__ A,
                                                           int64_t lda, int64_t sa, const cplx *__restrict__ B,
                                                           int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc,
                                                           int64_t sc, int z0) {
    using Z = ZArith<REAL>;
    using T = typename Z::T;
    __shared__ T Bs[SMALL_D][SMALL_D];
    const int z = z0 + blockIdx.z;
    A += (int64_t)z * sa;
    B += (int64_t)z * sb;
    C += (int64_t)z * sc;
    for (int x = threadIdx.x + blockDim.x * threadIdx.y; x < k * n; x += blockDim.x * blockDim.y) {
        const int kk = x % k, j = x / k;
        cplx v = B[kk + (int64_t)j * ldb];
        if (OPB == OP_R) v = cconj(v);
        Bs[kk][j] = Z::get(v);
    }
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int j0 = threadIdx.y * SMALL_G;
    if (i >= m || j0 >= n) return;
    T acc[SMALL_G];
#pragma unroll
    for (int q = 0; q < SMALL_G; q++) acc[q] = Z::zero();
    for (int kk = 0; kk < k; kk++) {
        const T a = Z::get(A[i + (int64_t)kk * lda]);
#pragma unroll
        for (int q = 0; q < SMALL_G; q++)
            if (j0 + q < n) Z::mac(acc[q], a, Bs[kk][j0 + q]);
    }
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int q = 0; q < SMALL_G; q++) {
        if (j0 + q >= n) break;
        Z::put(C + i + (int64_t)(j0 + q) * ldc, alpha, acc[q], beta, use_beta);
    }
}

// C(m x n) = alpha * A^H(m x k) * B(k x n) + beta * C with A (k x m); m, k <= SMALL_D.
template <bool REAL>
__global__ void __launch_bounds__(256) zgemm_lsmall_kernel(int m, int n, int k, cplx alpha, const cplx *__restrict__ A,
                                                           int64_t lda, int64_t sa, const cplx *__restrict__ B,
                                                           int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc,
                                                           int64_t sc, int z0) {
    using Z = ZArith<REAL>;
    using T = typename Z::T;
    __shared__ T As[SMALL_D][SMALL_D];   // As[kk][i] = conj(A(kk, i))
    const int z = z0 + blockIdx.z;
    A += (int64_t)z * sa;
    B += (int64_t)z * sb;
    C += (int64_t)z * sc;
    for (int x = threadIdx.x + blockDim.x * threadIdx.y; x < k * m; x += blockDim.x * blockDim.y) {
        const int kk = x % k, i = x / k;
        As[kk][i] = Z::get(cconj(A[kk + (int64_t)i * lda]));
    }
    __syncthreads();
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int i0 = threadIdx.y * SMALL_G;
    if (j >= n || i0 >= m) return;
    T acc[SMALL_G];
#pragma unroll
    for (int q = 0; q < SMALL_G; q++) acc[q] = Z::zero();
    for (int kk = 0; kk < k; kk++) {
        const T b = Z::get(B[kk + j * ldb]);
#pragma unroll
        for (int q = 0; q < SMALL_G; q++)
            if (i0 + q < m) Z::mac(acc[q], As[kk][i0 + q], b);
    }
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int q = 0; q < SMALL_G; q++) {
        if (i0 + q >= m) break;
        Z::put(C + (i0 + q) + j * ldc, alpha, acc[q], beta, use_beta);
    }
}

// Small-dimension dispatch; returns false when the shape is not one of the two forms.
static bool zgemm_small(Context &c, Op opa, Op opb, int m, int n, int k, cplx alpha, const cplx *A, int64_t lda,
                        int64_t sa, const cplx *B, int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc, int64_t sc,
                        int batch) {
    if (k < 1 || k > SMALL_D) return false;
    // a thread forms SMALL_G outputs: below about one warp per quarter SM the fine-grained
    // kernel, one output per thread, spreads the product further
    if ((double)m * n * batch < 32.0 * SMALL_G * 4.0 * std::max(1, c.num_sms)) return false;
    if (opa == OP_N && (opb == OP_N || opb == OP_R) && n <= SMALL_D && m >= 64) {
        const int gy = (n + SMALL_G - 1) / SMALL_G;
        const int bx = 256 / gy;   // gy <= 4, bx >= 64
        for (int z0 = 0; z0 < batch; z0 += 65535) {
            const int nz = std::min(65535, batch - z0);
            dim3 grid(grid1d(m, bx), 1, nz), block(bx, gy);
            auto *kern = c.real_now ? zgemm_rsmall_kernel<OP_N, true>
                         : opb == OP_N ? zgemm_rsmall_kernel<OP_N, false> : zgemm_rsmall_kernel<OP_R, false>;
            kern<<<grid, block, 0, c.stream>>>(m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, z0);
            DCG_LAUNCHED(c);
        }
        return true;
    }
    if (opa == OP_C && opb == OP_N && m <= SMALL_D && n >= 64) {
        const int gy = (m + SMALL_G - 1) / SMALL_G;
        const int bx = 256 / gy;
        for (int z0 = 0; z0 < batch; z0 += 65535) {
            const int nz = std::min(65535, batch - z0);
            dim3 grid(grid1d(n, bx), 1, nz), block(bx, gy);
            auto *kern = c.real_now ? zgemm_lsmall_kernel<true> : zgemm_lsmall_kernel<false>;
            kern<<<grid, block, 0, c.stream>>>(m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, z0);
            DCG_LAUNCHED(c);
        }
        return true;
    }
    return false;
}

template <int OPA, int OPB>
static void zgemm_launch(Context &c, int m, int n, int k, cplx alpha, const cplx *A, int64_t lda, int64_t sa,
                         const cplx *B, int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc, int64_t sc,
                         int batch, int upper, int tile) {
    const int bm = kZgBm[tile], bn = kZgBn[tile];
    // the fine-grained kernel reads its operands by (row, k) and (k, column); the grid's y extent
    // bounds the columns one launch covers
    const int ymax = 65535;
    if (!upper && grid1d(n, bn) > (unsigned)ymax) {
        const int64_t nc = (int64_t)ymax * bn;
        for (int64_t j0 = 0; j0 < n; j0 += nc) {
            const cplx *Bj = B + (OPB == OP_N || OPB == OP_R ? j0 * ldb : j0);
            zgemm_launch<OPA, OPB>(c, m, (int)std::min<int64_t>(nc, n - j0), k, alpha, A, lda, sa, Bj, ldb, sb, beta,
                                   C + j0 * ldc, ldc, sc, batch, upper, tile);
        }
        return;
    }
    for (int z0 = 0; z0 < batch; z0 += 65535) {
        int nz = batch - z0 < 65535 ? batch - z0 : 65535;
        dim3 grid(grid1d(m, bm), grid1d(n, bn), nz);
#define DCG_ZF(t, rm, rn, kg, qn)                                                                                  \
    if (tile == t) {                                                                                               \
        auto *kern = c.real_now ? zgemm_fine_kernel<rm, rn, kg, qn, true> : zgemm_fine_kernel<rm, rn, kg, qn, false>; \
        kern<<<grid, 256, 0, c.stream>>>(m, n, k, OPA, OPB, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, z0, upper); \
        DCG_LAUNCHED(c);                                                                                           \
        continue;                                                                                                  \
    }
        DCG_ZF(3, 4, 2, 1, 4) DCG_ZF(4, 2, 4, 1, 1) DCG_ZF(5, 1, 2, 4, 1) DCG_ZF(6, 1, 1, 8, 1)
#undef DCG_ZF
        if (tile == 1)
            zgemm_kernel<OPA, OPB, 8><<<grid, 256, 0, c.stream>>>(m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc,
                                                                  sc, z0, upper);
        else if (tile == 2)
            zgemm_kernel<OPA, OPB, 32><<<grid, 256, 0, c.stream>>>(m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C,
                                                                   ldc, sc, z0, upper);
        else
            zgemm_kernel<OPA, OPB, 16><<<grid, 256, 0, c.stream>>>(m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C,
                                                                   ldc, sc, z0, upper);
        DCG_LAUNCHED(c);
    }
}

// Output tiles of a tile shape (for a Hermitian product's upper half, those touching it).
static int64_t zg_tiles(int m, int n, int tile, int upper) {
    const int bm = kZgBm[tile], bn = kZgBn[tile];
    const int64_t tm = (m + bm - 1) / bm, tn = (n + bn - 1) / bn;
    if (!upper) return tm * tn;
    int64_t t = 0;
    for (int64_t j = 0; j < tn; j++) t += std::min<int64_t>(tm, ((j + 1) * bn + bm - 1) / bm);
    return t;
}

// C = alpha * sum_s P_s + beta * C over nsplit partial products (fixed summation order).
__global__ void splitk_reduce_kernel(int m, int n, int nsplit, const cplx *__restrict__ P, cplx alpha, cplx beta,
                                     cplx *C, int64_t ldc, int upper) {
    const int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t mn = (int64_t)m * n;
    if (idx >= mn) return;
    const int i = (int)(idx % m), j = (int)(idx / m);
    if (upper && i > j) return;
    cplx acc = mk(0.0, 0.0);
    for (int s = 0; s < nsplit; s++) acc = cadd(acc, P[s * mn + idx]);
    const int64_t o = i + (int64_t)j * ldc;
    cplx r = cmul(alpha, acc);
    if (beta.x != 0.0 || beta.y != 0.0) r = cadd(r, cmul(beta, C[o]));
    C[o] = r;
}

template <int OPA, int OPB>
static void zgemm_launch(Context &c, int m, int n, int k, cplx alpha, const cplx *A, int64_t lda, int64_t sa,
                         const cplx *B, int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc, int64_t sc,
                         int batch, int upper, int tile);
static int64_t zg_tiles(int m, int n, int tile, int upper);

// One split-K product with a given number of K chunks (>= 2): the chunks are computed as one
// batched GEMM into partial products, then reduced in a fixed order.
template <int OPA, int OPB>
static void zgemm_splitk_run(Context &c, int m, int n, int k, int nsplit, cplx alpha, const cplx *A, int64_t lda,
                             const cplx *B, int64_t ldb, cplx beta, cplx *C, int64_t ldc, int upper, int tile) {
    const int kc = (k + nsplit - 1) / nsplit;
    nsplit = (k + kc - 1) / kc;
    const int nfull = k / kc;             // chunks of exactly kc
    const int rem = k - nfull * kc;       // last, shorter chunk
    const int64_t mn = (int64_t)m * n;
    cplx *P = wsget<cplx>(c, "gemm.splitk", (size_t)mn * nsplit);
    const cplx one = mk(1.0, 0.0), zero = mk(0.0, 0.0);
    // K-chunk strides: A is m x k (OP_N/OP_R, chunk = columns) or k x m (OP_T/OP_C, chunk = rows)
    const int64_t sa = (OPA == OP_N || OPA == OP_R) ? (int64_t)kc * lda : kc;
    const int64_t sb = (OPB == OP_N || OPB == OP_R) ? kc : (int64_t)kc * ldb;
    zgemm_launch<OPA, OPB>(c, m, n, kc, one, A, lda, sa, B, ldb, sb, zero, P, m, mn, nfull, upper, tile);
    if (rem > 0)
        zgemm_launch<OPA, OPB>(c, m, n, rem, one, A + nfull * sa, lda, 0, B + nfull * sb, ldb, 0, zero, P + nfull * mn,
                               m, 0, 1, upper, tile);
    splitk_reduce_kernel<<<grid1d(mn, 256), 256, 0, c.stream>>>(m, n, nsplit, P, alpha, beta, C, ldc, upper);
    DCG_LAUNCHED(c);
}

// The tile shape and K split of one FP64 product.  zg_cost estimates a plan's time: the FP64
// operations of the fullest SM (padding included; 1.66 FMAs per clock and SM) plus the latency of
// a chunk of K per wave and of a launch.  A product whose tiles do not fill the GPU may be split
// along K into equal chunks of at least 32, computed as one batched GEMM into partial products
// and reduced in a fixed order.  The cheapest plan by the estimate is candidate 0, used for
// small products, while tuning is off and for calls that accumulate into C (beta != 0, which
// the timed trial runs would disturb); the autotuner times the plans within 1.3 of it.
constexpr double kTuneMinFp64Flops = 1.0e9;
constexpr int kZgMinChunk = 32;

struct ZgPlan {
    int tile, nsplit;
    double cost;   // estimated clocks
};

// Clocks of a plan on `sms` SMs.
static double zg_cost(int sms, bool real, int m, int n, int k, int upper, int batch, int tile, int nsplit) {
    const int bm = kZgBm[tile], bn = kZgBn[tile];
    const int kc = (k + nsplit - 1) / nsplit;
    const bool fine = tile >= kZgTiles;
    // multiply-adds of one tile: whole tiles and chunks of 16 for the coarse kernels, pieces of
    // 8 x 4 for the fine ones (their K groups share a tile, so a tile takes the same FP64 time)
    const double tm = (m + bm - 1) / bm, tn = (n + bn - 1) / bn;
    const double fm = fine ? 8.0 * ((m + 7) / 8) / (bm * tm) : 1.0, fn = fine ? 4.0 * ((n + 3) / 4) / (bn * tn) : 1.0;
    const double kp = fine ? kc : 16.0 * ((kc + 15) / 16);
    const double work = bm * bn * fm * fn * kp * (real ? 1.0 : 4.0) / 1.66;   // clocks of one tile alone on an SM
    const double blocks = (double)zg_tiles(m, n, tile, upper) * nsplit * batch;
    const double waves = std::ceil(blocks / sms);
    // a tile alone on its SM waits for its loads once per chunk (the fine kernels prefetch)
    const double bk = tile >= 5 ? 32.0 : 16.0;
    const double lat = (waves <= 1.5 ? (fine ? 500.0 : 1500.0) : 100.0) * std::ceil(kc / bk);
    double t = waves * work * (fine ? 1.04 : 1.0) + lat + 4000.0;
    if (nsplit > 1) t += 6000.0 + (double)m * n * nsplit * 2.0 * 32.0 / (sms * 64.0);   // the reduction
    return t;
}

static std::vector<ZgPlan> zg_candidates(Context &c, int m, int n, int k, int upper, int batch) {
    const int sms = std::max(1, c.num_sms);
    std::vector<ZgPlan> all, out;
    for (int t = c.real_now ? kZgTiles : 0; t < kZgShapes; t++) {   // the coarse kernels are complex only
        const int64_t tiles = zg_tiles(m, n, t, upper);
        all.push_back({t, 1, zg_cost(sms, c.real_now, m, n, k, upper, batch, t, 1)});
        if (batch != 1 || tiles >= 2 * sms) continue;
        for (int p = 2; p <= k / kZgMinChunk && p <= 64; p *= 2)
            all.push_back({t, p, zg_cost(sms, c.real_now, m, n, k, upper, batch, t, p)});
    }
    std::stable_sort(all.begin(), all.end(), [](const ZgPlan &x, const ZgPlan &y) { return x.cost < y.cost; });
    for (const ZgPlan &p : all)
        if (out.empty() || (p.cost <= 1.3 * all[0].cost && out.size() < 8)) out.push_back(p);
    return out;
}

// What a list of plans holds, for the autotuner's stored choices (FNV-1a; never 0).
static unsigned zg_list_id(const std::vector<ZgPlan> &cand) {
    unsigned h = 2166136261u;
    for (const ZgPlan &p : cand)
        for (int v : {kZgBm[p.tile], kZgBn[p.tile], p.nsplit}) h = (h ^ (unsigned)v) * 16777619u;
    return h ? h : 1u;
}

template <int OPA, int OPB>
static void zgemm_plan_run(Context &c, const ZgPlan &p, int m, int n, int k, cplx alpha, const cplx *A, int64_t lda,
                           int64_t sa, const cplx *B, int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc,
                           int64_t sc, int batch, int upper) {
    if (p.nsplit >= 2) zgemm_splitk_run<OPA, OPB>(c, m, n, k, p.nsplit, alpha, A, lda, B, ldb, beta, C, ldc, upper, p.tile);
    else zgemm_launch<OPA, OPB>(c, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, batch, upper, p.tile);
}

template <int OPA, int OPB>
static void zgemm_tuned(Context &c, int m, int n, int k, cplx alpha, const cplx *A, int64_t lda, int64_t sa,
                        const cplx *B, int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc, int64_t sc, int batch,
                        int upper) {
    const std::vector<ZgPlan> cand = zg_candidates(c, m, n, k, upper, batch);
    const TuneKey key{TUNE_ZGEMM, OPA * 8 + OPB + (c.real_now ? 64 : 0), m, n, k, upper + 2 * std::min(batch, 1 << 20)};
    // products under ~1 ms of FP64 work keep the heuristic: their trials would cost more than
    // tuning can return (and a served stream meets many shapes once)
    const double work = (c.real_now ? 2.0 : 8.0) * m * n * (double)k * batch;
    const bool trial_ok = beta.x == 0.0 && beta.y == 0.0 && work >= kTuneMinFp64Flops;
    const int pick = autotune(c, key, (int)cand.size(), zg_list_id(cand), trial_ok, [&](int q) {
        zgemm_plan_run<OPA, OPB>(c, cand[q], m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, batch, upper);
    });
    zgemm_plan_run<OPA, OPB>(c, cand[pick], m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, batch, upper);
}

void zgemm(Context &c, Op opa, Op opb, int m, int n, int k, cplx alpha, const cplx *A, int64_t lda, int64_t sa,
           const cplx *B, int64_t ldb, int64_t sb, cplx beta, cplx *C, int64_t ldc, int64_t sc, int batch) {
    if (m <= 0 || n <= 0 || batch <= 0) return;
    GemmTrace trace(c, "fp64", m, n, k, batch);
    if (zgemm_small(c, opa, opb, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, batch)) return;
#define DCG_ZG(a, b)                                                                                  \
    if (opa == a && opb == b) {                                                                       \
        zgemm_tuned<a, b>(c, m, n, k, alpha, A, lda, sa, B, ldb, sb, beta, C, ldc, sc, batch, 0);     \
        return;                                                                                       \
    }
    DCG_ZG(OP_N, OP_N) DCG_ZG(OP_N, OP_T) DCG_ZG(OP_N, OP_C) DCG_ZG(OP_N, OP_R)
    DCG_ZG(OP_T, OP_N) DCG_ZG(OP_T, OP_T) DCG_ZG(OP_T, OP_C) DCG_ZG(OP_T, OP_R)
    DCG_ZG(OP_C, OP_N) DCG_ZG(OP_C, OP_T) DCG_ZG(OP_C, OP_C) DCG_ZG(OP_C, OP_R)
    DCG_ZG(OP_R, OP_N) DCG_ZG(OP_R, OP_T) DCG_ZG(OP_R, OP_C) DCG_ZG(OP_R, OP_R)
#undef DCG_ZG
    throw Error{DCG_E_ARG, "zgemm: bad op"};
}

// Upper triangle of C = A A^H (n x n, A n x k, column-major): only the 64 x 64 tiles on or
// above the diagonal are computed (half the work of the full product), split along k when
// those tiles alone cannot fill the GPU.  The strictly lower part of C is left undefined; a
// Hermitian fill from the upper triangle completes it.
void zherk_upper(Context &c, int n, int k, const cplx *A, int64_t lda, cplx *C, int64_t ldc) {
    if (n <= 0) return;
    GemmTrace trace(c, "herk", n, n, k, 1);
    const cplx one = mk(1.0, 0.0), zero = mk(0.0, 0.0);
    zgemm_tuned<OP_N, OP_C>(c, n, n, k, one, A, lda, 0, A, lda, 0, zero, C, ldc, 0, 1, 1);
}

// ===================================================================== Hermitian fill
__global__ void herm_from_upper_kernel(int n, cplx *A, int64_t lda) {
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)n * n) return;
    int i = (int)(idx % n), j = (int)(idx / n);
    if (i > j) A[i + (int64_t)j * lda] = cconj(A[j + (int64_t)i * lda]);
    else if (i == j) A[i + (int64_t)j * lda].y = 0.0;
}

void herm_from_upper(Context &c, int n, cplx *A, int64_t lda) {
    if (n <= 0) return;
    herm_from_upper_kernel<<<grid1d((int64_t)n * n, 256), 256, 0, c.stream>>>(n, A, lda);
    DCG_LAUNCHED(c);
}

// ===================================================================== deterministic sum
__global__ void dsum_kernel(const double *x, int64_t n, double *out) {
    __shared__ double sh[32];
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += x[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) *out = s;
}

// Partial sums of contiguous chunks of x (chunk elements each), one block per chunk.
__global__ void dsum_part_kernel(const double *x, int64_t n, int64_t chunk, double *part) {
    __shared__ double sh[32];
    const int64_t lo = (int64_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
    double s = 0.0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) s += x[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// Sum of x[0..n) into *out.  Long vectors (the per-outer-index E2 terms of F, G and H run to
// millions) are summed in fixed chunks by many blocks, then the chunk sums in order: the order
// depends on n only, so the result is deterministic.
void dsum(Context &c, const double *x, int64_t n, double *out) {
    constexpr int64_t kChunk = 8192;
    if (n <= 4 * kChunk) {
        dsum_kernel<<<1, 1024, 0, c.stream>>>(x, n, out);
        DCG_LAUNCHED(c);
        return;
    }
    const int64_t nb = (n + kChunk - 1) / kChunk;
    double *part = wsget<double>(c, "dsum.part", (size_t)nb);
    dsum_part_kernel<<<(unsigned)nb, 256, 0, c.stream>>>(x, n, kChunk, part);
    DCG_LAUNCHED(c);
    dsum_kernel<<<1, 1024, 0, c.stream>>>(part, nb, out);
    DCG_LAUNCHED(c);
}

void fam_collect(Context &c) {
    for (auto &pr : c.fam_ev) {
        cudaEventSynchronize(pr.second);
        float ms = 0.f;
        cudaEventElapsedTime(&ms, pr.first, pr.second);
        c.fam_ms += ms;
        cudaEventDestroy(pr.first);
        cudaEventDestroy(pr.second);
    }
    c.fam_ev.clear();
}

// ===================================================================== LU solve
__global__ void lu_pivot_kernel(int n, int k, cplx *A, int64_t lda, int ncols, int *info) {
    __shared__ double best[1024];
    __shared__ int bidx[1024];
    double b = -1.0;
    int bi = k;
    for (int i = k + threadIdx.x; i < n; i += blockDim.x) {
        double a = cabs2(A[i + (int64_t)k * lda]);
        if (a > b) {
            b = a;
            bi = i;
        }
    }
    best[threadIdx.x] = b;
    bidx[threadIdx.x] = bi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            double o = best[threadIdx.x + s];
            int oi = bidx[threadIdx.x + s];
            if (o > best[threadIdx.x] || (o == best[threadIdx.x] && oi < bidx[threadIdx.x])) {
                best[threadIdx.x] = o;
                bidx[threadIdx.x] = oi;
            }
        }
        __syncthreads();
    }
    const int p = bidx[0];
    if (best[0] == 0.0) {
        if (threadIdx.x == 0 && *info == 0) *info = k + 1;
        return;
    }
    if (p != k)
        for (int j = threadIdx.x; j < ncols; j += blockDim.x) {
            cplx t = A[k + (int64_t)j * lda];
            A[k + (int64_t)j * lda] = A[p + (int64_t)j * lda];
            A[p + (int64_t)j * lda] = t;
        }
    __syncthreads();
    cplx inv = cdiv(mk(1.0, 0.0), A[k + (int64_t)k * lda]);
    for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) A[i + (int64_t)k * lda] = cmul(A[i + (int64_t)k * lda], inv);
}

__global__ void lu_update_kernel(int n, int k, cplx *A, int64_t lda, int ncols) {
    const int i = k + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = k + 1 + blockIdx.y;
    if (i >= n || j >= ncols) return;
    A[i + (int64_t)j * lda] = csub(A[i + (int64_t)j * lda], cmul(A[i + (int64_t)k * lda], A[k + (int64_t)j * lda]));
}

// back substitution U x = y, y in column n of the augmented matrix
__global__ void lu_backsub_kernel(int n, cplx *A, int64_t lda) {
    cplx *b = A + (int64_t)n * lda;
    for (int k = n - 1; k >= 0; k--) {
        __syncthreads();
        cplx xk = cdiv(b[k], A[k + (int64_t)k * lda]);
        __syncthreads();
        if (threadIdx.x == 0) b[k] = xk;
        for (int i = threadIdx.x; i < k; i += blockDim.x) b[i] = csub(b[i], cmul(A[i + (int64_t)k * lda], xk));
    }
}

int zgesv(Context &c, int n, cplx *A, int64_t lda, cplx *b) {
    // augmented copy [A | b]
    cplx *M = wsget<cplx>(c, "gesv.M", (size_t)n * (n + 1));
    int *info = wsget<int>(c, "gesv.info", 1);
    DCG_CUDA(cudaMemcpy2DAsync(M, n * sizeof(cplx), A, lda * sizeof(cplx), n * sizeof(cplx), n,
                               cudaMemcpyDeviceToDevice, c.stream));
    DCG_CUDA(cudaMemcpyAsync(M + (int64_t)n * n, b, n * sizeof(cplx), cudaMemcpyDeviceToDevice, c.stream));
    DCG_CUDA(cudaMemsetAsync(info, 0, sizeof(int), c.stream));
    for (int k = 0; k < n; k++) {
        lu_pivot_kernel<<<1, 1024, 0, c.stream>>>(n, k, M, n, n + 1, info);
        DCG_LAUNCHED(c);
        if (k + 1 < n || true) {
            dim3 g(grid1d(n - k - 1 > 0 ? n - k - 1 : 1, 128), n - k);
            if (n - k - 1 > 0) {
                lu_update_kernel<<<g, 128, 0, c.stream>>>(n, k, M, n, n + 1);
                DCG_LAUNCHED(c);
            }
        }
    }
    lu_backsub_kernel<<<1, 1024, 0, c.stream>>>(n, M, n);
    DCG_LAUNCHED(c);
    DCG_CUDA(cudaMemcpyAsync(b, M + (int64_t)n * n, n * sizeof(cplx), cudaMemcpyDeviceToDevice, c.stream));
    int hinfo = 0;
    DCG_CUDA(cudaMemcpyAsync(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost, c.stream));
    DCG_CUDA(cudaStreamSynchronize(c.stream));
    return hinfo;
}

}  // namespace dcg
