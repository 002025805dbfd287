// Block Davidson eigensolver for the lowest roots of the CASCI Hamiltonian (Davidson,
// J. Comput. Phys. 17, 87 (1975); block form of Liu, 1978), the large-ndet CASCI route that
// replaces the dense ZHEEV of casci.F90:55-70 (diag.F90:66-128) when only a few roots are
// wanted.  The Hamiltonian stays in HBM as CSR (the diagonal and the single and double
// excitations of each determinant, dcg_ci.cu); every step is a device kernel:
//   W = H V                        (the sigma vectors, one warp per row of H)
//   G = V^H W                      (Rayleigh matrix, symmetrised)
//   G Y = Y diag(theta)            (one-block cyclic Jacobi, below)
//   R = W Y - V Y diag(theta)      (residuals of the block's Ritz pairs)
//   T = R / (theta - diag(H))      (diagonal preconditioner)
//   T orthonormalised against V    (classical Gram-Schmidt applied twice), appended to V.
// The host only orchestrates: per step it reads the residual norms and the lengths of the
// new directions back.  Converged when every wanted root has |r| <= tol.
#include <algorithm>
#include <cmath>
#include <functional>
#include <numeric>
#include <vector>

#include "dcg_common.cuh"
#include "dcg_kernels.cuh"

namespace dcg {

namespace {

constexpr int kJacobiMaxN = 64;
constexpr int kJacobiThreads = 256;
constexpr int kJacobiMaxSweeps = 40;

__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

__device__ double block_sum_d(double v, double *sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum_d(v);
    __syncthreads();
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    double t = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
    if (wid == 0) t = warp_sum_d(t);
    if (threadIdx.x == 0) sh[0] = t;
    __syncthreads();
    const double r = sh[0];
    __syncthreads();
    return r;
}

// Player at position `pos` of round `s` of a round-robin tournament of np players (np even):
// position 0 stays, the others rotate.  Round s pairs positions k and np-1-k.
__device__ __forceinline__ int rr_player(int pos, int s, int np) {
    return pos == 0 ? 0 : 1 + (pos - 1 + s) % (np - 1);
}

// Element arithmetic of a real or a complex Hermitian matrix (real: every imaginary part is zero).
template <bool REAL>
struct JT {
    using T = cplx;
    static __device__ __forceinline__ T get(cplx v) { return v; }
    static __device__ __forceinline__ cplx put(T v) { return v; }
    static __device__ __forceinline__ double abs2(T v) { return fma(v.x, v.x, v.y * v.y); }
    static __device__ __forceinline__ double re(T v) { return v.x; }
    static __device__ __forceinline__ T conj(T v) { return cconj(v); }
    static __device__ __forceinline__ T unit(double d) { return mk(d, 0.0); }
    static __device__ __forceinline__ T times(double f, T v) { return mk(f * v.x, f * v.y); }
    // c x - s y, c x + s y
    static __device__ __forceinline__ T minus(double c, T x, T s, T y) {
        return mk(fma(c, x.x, fma(-s.x, y.x, s.y * y.y)), fma(c, x.y, fma(-s.x, y.y, -s.y * y.x)));
    }
    static __device__ __forceinline__ T plus(double c, T x, T s, T y) {
        return mk(fma(c, x.x, fma(s.x, y.x, -s.y * y.y)), fma(c, x.y, fma(s.x, y.y, s.y * y.x)));
    }
};
template <>
struct JT<true> {
    using T = double;
    static __device__ __forceinline__ T get(cplx v) { return v.x; }
    static __device__ __forceinline__ cplx put(T v) { return mk(v, 0.0); }
    static __device__ __forceinline__ double abs2(T v) { return v * v; }
    static __device__ __forceinline__ double re(T v) { return v; }
    static __device__ __forceinline__ T conj(T v) { return v; }
    static __device__ __forceinline__ T unit(double d) { return d; }
    static __device__ __forceinline__ T times(double f, T v) { return f * v; }
    static __device__ __forceinline__ T minus(double c, T x, T s, T y) { return fma(c, x, -s * y); }
    static __device__ __forceinline__ T plus(double c, T x, T s, T y) { return fma(c, x, s * y); }
};

// All eigenpairs of a small Hermitian matrix G (n <= 64, column-major, ldg; the matrix used is
// (G + G^H)/2) by cyclic Jacobi with the parallel round-robin ordering (Golub & Van Loan,
// Matrix Computations, 4th ed., 8.5.5): each round rotates n/2 disjoint pairs at once,
// A <- J^H A J, V <- V J.  The 2x2 Hermitian block [[a, |b| e^{i phi}], [., d]] is made real
// by the phase e^{i phi} and rotated by the symmetric Schur step (ibid. 8.5.2), so
// J_pp = J_qq = c, J_pq = s e^{i phi}, J_qp = -s e^{-i phi}.  Sweeps stop when the squared
// off-diagonal Frobenius norm is below 1e-30 of the whole (status 1 after 40 sweeps).
// Output: ascending eigenvalues w[n], eigenvectors Y (n x n, ldy).  One block, bound by its SM's
// FP64 unit and the chain of a round's angles: the angle and phase come from FP32 arithmetic
// (a rotated element then shrinks by ~1e-7 instead of vanishing, within the quadratic
// convergence) and only c, s and the phase's length are made exact in FP64; a round's
// two-sided update touches each pair of pairs once (A is Hermitian), beside the update of V.
template <bool REAL>
__global__ void __launch_bounds__(kJacobiThreads) jacobi_heev_kernel(int n, const int *__restrict__ n_dev,
                                                                       const cplx *__restrict__ G, int ldg,
                                                                       double *w, cplx *Y, int ldy, int *status) {
    using Z = JT<REAL>;
    using T = typename Z::T;
    extern __shared__ double2 jsm[];
    if (n_dev) n = *n_dev;   // dimension read on the device (graph replays of a Davidson step)
    const int np = n + (n & 1);   // padded to even: the dummy player pairs with nobody
    T *A = reinterpret_cast<T *>(jsm);   // np x np
    T *V = A + np * np;                   // np x np
    __shared__ double cs_c[kJacobiMaxN / 2];
    __shared__ T cs_s[kJacobiMaxN / 2];   // s e^{i phi}
    __shared__ int cs_p[kJacobiMaxN / 2], cs_q[kJacobiMaxN / 2], cs_on[kJacobiMaxN / 2];
    __shared__ double red[32];
    __shared__ int rank_sh[kJacobiMaxN];
    const int tid = threadIdx.x, nt = blockDim.x;
    double fro = 0.0;
    for (int e = tid; e < np * np; e += nt) {
        const int i = e % np, j = e / np;
        cplx a = mk(0.0, 0.0);
        if (i < n && j < n) {
            const cplx x = G[i + (int64_t)ldg * j], y = G[j + (int64_t)ldg * i];
            a = mk(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
            if (i == j) a.y = 0.0;
        }
        A[e] = Z::get(a);
        V[e] = Z::unit(i == j ? 1.0 : 0.0);
        fro += Z::abs2(Z::get(a));
    }
    fro = block_sum_d(fro, red);   // syncs the block
    // a norm whose FP32 reciprocal could leave the range: the matrix is scaled by a power of two
    // (exact) and the eigenvalues back
    const int ex = (((__double2hiint(fro) >> 20) & 0x7FF) - 1023) / 2;
    const bool rescale = fro > 0.0 && (ex < -60 || ex > 60) && ex < 512;
    const double up = rescale ? __hiloint2double((1023 - ex) << 20, 0) : 1.0;
    const double down = rescale ? __hiloint2double((1023 + ex) << 20, 0) : 1.0;
    if (rescale) {
        for (int e = tid; e < np * np; e += nt) A[e] = Z::times(up, A[e]);
        fro = fro * up * up;
        __syncthreads();
    }
    const float scale = fro > 0.0 ? (float)(1.0 / sqrt(fro)) : 1.0f;   // elements of A in FP32 range
    const int npair = np / 2, nblk = npair * (npair + 1) / 2;
    int sweep = 0;
    for (; sweep < kJacobiMaxSweeps; sweep++) {
        double off = 0.0;
        for (int e = tid; e < np * np; e += nt)
            if (e % np < e / np) off += 2.0 * Z::abs2(A[e]);
        off = block_sum_d(off, red);
        if (off <= 1e-30 * fro || fro == 0.0) break;
        for (int s = 0; s < np - 1; s++) {
            // rotation parameters of each pair from the current A
            for (int k = tid; k < npair; k += nt) {
                int p = rr_player(k, s, np), q = rr_player(np - 1 - k, s, np);
                if (p > q) {
                    const int t = p;
                    p = q;
                    q = t;
                }
                cs_p[k] = p;
                cs_q[k] = q;
                // a rotation whose off-diagonal element is below 1e-34 of the squared norm is
                // skipped (all of them together stay under the 1e-30 stopping test): the late
                // sweeps of the quadratic convergence then cost little FP64 work
                const T b = A[p + np * q];
                const bool on = q < n && Z::abs2(b) > 1e-34 * fro;
                cs_on[k] = on;
                if (on) {
                    const cplx bc = Z::put(b);
                    const float bx = (float)bc.x * scale, by = REAL ? 0.0f : (float)bc.y * scale;
                    const float d = (float)(Z::re(A[q + np * q]) - Z::re(A[p + np * p])) * scale;
                    const float ab = REAL ? fabsf(bx) : sqrtf(fmaf(bx, bx, by * by));
                    const float h = 0.5f * fabsf(d);
                    const float t = copysignf(ab / (h + sqrtf(fmaf(h, h, ab * ab))), d);
                    const double t64 = (double)t, c = fast_rsqrt(fma(t64, t64, 1.0)), sn = t64 * c;
                    cs_c[k] = c;
                    if constexpr (REAL) {
                        cs_s[k] = b >= 0.0 ? sn : -sn;
                    } else {
                        const double px = (double)(bx / ab), py = (double)(by / ab);
                        const double f = sn * fast_rsqrt(fma(px, px, py * py));
                        cs_s[k] = mk(f * px, f * py);
                    }
                }
            }
            __syncthreads();
            // A <- J^H A J, each block of a pair k and a pair l >= k once, and V <- V J
            for (int e = tid; e < nblk + np * npair; e += nt) {
                if (e < nblk) {
                    int l = (int)((sqrtf(8.0f * e + 1.0f) - 1.0f) * 0.5f);
                    while (l * (l + 1) / 2 > e) l--;
                    while ((l + 1) * (l + 2) / 2 <= e) l++;
                    const int k = e - l * (l + 1) / 2;
                    if (!cs_on[k] && !cs_on[l]) continue;
                    const int pk = cs_p[k], qk = cs_q[k], pl = cs_p[l], ql = cs_q[l];
                    T b11 = A[pk + np * pl], b12 = A[pk + np * ql], b21 = A[qk + np * pl], b22 = A[qk + np * ql];
                    if (cs_on[l]) {   // columns: p' = c p - conj(s) q, q' = s p + c q
                        const double c = cs_c[l];
                        const T sg = cs_s[l], sc = Z::conj(sg);
                        T u = Z::minus(c, b11, sc, b12), v = Z::plus(c, b12, sg, b11);
                        b11 = u, b12 = v;
                        u = Z::minus(c, b21, sc, b22), v = Z::plus(c, b22, sg, b21);
                        b21 = u, b22 = v;
                    }
                    if (cs_on[k]) {   // rows: p' = c p - s q, q' = conj(s) p + c q
                        const double c = cs_c[k];
                        const T sg = cs_s[k], sc = Z::conj(sg);
                        T u = Z::minus(c, b11, sg, b21), v = Z::plus(c, b21, sc, b11);
                        b11 = u, b21 = v;
                        u = Z::minus(c, b12, sg, b22), v = Z::plus(c, b22, sc, b12);
                        b12 = u, b22 = v;
                    }
                    if (k == l) {   // Hermitian to the bit
                        b11 = Z::unit(Z::re(b11));
                        b22 = Z::unit(Z::re(b22));
                        A[pk + np * pk] = b11;
                        A[qk + np * qk] = b22;
                        A[pk + np * qk] = b12;
                        A[qk + np * pk] = Z::conj(b12);
                    } else {
                        A[pk + np * pl] = b11, A[pl + np * pk] = Z::conj(b11);
                        A[pk + np * ql] = b12, A[ql + np * pk] = Z::conj(b12);
                        A[qk + np * pl] = b21, A[pl + np * qk] = Z::conj(b21);
                        A[qk + np * ql] = b22, A[ql + np * qk] = Z::conj(b22);
                    }
                } else {
                    const int i = (e - nblk) % np, k = (e - nblk) / np;
                    if (!cs_on[k]) continue;
                    const int p = cs_p[k], q = cs_q[k];
                    const double c = cs_c[k];
                    const T sg = cs_s[k], vp = V[i + np * p], vq = V[i + np * q];
                    V[i + np * p] = Z::minus(c, vp, Z::conj(sg), vq);
                    V[i + np * q] = Z::plus(c, vq, sg, vp);
                }
            }
            __syncthreads();
        }
    }
    // ascending order (ties by index), then the outputs
    for (int i = tid; i < n; i += nt) {
        const double di = Z::re(A[i + np * i]);
        int r = 0;
        for (int j = 0; j < n; j++) {
            const double dj = Z::re(A[j + np * j]);
            r += (dj < di) || (dj == di && j < i);
        }
        rank_sh[i] = r;
    }
    __syncthreads();
    for (int i = tid; i < n; i += nt) w[rank_sh[i]] = down * Z::re(A[i + np * i]);
    for (int e = tid; e < n * n; e += nt) {
        const int i = e % n, j = e / n;
        Y[i + (int64_t)ldy * rank_sh[j]] = Z::put(V[i + np * j]);
    }
    if (tid == 0 && sweep >= kJacobiMaxSweeps) *status = 1;
}

// Columns c of X (n x m) set to the unit vectors e_{idx[c]}.
__global__ void unit_cols_kernel(int n, int m, const int *__restrict__ idx, cplx *X, int64_t ldx) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)n * m) return;
    const int i = (int)(e % n), c = (int)(e / n);
    X[i + ldx * c] = mk(i == idx[c] ? 1.0 : 0.0, 0.0);
}

// ---- vector work in chunks of kDavChunk rows, one block each: partial sums go to part[...] and
// whoever needs the sum adds the chunks in order, so a sum depends on n alone.  One block for a
// whole vector left 151 SMs idle on 74,273 determinants (0.2 to 1 ms a kernel).
constexpr int kDavChunk = 1024, kDavThreads = 256;
constexpr int kDavShortSteps = 250;   // steps with the short subspace before V may grow to the long one
constexpr int kAxpyRows = 128;   // rows (and threads) of a block that subtracts: its loop over the vectors is the long one

// Sum of n values by one warp in a fixed order (every lane gets it).
__device__ __forceinline__ double warp_total(const double *x, int n, int stride = 1) {
    double s = 0.0;
    for (int i = threadIdx.x & 31; i < n; i += 32) s += x[(int64_t)i * stride];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Sums of a complex (re, im) pair over the block; real vectors carry no im.
template <bool REAL>
__device__ __forceinline__ void dav_block_sum(double &re, double &im, double *sh) {
    re = block_sum_d(re, sh);
    if (!REAL) im = block_sum_d(im, sh);
}

// conj(x) y added to (re, im)
template <bool REAL>
__device__ __forceinline__ void dav_dot(double &re, double &im, cplx x, cplx y) {
    re = fma(x.x, y.x, re);
    if (!REAL) {
        re = fma(x.y, y.y, re);
        im = fma(x.x, y.y, im);
        im = fma(-x.y, y.x, im);
    }
}

// ---- the Davidson step with its sizes on the device ------------------------------------
// A step's launches read the subspace size m and the running counts from DavState, so one
// captured sequence (a CUDA graph) serves every step.
struct DavState {
    int m;        // vectors in V (and W = H V)
    int mold;     // of them, those whose Rayleigh elements G already holds
    int cand;     // new directions accepted in this step
    int jac;      // a Jacobi solve ran out of sweeps (sticky)
    int restarted;
    int live[8], ok[8];   // direction q: tried, accepted
    int cap;      // vectors that V may hold now (at most mmax)
    int pad[2];
    double worst;  // largest residual norm of the wanted roots
};
// Column of direction q: after the accepted ones before it.
__device__ __forceinline__ int dav_col(const DavState *st, int q) {
    int m = st->m;
    for (int p = 0; p < q; p++) m += st->ok[p];
    return m;
}

// Partial G[i, j] = V[:, i]^H W[:, j], i <= j, for the columns j >= mold that G does not hold yet:
// block (i, j - mold, chunk).
template <bool REAL>
__global__ void __launch_bounds__(kDavThreads) rr_part_kernel(int n, const cplx *__restrict__ V, const cplx *__restrict__ W,
                                                              int64_t ld, cplx *part, int mmax,
                                                              const DavState *__restrict__ st) {
    __shared__ double sh[32];
    const int i = blockIdx.x, j = st->mold + blockIdx.y, m = st->m;
    if (j >= m || i > j) return;
    const cplx *a = V + ld * i, *b = W + ld * j;
    double re = 0.0, im = 0.0;
    const int k0 = blockIdx.z * kDavChunk, k1 = min(n, k0 + kDavChunk);
    for (int k = k0 + threadIdx.x; k < k1; k += kDavThreads) dav_dot<REAL>(re, im, a[k], b[k]);
    dav_block_sum<REAL>(re, im, sh);
    if (threadIdx.x == 0) part[i + (int64_t)mmax * (blockIdx.y + 16 * (int64_t)blockIdx.z)] = mk(re, im);
}
template <bool REAL>
__global__ void rr_sum_kernel(int nchunk, const cplx *__restrict__ part, int mmax, cplx *G, int ldg,
                              const DavState *__restrict__ st) {
    const int j = st->mold + blockIdx.x, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (j >= st->m) return;
    for (int i = threadIdx.x >> 5; i <= j; i += nw) {   // a warp per element
        const double *x = reinterpret_cast<const double *>(part + i + (int64_t)mmax * blockIdx.x);
        const int stride = 2 * mmax * 16;
        const double re = warp_total(x, nchunk, stride), im = REAL || i == j ? 0.0 : warp_total(x + 1, nchunk, stride);
        if (lane == 0) {
            G[i + (int64_t)ldg * j] = mk(re, im);
            G[j + (int64_t)ldg * i] = mk(re, -im);
        }
    }
}

// X = V Y[:, :nb] (z = 0) and HX = W Y[:, :nb] (z = 1) over the m columns of V and W.
template <bool REAL>
__global__ void ritz_kernel(int n, const cplx *__restrict__ V, const cplx *__restrict__ W, int64_t ld,
                            const cplx *__restrict__ Y, int ldy, cplx *X, cplx *HX, const DavState *__restrict__ st) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (r >= n) return;
    const cplx *A = blockIdx.z ? W : V;
    const int m = st->m;
    cplx acc = mk(0.0, 0.0);
    for (int q = 0; q < m; q++) {
        const cplx a = A[r + ld * q], y = __ldg(Y + q + (int64_t)ldy * c);
        if (REAL) acc.x = fma(a.x, y.x, acc.x);
        else cfma(acc, a, y);
    }
    (blockIdx.z ? HX : X)[r + ld * c] = acc;
}

// R[:, c] = HX[:, c] - theta[c] X[:, c], its squared norm by chunks to part[chunk + nchunk c];
// T[:, c] = R[:, c] / (theta[c] - hd) with the denominator kept away from 0.
template <bool REAL>
__global__ void __launch_bounds__(kDavThreads) residual_kernel(int n, const cplx *__restrict__ HX,
                                                               const cplx *__restrict__ X, int64_t ld,
                                                               const double *__restrict__ theta,
                                                               const double *__restrict__ hd, cplx *T, double *part) {
    __shared__ double sh[32];
    const int c = blockIdx.y;
    const double th = theta[c];
    double acc = 0.0;
    const int k0 = blockIdx.x * kDavChunk, k1 = min(n, k0 + kDavChunk);
    for (int i = k0 + threadIdx.x; i < k1; i += kDavThreads) {
        const cplx hx = HX[i + ld * c], x = X[i + ld * c];
        const cplx r = mk(fma(-th, x.x, hx.x), REAL ? 0.0 : fma(-th, x.y, hx.y));
        acc = fma(r.x, r.x, acc);
        if (!REAL) acc = fma(r.y, r.y, acc);
        double den = th - hd[i];
        if (fabs(den) < 1e-4) den = den < 0.0 ? -1e-4 : 1e-4;
        const double inv = 1.0 / den;
        T[i + ld * c] = mk(r.x * inv, REAL ? 0.0 : r.y * inv);
    }
    acc = block_sum_d(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x + (int64_t)gridDim.x * c] = acc;
}

// The residual norms of the block's roots (to h2), the worst of the wanted ones; the step's
// direction flags reset, and the restart decided: the next block would not fit.
__global__ void step_begin_kernel(int nwant, int nb, int nchunk, const double *__restrict__ part, double *h2,
                                  DavState *st) {
    __shared__ double v[8];
    for (int q = threadIdx.x >> 5; q < nb; q += blockDim.x >> 5) {   // a warp per root
        const double s = warp_total(part + (int64_t)nchunk * q, nchunk);
        if ((threadIdx.x & 31) == 0) v[q] = h2[q] = s;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double w = 0.0;
    for (int q = 0; q < nwant; q++) w = fmax(w, sqrt(v[q]));
    st->worst = w;
    for (int q = 0; q < 8; q++) st->live[q] = st->ok[q] = 0;
    st->restarted = st->m + nb > st->cap;
}

// Restart on the block's Ritz vectors: V, W <- X, HX.
__global__ void restart_copy_kernel(int n, int nb, const cplx *__restrict__ X, const cplx *__restrict__ HX,
                                    cplx *V, cplx *W, int64_t ld, const DavState *__restrict__ st) {
    if (!st->restarted) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)n * nb) return;
    const int i = (int)(e % n), c = (int)(e / n);
    V[i + ld * c] = X[i + ld * c];
    W[i + ld * c] = HX[i + ld * c];
}

__global__ void restart_set_kernel(int nb, DavState *st) {
    if (threadIdx.x == 0 && st->restarted) st->m = nb;
}

// Direction q: live when its residual is above tol, no direction before it was rejected and V has
// room; then T[:, q] goes to its column of V and its squared norm, by chunks, to part.
template <bool REAL>
__global__ void __launch_bounds__(kDavThreads) cand_begin_kernel(int n, int q, double tol,
                                                                 const double *__restrict__ h2,
                                                                 const cplx *__restrict__ T, cplx *V, int64_t ld,
                                                                 double *part, DavState *st) {
    __shared__ double sh[32];
    bool live = sqrt(h2[q]) > tol;
    for (int p = 0; p < q; p++)
        if (st->live[p] && !st->ok[p]) live = false;
    const int col = dav_col(st, q);
    live = live && col < st->cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->live[q] = live;
    if (!live) return;
    cplx *dst = V + ld * col;
    double acc = 0.0;
    const int k0 = blockIdx.x * kDavChunk, k1 = min(n, k0 + kDavChunk);
    for (int i = k0 + threadIdx.x; i < k1; i += kDavThreads) {
        const cplx x = T[i + ld * q];
        dst[i] = x;
        acc = fma(x.x, x.x, acc);
        if (!REAL) acc = fma(x.y, x.y, acc);
    }
    acc = block_sum_d(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// Classical Gram-Schmidt pass of direction q against the vectors before it: the coefficients by
// chunks (block (i, chunk)), then the subtraction, which adds the chunks and leaves the squared
// norm of what remains by its own chunks in part2.
template <bool REAL>
__global__ void __launch_bounds__(kDavThreads) cgs_dot_kernel(int n, int q, const cplx *__restrict__ V, int64_t ld,
                                                              cplx *cf, int mmax, const DavState *__restrict__ st) {
    __shared__ double sh[32];
    if (!st->live[q]) return;
    const int i = blockIdx.x, mm = dav_col(st, q);
    if (i >= mm) return;
    const cplx *a = V + ld * i, *b = V + ld * mm;
    double re = 0.0, im = 0.0;
    const int k0 = blockIdx.y * kDavChunk, k1 = min(n, k0 + kDavChunk);
    for (int k = k0 + threadIdx.x; k < k1; k += kDavThreads) dav_dot<REAL>(re, im, a[k], b[k]);
    dav_block_sum<REAL>(re, im, sh);
    if (threadIdx.x == 0) cf[i + (int64_t)mmax * blockIdx.y] = mk(re, im);
}

template <bool REAL>
__global__ void __launch_bounds__(kAxpyRows) cgs_axpy_kernel(int n, int q, int nchunk, cplx *V, int64_t ld,
                                                             const cplx *__restrict__ cf, int mmax, double *part2,
                                                             const DavState *__restrict__ st) {
    __shared__ double sh[32];
    __shared__ cplx c[kJacobiMaxN];
    if (!st->live[q]) return;
    const int mm = dav_col(st, q);
    if (nchunk == 1) {
        for (int i = threadIdx.x; i < mm; i += kAxpyRows) c[i] = cf[i];
    } else {
        for (int i = threadIdx.x >> 5; i < mm; i += kAxpyRows / 32) {   // a warp per coefficient
            const double *x = reinterpret_cast<const double *>(cf + i);
            const double re = warp_total(x, nchunk, 2 * mmax), im = REAL ? 0.0 : warp_total(x + 1, nchunk, 2 * mmax);
            if ((threadIdx.x & 31) == 0) c[i] = mk(re, im);
        }
    }
    __syncthreads();
    cplx *dst = V + ld * mm;
    double acc = 0.0;
    const int r = blockIdx.x * kAxpyRows + threadIdx.x;
    if (r < n) {
        cplx s = mk(0.0, 0.0);
        for (int p = 0; p < mm; p++) {
            const cplx v = V[r + ld * p];
            if (REAL) s.x = fma(v.x, c[p].x, s.x);
            else cfma(s, v, c[p]);
        }
        const cplx d = csub(dst[r], s);
        dst[r] = d;
        acc = fma(d.x, d.x, acc);
        if (!REAL) acc = fma(d.y, d.y, acc);
    }
    acc = block_sum_d(acc, sh);
    if (threadIdx.x == 0) part2[blockIdx.x] = acc;
}

// Accept direction q when it kept more than 1e-10 of its length (normalised, counted), else no
// direction after it is tried.
__global__ void __launch_bounds__(kDavThreads) cand_end_kernel(int n, int q, cplx *V, int64_t ld,
                                                               const double *__restrict__ part,
                                                               const double *__restrict__ part2, int npart2, DavState *st) {
    if (!st->live[q]) return;
    __shared__ double s_scale;
    __shared__ int s_ok;
    const int col = dav_col(st, q);
    if (threadIdx.x < 32) {
        const double n0 = warp_total(part, (int)gridDim.x), acc = warp_total(part2, npart2);
        if (threadIdx.x == 0) {
            s_ok = acc > 1e-20 * n0 && acc > 0.0;
            s_scale = s_ok ? 1.0 / sqrt(acc) : 0.0;
            if (blockIdx.x == 0) st->ok[q] = s_ok;   // read by later launches only
        }
    }
    __syncthreads();
    if (!s_ok) return;
    cplx *dst = V + ld * col;
    const double s = s_scale;
    const int k0 = blockIdx.x * kDavChunk, k1 = min(n, k0 + kDavChunk);
    for (int i = k0 + threadIdx.x; i < k1; i += kDavThreads) dst[i] = mk(dst[i].x * s, dst[i].y * s);
}

// Y[:, c] = H X[:, c] for K vectors and a CSR H (vals, or real rvals): one warp per row, the lanes
// striding the row's entries in order and a fixed shuffle tree summing them (deterministic).
// With st, X and Y are the cand accepted directions of V and W.  Bound by the FP64 unit (K FMAs
// an entry real, 4 K complex) and, real with few vectors, by the 12 bytes an entry.
template <int K, bool REAL>
__global__ void __launch_bounds__(256) csr_hx_kernel(int n, int k, const int64_t *__restrict__ rowptr,
                                                      const int *__restrict__ cols, const cplx *__restrict__ vals,
                                                      const double *__restrict__ rvals, const cplx *__restrict__ X,
                                                      cplx *Y, int64_t ld, const DavState *__restrict__ st) {
    const int row = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (st) {
        k = dav_col(st, 8) - st->m;
        X += ld * st->m;
        Y += ld * st->m;
    }
    if (row >= n || k == 0) return;
    double re[K], im[K];
#pragma unroll
    for (int c = 0; c < K; c++) re[c] = im[c] = 0.0;
    const int64_t e1 = rowptr[row + 1];
    for (int64_t e = rowptr[row] + lane; e < e1; e += 32) {
        const int j = __ldg(cols + e);
        if (REAL) {
            const double h = __ldg(rvals + e);
#pragma unroll
            for (int c = 0; c < K; c++)
                if (c < k) re[c] = fma(h, __ldg(&X[j + ld * c].x), re[c]);
        } else {
            const cplx h = __ldg(vals + e);
#pragma unroll
            for (int c = 0; c < K; c++) {
                if (c < k) {
                    const cplx x = __ldg(X + j + ld * c);
                    re[c] = fma(h.x, x.x, fma(-h.y, x.y, re[c]));
                    im[c] = fma(h.x, x.y, fma(h.y, x.x, im[c]));
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < K; c++) {
        if (c < k)
            for (int o = 16; o > 0; o >>= 1) {
                re[c] += __shfl_down_sync(0xffffffffu, re[c], o);
                if (!REAL) im[c] += __shfl_down_sync(0xffffffffu, im[c], o);
            }
    }
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < K; c++)
            if (c < k) Y[row + ld * c] = mk(re[c], im[c]);
    }
}

__global__ void step_end_kernel(DavState *st) {
    if (threadIdx.x != 0) return;
    const int cand = dav_col(st, 8) - st->m;
    st->cand = cand;
    st->mold = st->restarted ? 0 : st->m;
    st->m += cand;
}

}  // namespace

// Y (n x k) = H X for the CSR H, up to 8 vectors (st: the accepted directions of a step, at most kmax).
static void csr_hx(Context &c, const CsrMatrix &H, const cplx *X, cplx *Y, int64_t ld, int k, const DavState *st) {
    const int n = H.n;
    const int blocks = (int)(((int64_t)n * 32 + 255) / 256);
    const bool real = H.rvals != nullptr;
    auto *kern = k > 4 ? (real ? csr_hx_kernel<8, true> : csr_hx_kernel<8, false>)
                 : k > 2 ? (real ? csr_hx_kernel<4, true> : csr_hx_kernel<4, false>)
                         : (real ? csr_hx_kernel<2, true> : csr_hx_kernel<2, false>);
    kern<<<blocks, 256, 0, c.stream>>>(n, k, H.rowptr, H.cols, H.vals, H.rvals, X, Y, ld, st);
}

// Lowest nwant eigenpairs of the Hermitian CSR H (its diagonal kept beside it): eigenvalues to
// w[0..nwant), eigenvectors to the columns of Z (n x nwant, ldz = n), each with residual norm
// <= tol_rel * max(1, max_i |H_ii|).
//
// One step: the new elements of the Rayleigh matrix G = V^H W and its eigenpairs (Jacobi), the
// block's Ritz vectors X = V Y and images HX = W Y, their residuals and preconditioned
// corrections T, a restart V, W <- X, HX when the next block would not fit, then each
// unconverged correction orthonormalised against V (classical Gram-Schmidt twice) and
// appended, and W extended by H times the new directions.  Every size the step needs lives on
// the device (DavState), so the step is one fixed launch sequence: captured once as a CUDA
// graph and replayed, with one read of the state per step (the environment variable
// DCG_DAVIDSON_GRAPH=0 launches the sequence directly instead).
void davidson_lowest_csr(Context &c, const CsrMatrix &H, int nwant, double *w, cplx *Z, double tol_rel, int maxit) {
    const int n = H.n;
    const int nb = std::min(n, nwant + 2);   // block: the wanted roots and a margin for near-degeneracy
    // A long subspace saves iterations (each one product with H), a short one keeps the one-block
    // Jacobi short (its time grows with the cube): at 924 determinants and one root 12 vectors
    // took 16 steps and 4.9 ms where 24 took 14 and 6.8; at 74,273 determinants (0.9 ms a product)
    // the products decide.  Restarts every few steps can stall on nearly degenerate levels: of 240
    // runs (60 spectra of 252 to 8008 determinants, one to six roots) three with two roots at 8008
    // did not converge in 400 steps with the short one and took 124 to 259 with the long one.  So
    // V may grow to the long one after kDavShortSteps, with maxit steps from there.  Almost every
    // run is done by then; growing after 60 steps helped two roots (113 -> 79 ms) and cost six (179 ->
    // 229 ms, their 64 vectors).
    const double hx_s = (double)H.nnz * nb * (H.rvals ? 1.0 : 4.0) / 4.0e11;
    const int mmax = std::min(n, std::min(kJacobiMaxN, std::max(24, 8 * nb)));
    const int mshort = hx_s > 0.6e-3 ? mmax : std::min(mmax, std::max(12, 4 * nb));
    if (nwant < 1 || nb > mshort || n < 2) throw Error{DCG_E_ARG, "davidson: block does not fit the subspace"};
    const int64_t ld = n;
    cplx *V = wsget<cplx>(c, "dav.V", (size_t)n * mmax);
    cplx *W = wsget<cplx>(c, "dav.W", (size_t)n * mmax);
    cplx *X = wsget<cplx>(c, "dav.X", (size_t)n * nb);
    cplx *HX = wsget<cplx>(c, "dav.HX", (size_t)n * nb);
    cplx *T = wsget<cplx>(c, "dav.T", (size_t)n * nb);
    cplx *G = wsget<cplx>(c, "dav.G", (size_t)mmax * mmax);
    cplx *Y = wsget<cplx>(c, "dav.Y", (size_t)mmax * mmax);
    const int nchunk = (int)grid1d(n, kDavChunk);
    cplx *cf = wsget<cplx>(c, "dav.cf", (size_t)mmax * nchunk);
    cplx *rrp = wsget<cplx>(c, "dav.rrp", (size_t)mmax * 16 * nchunk);
    const int nrow = (int)grid1d(n, kAxpyRows);
    double *part = wsget<double>(c, "dav.part", (size_t)nchunk * 9 + nrow);   // residuals (8), then a direction's two norms
    double *pn0 = part + (size_t)nchunk * 8, *pn1 = pn0 + nchunk;
    double *th = wsget<double>(c, "dav.th", mmax);
    double *h2 = wsget<double>(c, "dav.h2", (size_t)nb);
    int *idx = wsget<int>(c, "dav.idx", nb);
    DavState *st = wsget<DavState>(c, "dav.st", 1);
    DavState *hst = reinterpret_cast<DavState *>(c.ws.host("dav.hst", sizeof(DavState)));

    // start: unit vectors on the nb lowest diagonal elements (ties by index)
    std::vector<double> hdh(n);
    DCG_CUDA(cudaMemcpyAsync(hdh.data(), H.diag, sizeof(double) * n, cudaMemcpyDeviceToHost, c.stream));
    DCG_CUDA(cudaStreamSynchronize(c.stream));
    double hscale = 1.0;
    for (double x : hdh) hscale = std::max(hscale, std::fabs(x));
    const double tol = tol_rel * hscale;
    std::vector<int> order(n);
    std::iota(order.begin(), order.end(), 0);
    std::partial_sort(order.begin(), order.begin() + nb, order.end(),
                      [&](int a, int b) { return hdh[a] < hdh[b] || (hdh[a] == hdh[b] && a < b); });
    DCG_CUDA(cudaMemcpyAsync(idx, order.data(), sizeof(int) * nb, cudaMemcpyHostToDevice, c.stream));
    unit_cols_kernel<<<grid1d((int64_t)n * nb, 256), 256, 0, c.stream>>>(n, nb, idx, V, ld);
    DCG_LAUNCHED(c);
    if (nb > 8) throw Error{DCG_E_ARG, "davidson: more than 8 directions per step"};
    csr_hx(c, H, V, W, ld, nb, nullptr);
    DCG_LAUNCHED(c);
    DavState s0{};
    s0.m = nb;
    s0.cap = mshort;
    DCG_CUDA(cudaMemcpyAsync(st, &s0, sizeof(DavState), cudaMemcpyHostToDevice, c.stream));

    const int np = mmax + (mmax & 1);
    const bool real = H.rvals != nullptr;
    const size_t jsmem = 2 * (real ? sizeof(double) : sizeof(cplx)) * (size_t)np * np;
    auto *k_jac = real ? jacobi_heev_kernel<true> : jacobi_heev_kernel<false>;
    DCG_CUDA(cudaFuncSetAttribute(k_jac, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  2 * (int)sizeof(cplx) * kJacobiMaxN * kJacobiMaxN));
    auto *k_rr = real ? rr_part_kernel<true> : rr_part_kernel<false>;
    auto *k_rrs = real ? rr_sum_kernel<true> : rr_sum_kernel<false>;
    auto *k_ritz = real ? ritz_kernel<true> : ritz_kernel<false>;
    auto *k_res = real ? residual_kernel<true> : residual_kernel<false>;
    auto *k_cand = real ? cand_begin_kernel<true> : cand_begin_kernel<false>;
    auto *k_dot = real ? cgs_dot_kernel<true> : cgs_dot_kernel<false>;
    auto *k_axpy = real ? cgs_axpy_kernel<true> : cgs_axpy_kernel<false>;
    auto enqueue_step = [&]() {
        k_rr<<<dim3(mmax, 2 * nb, nchunk), kDavThreads, 0, c.stream>>>(n, V, W, ld, rrp, mmax, st);
        k_rrs<<<2 * nb, 256, 0, c.stream>>>(nchunk, rrp, mmax, G, mmax, st);
        k_jac<<<1, kJacobiThreads, jsmem, c.stream>>>(mmax, &st->m, G, mmax, th, Y, mmax, &st->jac);
        k_ritz<<<dim3(grid1d(n, 128), nb, 2), 128, 0, c.stream>>>(n, V, W, ld, Y, mmax, X, HX, st);
        k_res<<<dim3(nchunk, nb), kDavThreads, 0, c.stream>>>(n, HX, X, ld, th, H.diag, T, part);
        step_begin_kernel<<<1, 256, 0, c.stream>>>(nwant, nb, nchunk, part, h2, st);
        restart_copy_kernel<<<grid1d((int64_t)n * nb, 256), 256, 0, c.stream>>>(n, nb, X, HX, V, W, ld, st);
        restart_set_kernel<<<1, 32, 0, c.stream>>>(nb, st);
        for (int q = 0; q < nb; q++) {
            k_cand<<<nchunk, kDavThreads, 0, c.stream>>>(n, q, tol, h2, T, V, ld, pn0, st);
            for (int pass = 0; pass < 2; pass++) {
                k_dot<<<dim3(mmax, nchunk), kDavThreads, 0, c.stream>>>(n, q, V, ld, cf, mmax, st);
                k_axpy<<<nrow, kAxpyRows, 0, c.stream>>>(n, q, nchunk, V, ld, cf, mmax, pn1, st);
            }
            cand_end_kernel<<<nchunk, kDavThreads, 0, c.stream>>>(n, q, V, ld, pn0, pn1, nrow, st);
        }
        csr_hx(c, H, V, W, ld, nb, st);
        step_end_kernel<<<1, 32, 0, c.stream>>>(st);
        DCG_CUDA(cudaMemcpyAsync(hst, st, sizeof(DavState), cudaMemcpyDeviceToHost, c.stream));
    };
    const int step_kernels = 10 + 6 * nb;   // kernels per step

    static const bool use_graph = [] {
        const char *e = getenv("DCG_DAVIDSON_GRAPH");
        return !(e && e[0] == '0');
    }();
    cudaGraphExec_t exec = nullptr;
    if (use_graph) {
        cudaGraph_t graph = nullptr;
        DCG_CUDA(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal));
        enqueue_step();
        DCG_CUDA(cudaStreamEndCapture(c.stream, &graph));
        const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) throw Error{DCG_E_CUDA, std::string("davidson graph: ") + cudaGetErrorString(e)};
    }
    struct ExecGuard {
        cudaGraphExec_t g;
        ~ExecGuard() {
            if (g) cudaGraphExecDestroy(g);
        }
    } guard{exec};

    bool converged = false;
    c.casci_iters = 0;
    if (mshort < mmax) maxit += kDavShortSteps;
    for (int it = 0; it < maxit; it++) {
        if (it == kDavShortSteps && mshort < mmax)
            DCG_CUDA(cudaMemcpyAsync(&st->cap, &mmax, sizeof(int), cudaMemcpyHostToDevice, c.stream));
        if (exec) {
            DCG_CUDA(cudaGraphLaunch(exec, c.stream));
            c.launches += step_kernels;
        } else {
            enqueue_step();
            c.launches += step_kernels;
        }
        DCG_CUDA(cudaStreamSynchronize(c.stream));
        c.casci_iters = it + 1;
        if (hst->worst <= tol) {
            converged = true;
            break;
        }
        if (hst->cand == 0) break;   // stagnated: reported below
    }
    if (!converged || hst->jac != 0)
        throw Error{DCG_E_NUMERIC, "CASCI Davidson did not converge to |r| <= " + std::to_string(tol)};
    DCG_CUDA(cudaMemcpyAsync(w, th, sizeof(double) * nwant, cudaMemcpyDeviceToDevice, c.stream));
    DCG_CUDA(cudaMemcpyAsync(Z, X, sizeof(cplx) * (size_t)n * nwant, cudaMemcpyDeviceToDevice, c.stream));
}

}  // namespace dcg
