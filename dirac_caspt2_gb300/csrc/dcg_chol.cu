// Blocked Cholesky factorisation A = L L^H of a Hermitian matrix and the solve A X = B on the
// device (Golub & Van Loan, Matrix Computations, 4th ed., 4.2.8-4.2.9: right-looking block
// form).  Per 48-column panel: the diagonal block is factored in one block's shared memory,
// the rows below it by a triangular solve against it, and the trailing matrix by one FP64
// GEMM.  The factorisation records the first non-positive pivot (the matrix is then not
// positive definite).
#include "dcg_common.cuh"

namespace dcg {

namespace {

constexpr int CH_NB = 48;   // panel width: the 48 x 49 complex tile fits the 48 KB of static shared memory
constexpr int CH_SLAB = 256;   // columns of one trailing update: below a few slabs the square costs no more than its launches

// a -= x conj(y) and a -= x y, complex or real
template <bool REAL>
__device__ __forceinline__ void ch_sub_conj(cplx &a, cplx x, cplx y) {
    a.x = fma(-x.x, y.x, a.x);
    if (!REAL) {
        a.x = fma(-x.y, y.y, a.x);
        a.y = fma(-x.y, y.x, a.y);
        a.y = fma(x.x, y.y, a.y);
    }
}

// Factor the kb x kb diagonal block at A (lower triangle read and written), in shared memory.
// info: the first failing global pivot index + 1 (0 keeps going; a set info skips the work).
// Bound by the chain of its columns (one reciprocal square root, one scaling, one update): a
// warp's FP64 instruction holds a quarter of the SM for 77 clocks, so the root is one warp's
// alone and the update takes four FMAs an element.  48 columns in 79 us (125 us with a root and
// a division in every thread).
template <bool REAL>
__global__ void __launch_bounds__(512) chol_panel_kernel(int kb, int k0, cplx *A, int64_t lda, int *info) {
    __shared__ cplx s[CH_NB][CH_NB + 1];   // s[column][row]
    __shared__ double s_r[2];               // 1 / sqrt(pivot), sqrt(pivot)
    __shared__ int bad;
    if (*info != 0) return;
    for (int e = threadIdx.x; e < kb * kb; e += blockDim.x) {
        const int i = e % kb, j = e / kb;
        s[j][i] = A[i + (int64_t)j * lda];
    }
    if (threadIdx.x == 0) bad = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int j = 0; j < kb; j++) {
        if (warp == 0) {
            const double piv = s[j][j].x;
            if (!(piv > 0.0)) {   // also catches NaN
                if (lane == 0) bad = k0 + j + 1;
            } else {
                const bool safe = piv > 1e-290 && piv < 1e290;
                const double ri = safe ? fast_rsqrt(piv) : 1.0 / sqrt(piv);
                if (lane == 0) {
                    s_r[0] = ri;
                    s_r[1] = piv * ri;
                }
                __syncwarp();
                for (int i = j + 1 + lane; i < kb; i += 32) s[j][i] = mk(s[j][i].x * ri, REAL ? 0.0 : s[j][i].y * ri);
            }
        }
        __syncthreads();
        if (bad) break;
        if (threadIdx.x == 0) s[j][j] = mk(s_r[1], 0.0);
        // trailing lower part: s(i, l) -= s(i, j) conj(s(l, j)), j < l <= i: a warp per column
        for (int l = j + 1 + warp; l < kb; l += nw) {
            const cplx y = s[j][l];
            for (int i = l + lane; i < kb; i += 32) ch_sub_conj<REAL>(s[l][i], s[j][i], y);
        }
        __syncthreads();
    }
    if (bad) {
        if (threadIdx.x == 0) *info = bad;
        return;
    }
    for (int e = threadIdx.x; e < kb * kb; e += blockDim.x) {
        const int i = e % kb, j = e / kb;
        if (i >= j) A[i + (int64_t)j * lda] = s[j][i];
    }
}

// Triangular solves against the kb x kb factor L11 for CH_RHS vectors a block, each vector's
// element l in thread (l, vector):
//   CH_ROWS     X L11^H = A21, a vector per row of A21 (elements lda apart): the rows below a panel
//   CH_FORWARD  L11 Y = B, a vector per column of B
//   CH_BACKWARD L11^H X = B
// Column by column: the element's owner divides, every later element subtracts its multiple.
// One thread a vector took 300 us for any number of vectors (1,128 complex multiply-adds in a
// row at 77 clocks an FP64 instruction); this form takes 40 us.
constexpr int CH_RHS = 8;
enum ChSolve { CH_ROWS, CH_FORWARD, CH_BACKWARD };
template <bool REAL, int MODE>
__global__ void __launch_bounds__(CH_RHS *CH_NB) chol_solve_kernel(int kb, int nrhs, const cplx *L11, int64_t ldl, cplx *B,
                                                                    int64_t ldb, const int *info) {
    __shared__ cplx c[CH_NB][CH_NB + 1];   // c[j][l]: what element l subtracts of element j
    __shared__ double inv[CH_NB];
    __shared__ cplx xs[2][CH_RHS];
    if (info && *info != 0) return;
    for (int e = threadIdx.x; e < kb * kb; e += blockDim.x) {
        const int i = e % kb, j = e / kb;
        if (i < j) continue;
        const cplx v = L11[i + (int64_t)j * ldl];
        if (i == j) inv[j] = 1.0 / v.x;
        else if (MODE == CH_BACKWARD) c[i][j] = cconj(v);
        else c[j][i] = MODE == CH_ROWS ? cconj(v) : v;
    }
    const int r = threadIdx.x % CH_RHS, l = threadIdx.x / CH_RHS, q = blockIdx.x * CH_RHS + r;
    const bool have = q < nrhs && l < kb;
    cplx *p = B + (MODE == CH_ROWS ? q + (int64_t)l * ldb : l + (int64_t)q * ldb);
    cplx v = have ? *p : mk(0.0, 0.0);
    __syncthreads();
    for (int t = 0; t < kb; t++) {
        const int j = MODE == CH_BACKWARD ? kb - 1 - t : t;
        if (l == j) {
            v = mk(v.x * inv[j], REAL ? 0.0 : v.y * inv[j]);
            xs[t & 1][r] = v;
        }
        __syncthreads();   // xs alternates, so one barrier a step is enough
        if (MODE == CH_BACKWARD ? l < j : l > j && l < kb) {
            const cplx x = xs[t & 1][r], y = c[j][l];
            v.x = fma(-x.x, y.x, v.x);
            if (!REAL) {
                v.x = fma(x.y, y.y, v.x);
                v.y = fma(-x.x, y.y, v.y);
                v.y = fma(-x.y, y.x, v.y);
            }
        }
    }
    if (have) *p = v;
}

template <int MODE>
void launch_chol_solve(Context &c, int kb, int nrhs, const cplx *L11, int64_t ldl, cplx *B, int64_t ldb, const int *info) {
    auto *kern = c.real_now ? chol_solve_kernel<true, MODE> : chol_solve_kernel<false, MODE>;
    kern<<<grid1d(nrhs, CH_RHS), CH_RHS * CH_NB, 0, c.stream>>>(kb, nrhs, L11, ldl, B, ldb, info);
    DCG_LAUNCHED(c);
}

}  // namespace

void zpotrf_lower(Context &c, int n, cplx *A, int64_t lda, int *info) {
    DCG_CUDA(cudaMemsetAsync(info, 0, sizeof(int), c.stream));
    const cplx mone = mk(-1.0, 0.0), one = mk(1.0, 0.0);
    for (int k0 = 0; k0 < n; k0 += CH_NB) {
        const int kb = std::min(CH_NB, n - k0);
        cplx *A11 = A + k0 + (int64_t)k0 * lda;
        auto *panel = c.real_now ? chol_panel_kernel<true> : chol_panel_kernel<false>;
        panel<<<1, 512, 0, c.stream>>>(kb, k0, A11, lda, info);
        DCG_LAUNCHED(c);
        const int m = n - k0 - kb;
        if (m <= 0) break;
        cplx *A21 = A11 + kb;
        launch_chol_solve<CH_ROWS>(c, kb, m, A11, lda, A21, lda, info);
        // A22 -= A21 A21^H, the lower part alone (the upper one is never read): by column slabs
        cplx *A22 = A21 + (int64_t)kb * lda;
        for (int j0 = 0; j0 < m; j0 += CH_SLAB)
            zgemm(c, OP_N, OP_C, m - j0, std::min(CH_SLAB, m - j0), kb, mone, A21 + j0, lda, 0, A21 + j0, lda, 0, one,
                  A22 + j0 + (int64_t)j0 * lda, lda, 0, 1);
    }
}

void zpotrs_lower(Context &c, int n, const cplx *L, int64_t lda, cplx *B, int64_t ldb, int nrhs) {
    if (n <= 0 || nrhs <= 0) return;
    const cplx mone = mk(-1.0, 0.0), one = mk(1.0, 0.0);
    for (int k0 = 0; k0 < n; k0 += CH_NB) {   // L Y = B
        const int kb = std::min(CH_NB, n - k0);
        const cplx *L11 = L + k0 + (int64_t)k0 * lda;
        launch_chol_solve<CH_FORWARD>(c, kb, nrhs, L11, lda, B + k0, ldb, nullptr);
        const int m = n - k0 - kb;
        if (m > 0) zgemm(c, OP_N, OP_N, m, nrhs, kb, mone, L11 + kb, lda, 0, B + k0, ldb, 0, one, B + k0 + kb, ldb, 0, 1);
    }
    for (int k0 = ((n - 1) / CH_NB) * CH_NB; k0 >= 0; k0 -= CH_NB) {   // L^H X = Y
        const int kb = std::min(CH_NB, n - k0);
        const cplx *L11 = L + k0 + (int64_t)k0 * lda;
        const int m = n - k0 - kb;
        if (m > 0) zgemm(c, OP_C, OP_N, kb, nrhs, m, mone, L11 + kb, lda, 0, B + k0 + kb, ldb, 0, one, B + k0, ldb, 0, 1);
        launch_chol_solve<CH_BACKWARD>(c, kb, nrhs, L11, lda, B + k0, ldb, nullptr);
    }
}

}  // namespace dcg

namespace dcg {

namespace {

__device__ __forceinline__ double wsum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Wm[m + Mp i] = 1 / (D_m + alpha_i) (complex, zero imaginary part); A = U o Wm.
__global__ void wb_weights_kernel(int Mp, int nouter, const double *__restrict__ Dd, const double *__restrict__ alpha,
                                  const cplx *__restrict__ U, int64_t ldu, cplx *Wm, cplx *A) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)Mp * nouter) return;
    const int m = (int)(e % Mp), i = (int)(e / Mp);
    const double w = 1.0 / (Dd[m] + alpha[i]);
    Wm[e] = mk(w, 0.0);
    const cplx u = U[m + ldu * i];
    A[e] = mk(u.x * w, u.y * w);
}

// Phi[p + npair m] = conj(Ps[m, k]) Ps[m, l] for the packed pairs p = (k <= l) of r columns.
__global__ void wb_phi_kernel(int Mp, int r, const cplx *__restrict__ Ps, int64_t ldp, cplx *Phi) {
    const int npair = r * (r + 1) / 2;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)npair * Mp) return;
    const int p = (int)(e % npair), m = (int)(e / npair);
    int q = p, k = 0;
    while (q >= r - k) {
        q -= r - k;
        k++;
    }
    const int l = k + q;
    Phi[e] = cmul(cconj(Ps[m + ldp * k]), Ps[m + ldp * l]);
}

// Per outer index i (one block): C_i (r x r Hermitian, unpacked from column i of Cp into shared
// memory) x = b_i by Gaussian elimination with partial pivoting (rows updated in parallel);
// x to X[:, i].
__global__ void __launch_bounds__(256) wb_solve_kernel(int r, const cplx *__restrict__ Cp, const cplx *__restrict__ Bv,
                                                       cplx *X) {
    extern __shared__ double2 wsm[];
    cplx *C = wsm, *xv = C + r * r;
    __shared__ int piv_s;
    const int i = blockIdx.x, npair = r * (r + 1) / 2;
    const cplx *cp = Cp + (int64_t)npair * i;
    for (int p = threadIdx.x; p < npair; p += blockDim.x) {
        int q = p, k = 0;
        while (q >= r - k) {
            q -= r - k;
            k++;
        }
        const int l = k + q;
        const cplx v = cp[p];
        C[k + r * l] = v;
        C[l + r * k] = cconj(v);
    }
    for (int k = threadIdx.x; k < r; k += blockDim.x) xv[k] = Bv[k + (int64_t)r * i];
    __syncthreads();
    for (int k = 0; k < r; k++) {
        if (threadIdx.x == 0) {
            int p = k;
            double best = cabs2(C[k + r * k]);
            for (int q = k + 1; q < r; q++) {
                const double v = cabs2(C[q + r * k]);
                if (v > best) {
                    best = v;
                    p = q;
                }
            }
            piv_s = p;
        }
        __syncthreads();
        const int p = piv_s;
        if (p != k) {
            for (int j = threadIdx.x; j < r; j += blockDim.x) {
                const cplx t = C[k + r * j];
                C[k + r * j] = C[p + r * j];
                C[p + r * j] = t;
            }
            if (threadIdx.x == 0) {
                const cplx t = xv[k];
                xv[k] = xv[p];
                xv[p] = t;
            }
        }
        __syncthreads();
        const cplx inv = cdiv(mk(1.0, 0.0), C[k + r * k]);
        for (int q = k + 1 + threadIdx.x; q < r; q += blockDim.x) {
            const cplx f = cmul(C[q + r * k], inv);
            for (int j = k + 1; j < r; j++) C[q + r * j] = csub(C[q + r * j], cmul(f, C[k + r * j]));
            xv[q] = csub(xv[q], cmul(f, xv[k]));
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = r - 1; k >= 0; k--) {
            cplx s = xv[k];
            for (int j = k + 1; j < r; j++) s = csub(s, cmul(C[k + r * j], xv[j]));
            xv[k] = cdiv(s, C[k + r * k]);
        }
    __syncthreads();
    for (int k = threadIdx.x; k < r; k += blockDim.x) X[k + (int64_t)r * i] = xv[k];
}

// Per outer index i: z = Wm o Zm; e2o = -Re u^H z, sco = |z|^2 (fixed-order block reduction).
__global__ void __launch_bounds__(256) wb_e2_kernel(int Mp, const cplx *__restrict__ U, int64_t ldu,
                                                    const cplx *__restrict__ Zm, const cplx *__restrict__ Wm,
                                                    double *e2o, double *sco) {
    __shared__ double red[2][8];
    const int i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double e = 0.0, s2 = 0.0;
    for (int m = threadIdx.x; m < Mp; m += blockDim.x) {
        const double w = Wm[m + (int64_t)Mp * i].x;
        const cplx zz = Zm[m + (int64_t)Mp * i];
        const cplx z = mk(zz.x * w, zz.y * w), u = U[m + ldu * i];
        e += u.x * z.x + u.y * z.y;
        s2 += z.x * z.x + z.y * z.y;
    }
    e = wsum(e);
    s2 = wsum(s2);
    if (lane == 0) {
        red[0][warp] = e;
        red[1][warp] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double te = 0.0, ts = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            te += red[0][w];
            ts += red[1][w];
        }
        e2o[i] = -te;
        sco[i] = ts;
    }
}

}  // namespace

// With M_i = D + alpha_i (diagonal over the Mp determinants), the compression of M_i to the
// orthogonal complement of the r orthonormal columns of Ps has, on that complement, the inverse
// M^-1 - M^-1 Ps C^-1 Ps^H M^-1 with C = Ps^H M^-1 Ps (r x r).  For u = U[:, i] in the
// complement: z = M^-1 (u - Ps C^-1 b) with b = Ps^H M^-1 u, and e2o = -Re u^H z,
// sco = |z|^2.  The r x r matrices of all outer indices come from one GEMM of the packed pair
// products of Ps with the weights 1 / (D + alpha); then one pivoted r x r solve per index.
void launch_woodbury_e2(Context &c, int Mp, int r, const cplx *U, int64_t ldu, const cplx *Ps, int64_t ldp,
                        const double *Dd, const double *alpha, int nouter, double *e2o, double *sco) {
    if (nouter <= 0) return;
    const cplx one = mk(1.0, 0.0), zero = mk(0.0, 0.0), mone = mk(-1.0, 0.0);
    const int npair = r * (r + 1) / 2;
    const size_t mo = (size_t)Mp * nouter;
    constexpr int kWbMaxR = 112;   // (r^2 + r) complex in one block's shared memory
    cplx *Wm = wsget<cplx>(c, "wb.W", mo);
    cplx *A = wsget<cplx>(c, "wb.A", mo);
    cplx *Phi = wsget<cplx>(c, "wb.Phi", (size_t)npair * Mp);
    cplx *Cp = wsget<cplx>(c, "wb.C", (size_t)npair * nouter);
    cplx *Bv = wsget<cplx>(c, "wb.B", (size_t)r * nouter);
    cplx *X = wsget<cplx>(c, "wb.X", (size_t)r * nouter);
    cplx *Zm = wsget<cplx>(c, "wb.Z", mo);
    wb_weights_kernel<<<grid1d((int64_t)mo, 256), 256, 0, c.stream>>>(Mp, nouter, Dd, alpha, U, ldu, Wm, A);
    DCG_LAUNCHED(c);
    wb_phi_kernel<<<grid1d((int64_t)npair * Mp, 256), 256, 0, c.stream>>>(Mp, r, Ps, ldp, Phi);
    DCG_LAUNCHED(c);
    // C_i, packed: r(r+1)/2 x nouter x Mp, the largest product of the route.  On the split
    // path it runs on the tensor cores unless it is smaller than their fixed cost (C_i enters a
    // well-conditioned r x r solve, not the metric's inverse).
    if (c.precision == DCG_PREC_SPLIT && npair >= 128 && (double)npair * nouter * Mp >= 1.25e6)
        zgemm_split(c, npair, nouter, Mp, 1, Phi, 1, npair, 0, Wm, Mp, 0, Cp, 1, npair, 0, false, c.split_lbo,
                    c.split_sbo);
    else
        zgemm(c, OP_N, OP_N, npair, nouter, Mp, one, Phi, npair, 0, Wm, Mp, 0, zero, Cp, npair, 0, 1);
    zgemm(c, OP_C, OP_N, r, nouter, Mp, one, Ps, ldp, 0, A, Mp, 0, zero, Bv, r, 0, 1);            // b_i
    if (r > kWbMaxR) throw Error{DCG_E_ARG, "deflated Gram route: more eigenvalues under the cutoff than it takes"};
    const size_t smem = sizeof(cplx) * ((size_t)r * r + (size_t)r);
    DCG_CUDA(cudaFuncSetAttribute(wb_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    wb_solve_kernel<<<nouter, 256, smem, c.stream>>>(r, Cp, Bv, X);
    DCG_LAUNCHED(c);
    DCG_CUDA(cudaMemcpy2DAsync(Zm, (size_t)Mp * sizeof(cplx), U, (size_t)ldu * sizeof(cplx), (size_t)Mp * sizeof(cplx),
                               nouter, cudaMemcpyDeviceToDevice, c.stream));
    zgemm(c, OP_N, OP_N, Mp, nouter, r, mone, Ps, ldp, 0, X, r, 0, one, Zm, Mp, 0, 1);               // u - Ps x
    wb_e2_kernel<<<nouter, 256, 0, c.stream>>>(Mp, U, ldu, Zm, Wm, e2o, sco);
    DCG_LAUNCHED(c);
}

}  // namespace dcg
