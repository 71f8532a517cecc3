// FP64 Cholesky of the Coulomb metric, the inverse of its factor, and the
// formation of the fitted tensor B = L^{-1} (P|mu nu).
//
// The reference forms B = M^{-1/2} (P|mu nu) from an eigendecomposition,
// dropping eigenvalues below 1e-10 of the largest
// (hafnium/integrals/density_fitting.py:97-107, 181-197). Any factor with
// L L^T = M gives the same fitted integrals B^T B when nothing is dropped
// (the invariance the reference tests at tests/unit/test_density_fitting.py:177-195),
// so a Cholesky factor replaces the inverse square root. The smallest pivot
// relative to the largest diagonal is reported so the caller can see how close
// the metric is to the reference's drop threshold.
#include <algorithm>
#include <cmath>

#include "dgemm.cuh"
#include "linalg.cuh"
#include "md.cuh"

namespace hf {

namespace {
constexpr int NB = 64;

// One panel: every CTA factors the nb x nb diagonal block at (k0, k0) itself (the
// same values everywhere; a launch of its own cost more), CTA 0 writes the factor
// to diag (64 x 64, not into A, which the other CTAs still read), and each thread
// turns one row below it into L_ik = A_ik L_kk^-T by forward substitution.
//
// Both are serial chains over the 64 columns, so they hold one barrier per column
// and one division: 256 threads keep the block as 4 x 4 register tiles (rows and
// columns cyclic over a 16 x 16 grid); a column goes through shared memory
// unscaled, every thread takes the pivot's root and its reciprocal itself. The
// substitution runs right-looking (once x[q] is known it is subtracted from every
// later entry) with the pivots' reciprocals, taken once. Every quotient is corrected
// to a division's exact rounding (divide_by): the metric's condition amplifies an ulp
// of the factor to 1e-12 in J. A CTA takes
// 64 rows, moved through shared memory (a thread's own row is 512 bytes apart from
// its neighbour's). Measured (N = 1808): 54 + 46 us for two kernels with divisions,
// 47 us for this one without the staging, 33 us with it.
// blockIdx.y: the matrix of a batch.
__global__ void __launch_bounds__(256) k_panel(double* A, int64_t lda, int64_t strideA, int k0, int nb, int n,
                                               double* diag, int64_t strideD, int* info, double* piv_min) {
    A += blockIdx.y * strideA;
    diag += blockIdx.y * strideD;
    info += blockIdx.y;
    piv_min += blockIdx.y;
    extern __shared__ double panel_smem[];
    double (*l)[NB + 1] = reinterpret_cast<double (*)[NB + 1]>(panel_smem);  // the factor
    double (*t)[NB + 1] = l + NB;                                            // this CTA's rows
    __shared__ double col[2][NB];
    __shared__ double inv[NB];
    __shared__ int s_bad;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    double r[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = ty + 16 * a, j = tx + 16 * b;
            // past nb: the identity
            r[a][b] = (i < nb && j <= i) ? A[(int64_t)(k0 + i) * lda + k0 + j] : (i == j && i >= nb ? 1.0 : 0.0);
        }
    if (tid == 0) s_bad = NB;
    {
        // this CTA's rows, on their way while the block is factored
        const int row0 = k0 + nb + blockIdx.x * NB;
        for (int e = tid; e < NB * NB; e += 256)
            t[e / NB][e % NB] = (row0 + e / NB < n && e % NB < nb) ? A[(int64_t)(row0 + e / NB) * lda + k0 + e % NB] : 0.0;
    }
#pragma unroll
    for (int b4 = 0; b4 < 4; ++b4)
#pragma unroll 1
        for (int jj = 0; jj < 16; ++jj) {
            const int j = 16 * b4 + jj;
            double* c = col[j & 1];
            if (tx == jj)
#pragma unroll
                for (int a = 0; a < 4; ++a) c[ty + 16 * a] = r[a][b4];
            __syncthreads();
            const double d = c[j];
            const bool bad = !(d > 0.0);
            const double p = bad ? 1.0 : sqrt(d), s = 1.0 / p;
            double li[4], lc[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                li[a] = divide_by(c[ty + 16 * a], p, s);
                lc[a] = divide_by(c[tx + 16 * a], p, s);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = b4; b < 4; ++b)
                    if (tx + 16 * b > j) r[a][b] -= li[a] * lc[b];
            if (tx == jj) {
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const int i = ty + 16 * a;
                    r[a][b4] = i > j ? li[a] : (i == j ? p : 0.0);
                }
                if (bad && ty == 0) atomicMin(&s_bad, j);
            }
        }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) l[ty + 16 * a][tx + 16 * b] = r[a][b];
    __syncthreads();
    if (tid < NB) inv[tid] = 1.0 / l[tid][tid];
    if (blockIdx.x == 0) {
        for (int e = tid; e < NB * NB; e += 256) diag[e] = l[e / NB][e % NB];
        if (tid == 0) {
            if (s_bad < nb && *info == 0) *info = k0 + s_bad + 1;
            double m = *piv_min;
            for (int j = 0; j < nb; ++j)
                if (j != s_bad) m = fmin(m, l[j][j]);
            *piv_min = m;
        }
    }
    __syncthreads();
    const int row0 = k0 + nb + blockIdx.x * NB, rows = min(NB, n - row0);
    if (rows <= 0) return;
    if (tid < NB) {
        double x[NB];
#pragma unroll
        for (int j = 0; j < NB; ++j) x[j] = t[tid][j];
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            x[q] = divide_by(x[q], l[q][q], inv[q]);
#pragma unroll
            for (int j = q + 1; j < NB; ++j) x[j] -= x[q] * l[j][q];
        }
#pragma unroll
        for (int j = 0; j < NB; ++j) t[tid][j] = x[j];
    }
    __syncthreads();
    for (int e = tid; e < rows * NB; e += 256)
        if (e % NB < nb) A[(int64_t)(row0 + e / NB) * lda + k0 + e % NB] = t[e / NB][e % NB];
}

// The factor's lower triangle: diagonal blocks from diag, zeros above the diagonal.
__global__ void k_finish_lower(double* A, int64_t lda, int64_t strideA, int n, const double* __restrict__ diag,
                               int64_t strideD) {
    A += blockIdx.y * strideA;
    diag += blockIdx.y * strideD;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)n * n) return;
    const int i = (int)(e / n), j = (int)(e % n);
    const int k = i / NB;
    if (j > i) A[(int64_t)i * lda + j] = 0.0;
    else if (j / NB == k) A[(int64_t)i * lda + j] = diag[(int64_t)k * NB * NB + (i - k * NB) * NB + (j - k * NB)];
}

// out = max_i |A_ii|
__global__ void __launch_bounds__(1024) k_max_diagonal(const double* __restrict__ A, int64_t lda, int n, double* out) {
    __shared__ double w[32];
    double m = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(A[(int64_t)i * (lda + 1)]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 32; ++k) m = fmax(m, w[k]);
        *out = m;
    }
}

// Inverse of the lower-triangular diagonal blocks (k0, k0), k0 = 64 blockIdx.x,
// all at once (they are independent): one CTA per block, one thread per column,
// the substitution of k_panel on the unit vectors. Writes Linv (row-major) and
// LinvT. blockIdx.y: the matrix of a batch.
__global__ void __launch_bounds__(64) k_trtri_diag(const double* L, int64_t ld, int64_t strideL, int n, double* Linv,
                                                   double* LinvT) {
    L += blockIdx.y * strideL;
    Linv += blockIdx.y * strideL;
    LinvT += blockIdx.y * strideL;
    const int k0 = blockIdx.x * NB;
    const int nb = (n - k0 < NB) ? n - k0 : NB;
    __shared__ double l[NB][NB + 1];
    __shared__ double inv[NB];
    for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
        const int i = e / NB, j = e % NB;
        l[i][j] = (i < nb && j <= i) ? L[(int64_t)(k0 + i) * ld + k0 + j] : (i == j ? 1.0 : 0.0);
    }
    __syncthreads();
    inv[threadIdx.x] = 1.0 / l[threadIdx.x][threadIdx.x];
    __syncthreads();
    const int c = threadIdx.x;
    if (c >= nb) return;
    double x[NB];
#pragma unroll
    for (int r = 0; r < NB; ++r) x[r] = r == c ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        x[q] = divide_by(x[q], l[q][q], inv[q]);
#pragma unroll
        for (int j = q + 1; j < NB; ++j) x[j] -= x[q] * l[j][q];
    }
#pragma unroll
    for (int r = 0; r < NB; ++r) {
        if (r >= nb) continue;
        Linv[(int64_t)(k0 + r) * ld + k0 + c] = x[r];
        LinvT[(int64_t)(k0 + c) * ld + k0 + r] = x[r];
    }
}

__global__ void k_transpose(const double* in, double* out, int n, int64_t ld, int64_t stride) {
    in += blockIdx.z * stride;
    out += blockIdx.z * stride;
    __shared__ double t[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = by + j, c = bx + threadIdx.x;
        t[j][threadIdx.x] = (r < n && c < n) ? in[(int64_t)r * ld + c] : 0.0;
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += blockDim.y) {
        const int r = bx + j, c = by + threadIdx.x;
        if (r < n && c < n) out[(int64_t)r * ld + c] = t[threadIdx.x][j];
    }
}
}  // namespace

cudaError_t cholesky_lower(double* A, int n, int64_t lda, int* d_info, double* d_piv_min, double* work,
                           cudaStream_t stream, int count, int64_t strideA) {
    const int64_t sw = (int64_t)cholesky_work_doubles(n);
    constexpr int panel_bytes = 2 * NB * (NB + 1) * (int)sizeof(double);
    cudaError_t attr = cudaFuncSetAttribute(k_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_bytes);
    if (attr != cudaSuccess) return attr;
    for (int k0 = 0; k0 < n; k0 += NB) {
        const int nb = (n - k0 < NB) ? n - k0 : NB;
        const int rem = n - k0 - nb;
        k_panel<<<dim3(rem > 0 ? (rem + NB - 1) / NB : 1, count), 256, panel_bytes, stream>>>(
            A, lda, strideA, k0, nb, n, work + (int64_t)(k0 / NB) * NB * NB, sw, d_info, d_piv_min);
        if (rem > 0) {
            GemmArgs g{};
            g.M = g.N = rem;
            g.K = nb;
            g.A = g.B = A + (int64_t)(k0 + nb) * lda + k0;
            g.lda = g.ldb = lda;
            g.C = A + (int64_t)(k0 + nb) * lda + k0 + nb;
            g.ldc = lda;
            g.alpha = -1.0;
            g.beta = 1.0;
            g.kmode = 0;
            g.epi = 2;
            g.tile = 5;
            g.strideA = g.strideB = g.strideC = strideA;
            cudaError_t e = dgemm_nt(g, count, stream);
            if (e != cudaSuccess) return e;
        }
    }
    const int64_t total = (int64_t)n * n;
    k_finish_lower<<<dim3((unsigned)((total + 255) / 256), count), 256, 0, stream>>>(A, lda, strideA, n, work, sw);
    return cudaGetLastError();
}

size_t cholesky_work_doubles(int n) { return (size_t)((n + NB - 1) / NB) * NB * NB; }

cudaError_t max_diagonal(const double* A, int n, int64_t lda, double* out, cudaStream_t stream) {
    k_max_diagonal<<<1, 1024, 0, stream>>>(A, lda, n, out);
    return cudaGetLastError();
}

cudaError_t triangular_inverse(const double* L, int n, int64_t ld, double* Linv, double* LinvT, double* work,
                               cudaStream_t stream, int count, int64_t stride, int64_t strideW) {
    const size_t bytes = sizeof(double) * (size_t)(count > 1 ? (count - 1) * stride : 0) + sizeof(double) * (size_t)n * ld;
    cudaMemsetAsync(Linv, 0, bytes, stream);
    cudaMemsetAsync(LinvT, 0, bytes, stream);
    k_trtri_diag<<<dim3((n + NB - 1) / NB, count), 64, 0, stream>>>(L, ld, stride, n, Linv, LinvT);
    for (int k0 = NB; k0 < n; k0 += NB) {
        const int nb = (n - k0 < NB) ? n - k0 : NB;
        // Wt[c][m] = sum_{k in [c, k0)} L[k0 + m][k] Linv[k][c]   (c < k0)
        GemmArgs g{};
        g.M = nb;
        g.N = k0;
        g.K = k0;
        g.A = L + (int64_t)k0 * ld;
        g.lda = ld;
        g.B = LinvT;
        g.ldb = ld;
        g.C = work;
        g.ldc = NB;
        g.alpha = 1.0;
        g.kmode = 1;
        g.epi = 1;
        g.tile = 5;
        g.strideA = g.strideB = stride;
        g.strideC = strideW;
        cudaError_t e = dgemm_nt(g, count, stream);
        if (e != cudaSuccess) return e;
        // Linv[k0 + m][c] = -sum_j Linv_kk[m][j] W[j][c]; stored transposed into LinvT.
        GemmArgs h{};
        h.M = nb;
        h.N = k0;
        h.K = nb;
        h.A = Linv + (int64_t)k0 * ld + k0;
        h.lda = ld;
        h.B = work;
        h.ldb = NB;
        h.C = LinvT + k0;
        h.ldc = ld;
        h.alpha = -1.0;
        h.epi = 1;
        h.tile = 5;
        h.strideA = h.strideC = stride;
        h.strideB = strideW;
        e = dgemm_nt(h, count, stream);
        if (e != cudaSuccess) return e;
    }
    dim3 grid((n + 31) / 32, (n + 31) / 32, count);
    k_transpose<<<grid, dim3(32, 8), 0, stream>>>(LinvT, Linv, n, ld, stride);
    return cudaGetLastError();
}

size_t inverse_work_doubles(int n) { return (size_t)n * NB; }

cudaError_t apply_inverse_factor(const double* Linv, int n, int64_t ld, const double* T, int64_t ldt, int64_t ncols,
                                 double* B, int64_t ldb, cudaStream_t stream, int row0, int row1) {
    if (row1 < 0) row1 = n;
    GemmArgs g{};
    g.M = row1 - row0;
    g.N = (int)ncols;
    g.K = row1;  // L^-1 is lower triangular: rows below row1 need columns below row1
    g.koff = row0;
    g.A = Linv + (int64_t)row0 * ld;
    g.lda = ld;
    g.B = T;
    g.ldb = ldt;
    g.C = B;
    g.ldc = ldb;
    g.alpha = 1.0;
    g.beta = 0.0;
    g.kmode = 2;
    g.epi = 0;
    g.tile = 5;  // 64 x 64 with 2 stages of 32-wide k slices: the fastest tile for this product
    return dgemm_nt(g, 1, stream);
}

}  // namespace hf
