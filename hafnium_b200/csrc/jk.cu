// Coulomb and exchange builds over the packed fitted tensor.
//
// Reference: hafnium/scf/coulomb_exchange.py:176-190. The reference holds B as
// [aux, ao, ao] and computes J = (B . vec D) . B and K = sum_P B_P D B_P. Here B
// is stored once per auxiliary index as the upper-triangle 64x64 tiles of
// B_P (layout: B[q][tile][64][64], tile (I, J >= I) at I*nt - I(I-1)/2 + J - I):
//
//   J:  c_q = sum_t w_t <B_q[t], D[t]>  (w = 1 on diagonal tiles, 2 above), then
//       J[t] = sum_q c_q B_q[t]; both passes stream B once from HBM.
//   K:  with D = C W C^T (W diagonal), X_q = B_q C and K = sum_q X_q W X_q^T.
//       The half-transform runs per q on DMMA tensor cores reading the tiles of
//       B_q (transposed for tiles below the diagonal); the second product is a
//       GEMM over the q-chunk, only upper 64x64 output tiles computed.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "dgemm.cuh"
#include "jk.cuh"

namespace hf {

namespace {

__device__ __forceinline__ const double* cluster_tensor(const double* const* Btab, const double* B, int c) {
    return Btab ? Btab[c] : B;
}

// Dw[t][r][c] = scale w_t D[64I + r][64J + c], zero outside n; cluster blockIdx.y.
__global__ void k_pack_density(const double* __restrict__ D, int64_t strideD, double scale, int64_t n, int nt,
                               double* __restrict__ Dw, int64_t strideW, const int* __restrict__ active) {
    const int cl = blockIdx.y;
    if (active && active[cl] == 0) return;
    D += cl * strideD;
    Dw += cl * strideW;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t ntiles = (int64_t)nt * (nt + 1) / 2;
    if (e >= ntiles * 4096) return;
    const int64_t t = e >> 12;
    const int r = (int)((e >> 6) & 63), c = (int)(e & 63);
    // tile index -> (I, J): rows of the upper triangle, row I holds nt - I tiles
    int I = 0;
    int64_t base = 0;
    while (base + (nt - I) <= t) {
        base += nt - I;
        ++I;
    }
    const int J = I + (int)(t - base);
    const int64_t mu = 64 * (int64_t)I + r, nu = 64 * (int64_t)J + c;
    double v = 0.0;
    if (mu < n && nu < n) v = (I == J ? scale : 2.0 * scale) * D[mu * n + nu];
    Dw[e] = v;
}

// c[q] = sum_e B[q][e] Dw[e]; one CTA per (q, cluster), 128-bit loads.
__global__ void __launch_bounds__(512) k_coulomb_charges(const double* const* __restrict__ Btab,
                                                         const double* __restrict__ B, int64_t ldb, int64_t nelem,
                                                         const double* __restrict__ Dw, double* __restrict__ c,
                                                         int64_t strideW, const int* __restrict__ active) {
    const int q = blockIdx.x, cl = blockIdx.y;
    if (active && active[cl] == 0) return;
    B = cluster_tensor(Btab, B, cl);
    Dw += cl * strideW;
    c += cl * strideW;
    const double2* row = reinterpret_cast<const double2*>(B + (int64_t)q * ldb);
    const double2* d = reinterpret_cast<const double2*>(Dw);
    const int64_t n2 = nelem / 2;
    double s0 = 0.0, s1 = 0.0;
    int64_t i = threadIdx.x;
    for (; i + 3 * blockDim.x < n2; i += 4 * blockDim.x) {
        double2 b0 = __ldcs(row + i), b1 = __ldcs(row + i + blockDim.x), b2 = __ldcs(row + i + 2 * blockDim.x),
                b3 = __ldcs(row + i + 3 * blockDim.x);
        double2 d0 = __ldg(d + i), d1 = __ldg(d + i + blockDim.x), d2 = __ldg(d + i + 2 * blockDim.x),
                d3 = __ldg(d + i + 3 * blockDim.x);
        s0 += b0.x * d0.x + b1.x * d1.x + b2.x * d2.x + b3.x * d3.x;
        s1 += b0.y * d0.y + b1.y * d1.y + b2.y * d2.y + b3.y * d3.y;
    }
    for (; i < n2; i += blockDim.x) {
        double2 b0 = __ldcs(row + i), d0 = __ldg(d + i);
        s0 += b0.x * d0.x;
        s1 += b0.y * d0.y;
    }
    double s = s0 + s1;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ double part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = (threadIdx.x < blockDim.x / 32) ? part[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) c[q] = v;
    }
}

// Jt[e] += sum_{q in slab} c[q] B[q][e]; each thread owns two adjacent elements.
constexpr int kJSlab = 256;
__global__ void __launch_bounds__(256) k_coulomb_assemble(const double* const* __restrict__ Btab,
                                                          const double* __restrict__ B, int64_t ldb, int64_t nelem,
                                                          int naux, const double* __restrict__ c,
                                                          double* __restrict__ Jt, int64_t strideW,
                                                          const int* __restrict__ active) {
    const int cl = blockIdx.z;
    if (active && active[cl] == 0) return;
    B = cluster_tensor(Btab, B, cl);
    c += cl * strideW;
    Jt += cl * strideW;
    const int64_t e2 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * e2 >= nelem) return;
    const int q0 = blockIdx.y * kJSlab;
    const int q1 = min(naux, q0 + kJSlab);
    double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
    int q = q0;
    for (; q + 1 < q1; q += 2) {
        const double2 x = __ldcs(reinterpret_cast<const double2*>(B + (int64_t)q * ldb) + e2);
        const double2 y = __ldcs(reinterpret_cast<const double2*>(B + (int64_t)(q + 1) * ldb) + e2);
        const double cq = __ldg(c + q), cr = __ldg(c + q + 1);
        a0 += cq * x.x;
        a1 += cq * x.y;
        b0 += cr * y.x;
        b1 += cr * y.y;
    }
    if (q < q1) {
        const double2 x = __ldcs(reinterpret_cast<const double2*>(B + (int64_t)q * ldb) + e2);
        const double cq = __ldg(c + q);
        a0 += cq * x.x;
        a1 += cq * x.y;
    }
    atomicAdd(Jt + 2 * e2, a0 + b0);
    atomicAdd(Jt + 2 * e2 + 1, a1 + b1);
}

// Full symmetric matrix from upper 64x64 tiles: J[mu][nu] = tiles(min, max).
__global__ void k_unpack_tiles(const double* __restrict__ Jt, int64_t strideW, int64_t n, int nt,
                               double* __restrict__ J, int64_t strideJ, const int* __restrict__ active) {
    const int cl = blockIdx.y;
    if (active && active[cl] == 0) return;
    Jt += cl * strideW;
    J += cl * strideJ;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    int64_t mu = e / n, nu = e % n;
    int I = (int)(mu >> 6), Jc = (int)(nu >> 6);
    if (I > Jc) {
        const int64_t t = mu;
        mu = nu;
        nu = t;
        const int ti = I;
        I = Jc;
        Jc = ti;
    }
    const int64_t tile = (int64_t)I * nt - (int64_t)I * (I - 1) / 2 + (Jc - I);
    J[e] = Jt[tile * 4096 + (mu & 63) * 64 + (nu & 63)];
}

// K[mu][nu] from the upper-tile-valid padded matrix Kp (row stride ldk).
__global__ void k_symmetrize_upper(const double* __restrict__ Kp, int64_t ldk, int64_t n, double* __restrict__ K,
                                   int64_t strideK, const int* __restrict__ active) {
    const int cl = blockIdx.y;
    if (active && active[cl] == 0) return;
    Kp += cl * ldk * ldk;
    K += cl * strideK;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t mu = e / n, nu = e % n;
    K[e] = mu <= nu ? Kp[mu * ldk + nu] : Kp[nu * ldk + mu];
}

// X[p][ql][i] = sum_r B_q[p][r] Ct[i][r] for q = q0 + ql: 64 x 64 tiles, 4 warps,
// mma.sync.m16n8k8 (FP64), a 2-stage pipeline of 32-wide k slices moved by
// 16-byte cp.async copies (three CTAs per SM; 128 x 64 tiles with 3 stages of 16
// were 4 % slower). The A operand comes from the packed tiles: tile (Ip, J) when
// Ip <= J, else tile (J, Ip) read in its own orientation and transposed by the
// fragment loads.
// The column tile is 32, 48, 64 or 80 wide, whichever pads the factor least: 160
// orbitals are two tiles of 80, not three of 64, and the 10 of a water dimer one of
// 32. 80-wide tiles keep three CTAs per SM with 3 stages of 16-wide slices.
constexpr int XBM = 64;
constexpr int XLDT = 64 + 4;  // pitch of a k-major half: conflict-free fragment loads
template <int XBN>
struct HalfShape {
    static constexpr int BK = XBN == 80 ? 16 : 32, ST = XBN == 80 ? 3 : 2, LD = BK + 4;
    static constexpr int NW = XBN == 32 ? 1 : 2;   // warps along the columns
    static constexpr int WN = XBN / NW, J = WN / 8;  // a warp: 32 x WN outputs
    static constexpr int THREADS = 64 * NW;
    static constexpr int SMEM = ST * (XBM + XBN) * LD * (int)sizeof(double);
    static_assert(BK * XLDT <= 64 * LD, "a k-major half fits in the p-major half's space");
    static_assert(64 % BK == 0, "a k slice stays inside one packed tile");
    static_assert(WN % 8 == 0 && (XBN * BK / 2) % THREADS == 0, "whole mma tiles and copies");
};

__device__ __forceinline__ uint32_t xsmem(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// 16-byte asynchronous copy (both addresses 16-byte aligned); an invalid piece
// copies nothing and zero-fills.
__device__ __forceinline__ void xcp16(double* dst, const double* src, const double* base, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(xsmem(dst)), "l"(valid ? src : base),
                 "r"(valid ? 16 : 0));
}

__device__ __forceinline__ void xmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

template <int XBN>
__global__ void __launch_bounds__(HalfShape<XBN>::THREADS, 3) k_exchange_half(const double* const* __restrict__ Btab,
                                                             const double* __restrict__ B, int64_t ldb, int q0, int nt,
                                                             const double* __restrict__ Ct, int64_t ldc_t,
                                                             int64_t strideCt, int n, int npad,
                                                             double* __restrict__ X,
                                                             int64_t ldx, int64_t strideX, int opad,
                                                             const int* __restrict__ active, int transposed) {
    using SH = HalfShape<XBN>;
    constexpr int XBK = SH::BK, XST = SH::ST, XLD = SH::LD, XTHREADS = SH::THREADS, J = SH::J;
    const int row_tiles = (npad + XBM - 1) / XBM;
    const int cl = blockIdx.y / row_tiles;
    if (active && active[cl] == 0) return;
    const int m0 = (blockIdx.y % row_tiles) * XBM, n0 = blockIdx.x * XBN;
    const int ql = blockIdx.z;
    B = cluster_tensor(Btab, B, cl);
    Ct += cl * strideCt;
    X += cl * strideX;
    const double* Bq = B + (int64_t)(q0 + ql) * ldb;
    extern __shared__ double xs[];
    double* As = xs;
    double* Bs = xs + XST * XBM * XLD;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gq = lane >> 2, tq = lane & 3;
    const int wm = warp / SH::NW * 32, wn = warp % SH::NW * SH::WN;
    const int nk = (n + XBK - 1) / XBK;  // B_q is zero past n
    // a warp whose rows are all past n, or whose columns are all past the factor's, only loads
    const bool live = m0 + wm < n && n0 + wn < opad;

    // Each stage holds the A rows as two 64-row halves. A half whose tile lies on
    // or above the diagonal (Ip <= J) is stored p-major ([p][k], pitch XLD) from
    // tile (Ip, J); a half below it reads tile (J, Ip), where k is the slow index,
    // and is stored k-major ([k][p], pitch XLDT) so that both the global reads and
    // the shared writes are contiguous; the fragment loads read it transposed.
    auto tile_at = [&](int I, int Jc) -> const double* {
        return Bq + ((int64_t)I * nt - (int64_t)I * (I - 1) / 2 + (Jc - I)) * 4096;
    };
    auto load = [&](int stage, int k0) {
        double* as = As + stage * XBM * XLD;
        double* bs = Bs + stage * XBN * XLD;
        const int Jt = k0 >> 6, kin = k0 & 63;
        constexpr int PIECES = 64 * XBK / 2;  // 16-byte pieces of a 64 x XBK half
#pragma unroll
        for (int h = 0; h < XBM / 64; ++h) {
            const int p0 = m0 + 64 * h;
            const int Ip = p0 >> 6;
            double* ah = as + h * 64 * XLD;
            const bool valid = p0 < npad;
            const bool below = Ip > Jt;
            const double* tile = valid ? (below ? tile_at(Jt, Ip) : tile_at(Ip, Jt)) : Bq;
#pragma unroll
            for (int c = 0; c < PIECES / XTHREADS; ++c) {
                const int e = tid + c * XTHREADS;
                if (!below) {
                    const int r = e / (XBK / 2), kp = (e % (XBK / 2)) * 2;
                    xcp16(ah + r * XLD + kp, tile + r * 64 + kin + kp, Bq, valid);
                } else {
                    const int k = e >> 5, pp = (e & 31) * 2;
                    xcp16(ah + k * XLDT + pp, tile + (kin + k) * 64 + pp, Bq, valid);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < XBN * XBK / 2 / XTHREADS; ++c) {
            const int e = tid + c * XTHREADS;  // the 16-byte pieces of the XBN x XBK tile of Ct
            const int r = e / (XBK / 2), kp = (e % (XBK / 2)) * 2;
            xcp16(bs + r * XLD + kp, Ct + (int64_t)(n0 + r) * ldc_t + k0 + kp, Ct, n0 + r < opad);
        }
    };

    double acc[2][J][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[i][j][v] = 0.0;
#pragma unroll
    for (int s = 0; s < XST - 1; ++s) {
        if (s < nk) load(s, s * XBK);
        asm volatile("cp.async.commit_group;\n" ::);
    }
    for (int it = 0; it < nk; ++it) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(XST - 2));
        __syncthreads();
        const int nxt = it + XST - 1;
        if (nxt < nk) load(nxt % XST, nxt * XBK);
        asm volatile("cp.async.commit_group;\n" ::);
        const double* as = As + (it % XST) * XBM * XLD;
        const double* bs = Bs + (it % XST) * XBN * XLD;
        // this warp's 32 rows lie in one half; that half's layout for this k tile
        const int hh = wm >> 6, lr = wm & 63;
        const bool below = ((m0 >> 6) + hh) > ((it * XBK) >> 6);
        const double* ah = as + hh * 64 * XLD;
        if (!live) continue;
#pragma unroll
        for (int kk = 0; kk < XBK; kk += 8) {
            double af[2][4], bf[J][2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int row = lr + i * 16 + gq;
                if (!below) {
                    const double* r0 = ah + row * XLD + kk + tq;
                    af[i][0] = r0[0];
                    af[i][1] = r0[8 * XLD];
                    af[i][2] = r0[4];
                    af[i][3] = r0[8 * XLD + 4];
                } else {
                    const double* c0 = ah + (kk + tq) * XLDT + row;
                    af[i][0] = c0[0];
                    af[i][1] = c0[8];
                    af[i][2] = c0[4 * XLDT];
                    af[i][3] = c0[4 * XLDT + 8];
                }
            }
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const double* c0 = bs + (wn + j * 8 + gq) * XLD + kk + tq;
                bf[j][0] = c0[0];
                bf[j][1] = c0[4];
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < J; ++j) xmma(acc[i][j], af[i], bf[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    if (transposed) {
        // Xt[(ql, i)][p]: row (ql opad + i), row stride npad
        double* xt = X + (int64_t)ql * opad * npad;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int m = m0 + wm + i * 16 + gq + h * 8;
                    const int nn = n0 + wn + j * 8 + 2 * tq;
                    if (m < npad && nn < opad) {
                        xt[(int64_t)nn * npad + m] = acc[i][j][2 * h];
                        xt[(int64_t)(nn + 1) * npad + m] = acc[i][j][2 * h + 1];
                    }
                }
        return;
    }
    double* xo = X + (int64_t)ql * opad;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < J; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = m0 + wm + i * 16 + gq + h * 8;
                const int nn = n0 + wn + j * 8 + 2 * tq;
                if (m < npad && nn < opad)
                    *reinterpret_cast<double2*>(xo + (int64_t)m * ldx + nn) = make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
            }
}

// Pivoted Cholesky of a symmetric PSD n x n matrix D in one CTA per cluster:
// rows of Lc ([rank][n]) with D ~= Lc^T Lc, stopping after maxr rows or when the
// largest remaining diagonal entry falls to tol times the largest initial one.
// out = {rank, indefinite}.
__global__ void __launch_bounds__(1024) k_pivoted_cholesky(const double* __restrict__ D, int64_t strideD, int n,
                                                           double tol, int maxr, double* __restrict__ Lc,
                                                           int64_t strideL, int* __restrict__ out,
                                                           const int* __restrict__ active) {
    const int cl = blockIdx.x;
    if (active && active[cl] == 0) return;
    D += cl * strideD;
    Lc += cl * strideL;
    out += 2 * cl;
    extern __shared__ double sm[];
    double* d = sm;                                  // n
    unsigned char* used = (unsigned char*)(sm + n);  // n
    __shared__ double rv[32];
    __shared__ int ri[32];
    __shared__ double s_dmax0, s_piv;
    __shared__ int s_p, s_stop;
    const int tid = threadIdx.x;
    for (int i = tid; i < n; i += blockDim.x) {
        d[i] = D[(int64_t)i * n + i];
        used[i] = 0;
    }
    __syncthreads();
    // largest |diagonal|
    double m = 0.0;
    for (int i = tid; i < n; i += blockDim.x) m = fmax(m, fabs(d[i]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((tid & 31) == 0) rv[tid >> 5] = m;
    __syncthreads();
    if (tid == 0) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) v = fmax(v, rv[w]);
        s_dmax0 = v;
    }
    __syncthreads();
    int k = 0;
    for (; k < maxr; ++k) {
        double best = -1.0;
        int bi = -1;
        for (int i = tid; i < n; i += blockDim.x)
            if (!used[i] && d[i] > best) {
                best = d[i];
                bi = i;
            }
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi >= 0 && (bi < 0 || oi < bi))) {
                best = ob;
                bi = oi;
            }
        }
        if ((tid & 31) == 0) {
            rv[tid >> 5] = best;
            ri[tid >> 5] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            double b = -1.0;
            int p = -1;
            for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w)
                if (rv[w] > b || (rv[w] == b && ri[w] >= 0 && (p < 0 || ri[w] < p))) {
                    b = rv[w];
                    p = ri[w];
                }
            s_stop = (p < 0 || !(b > tol * s_dmax0)) ? 1 : 0;
            s_p = p;
            s_piv = s_stop ? 0.0 : sqrt(b);
        }
        __syncthreads();
        if (s_stop) break;
        const int p = s_p;
        const double piv = s_piv;
        for (int i = tid; i < n; i += blockDim.x) {
            double l = 0.0;
            if (i == p) l = piv;
            else if (!used[i]) {
                double s = D[(int64_t)p * n + i];
                for (int j = 0; j < k; ++j) s -= Lc[(int64_t)j * n + i] * Lc[(int64_t)j * n + p];
                l = s / piv;
            }
            Lc[(int64_t)k * n + i] = l;
        }
        __syncthreads();
        for (int i = tid; i < n; i += blockDim.x) {
            if (i == p) used[i] = 1;
            else if (!used[i]) {
                const double l = Lc[(int64_t)k * n + i];
                d[i] -= l * l;
            }
        }
        __syncthreads();
    }
    // indefinite if a remaining diagonal entry is clearly negative
    int bad = 0;
    for (int i = tid; i < n; i += blockDim.x)
        if (!used[i] && d[i] < -1e3 * tol * s_dmax0) bad = 1;
    bad = __syncthreads_or(bad);
    if (tid == 0) {
        out[0] = k;
        out[1] = bad;
    }
}

// Blocked pivoted Cholesky of one matrix: the pivots and the factor of
// k_pivoted_cholesky up to rounding, with the rows that pivots already taken
// subtract kept in a working copy W = D - sum L L^T that a DMMA product updates
// once per panel.
//
// A panel is one CTA's chain of pivots, so a pivot's latency is what counts. The
// panel's rows of L sit in shared memory (as many pivots per panel as fit: 158 at
// n = 160, 86 at n = 288, 14 at n = 1536, 8 at n = 2560; past that 32, with the rows
// in global memory), the pivot is found with one barrier (64-bit keys of value and
// index, reduced by two 32-bit warp reductions each), the pivot's row of W is on its
// way while the corrections are summed, and no division is in the chain. Per pivot
// about 0.6 us, where the rows of L in global memory and two shuffled reductions took
// 4 (n = 48) to 20 us (n = 1536).
struct PivotState {
    double dmax0;  // the largest initial diagonal entry
    int k;         // pivots taken
    int stop;      // 1 once the remaining diagonal falls below tol dmax0 or k reaches maxr
    int bad;       // 1 when a remaining diagonal entry is clearly negative (set with stop)
    int active;    // the trailing update of this panel has work (DMMA batch flag)
};

// The largest 64-bit key of a warp, in every lane.
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long key) {
    const unsigned hi = (unsigned)(key >> 32);
    const unsigned top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned low = __reduce_max_sync(0xffffffffu, hi == top ? (unsigned)key : 0u);
    return ((unsigned long long)top << 32) | low;
}

constexpr int kPivotThreads = 1024;
constexpr int kPivotRows = 22;  // rows per thread that the shared diagonal has room for (n <= 22528)

// One panel of up to `width` pivots of W (D itself for the first). Shared: d[n],
// Lp[n][pitch] when it fits (else Lp is the global copy). WIDE, for larger n: the
// diagonal and the used flags stay in global memory, keys have room for 2^20 rows.
template <bool WIDE>
__global__ void __launch_bounds__(kPivotThreads) k_pc_panel(const double* __restrict__ W, int n, double tol, int maxr,
                                                            double* __restrict__ Lc, double* __restrict__ Lg,
                                                            int width, int pitch, int in_smem,
                                                            double* __restrict__ dg, unsigned char* __restrict__ used,
                                                            int first, PivotState* st, PivotState* host) {
    extern __shared__ double psm[];
    __shared__ unsigned long long keys[2][32];
    __shared__ int s_bad;
    constexpr int kBits = WIDE ? 20 : 16;  // of a key: the index
    constexpr unsigned long long kIndex = (1ull << kBits) - 1;
    double* d = WIDE ? dg : psm;
    double* Lp = !WIDE && in_smem ? psm + n : Lg;
    const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, warps = T >> 5;
    if (!first && st->stop) {
        if (tid == 0) {
            st->active = 0;
            if (host) *host = *st;
        }
        return;
    }
    unsigned mine = 0;  // bit m: row tid + m T has been a pivot
    auto taken = [&](int i, int m) { return WIDE ? used[i] != 0 : (mine >> m & 1) != 0; };
    double top = 0.0;
    for (int i = tid, m = 0; i < n; i += T, ++m) {
        const double v = first ? W[(int64_t)i * n + i] : dg[i];
        d[i] = v;
        if (first) {
            top = fmax(top, fabs(v));
            if (WIDE) used[i] = 0;
        } else if (!WIDE && used[i]) {
            mine |= 1u << m;
        }
    }
    if (tid == 0) s_bad = 0;
    double dmax0;
    if (first) {
        const unsigned long long k = warp_max_key((unsigned long long)__double_as_longlong(top));
        if (lane == 0) keys[1][warp] = k;
        __syncthreads();
        dmax0 = __longlong_as_double((long long)warp_max_key(lane < warps ? keys[1][lane] : 0ull));
        __syncthreads();
    } else {
        dmax0 = st->dmax0;
        __syncthreads();
    }
    const int k0 = first ? 0 : st->k;
    const int b = min(width, maxr - k0);
    int j = 0;
    for (; j < b; ++j) {
        // the largest remaining diagonal entry, the lowest index among those equal to 2^-36 (2^-32) of it
        unsigned long long key = 0;
        for (int i = tid, m = 0; i < n; i += T, ++m)
            if (!taken(i, m) && d[i] > 0.0) {
                const unsigned long long k =
                    ((unsigned long long)__double_as_longlong(d[i]) & ~kIndex) | (kIndex - (unsigned long long)i);
                key = k > key ? k : key;
            }
        key = warp_max_key(key);
        if (lane == 0) keys[j & 1][warp] = key;
        __syncthreads();
        key = warp_max_key(lane < warps ? keys[j & 1][lane] : 0ull);
        const int p = key ? (int)(kIndex - (key & kIndex)) : 0;
        const double best = key ? d[p] : 0.0;
        if (!(best > tol * dmax0)) break;
        const double piv = sqrt(best), inv = 1.0 / piv;
        const double* __restrict__ w = W + (int64_t)p * n;
        const double* lp = Lp + (int64_t)p * pitch;
        // each thread owns rows i = tid + m T: it alone writes their entries of L, their diagonal and their
        // used bit, so the search's barrier suffices
        for (int i = tid, m = 0; i < n; i += T, ++m) {
            double l = 0.0;
            if (i == p) {
                l = piv;
                if (WIDE) used[i] = 1;
                else mine |= 1u << m;
            } else if (!taken(i, m)) {
                const double wi = w[i];
                const double* li = Lp + (int64_t)i * pitch;
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                int q = 0;
                for (; q + 3 < j; q += 4) {
                    s0 += li[q] * lp[q];
                    s1 += li[q + 1] * lp[q + 1];
                    s2 += li[q + 2] * lp[q + 2];
                    s3 += li[q + 3] * lp[q + 3];
                }
                for (; q < j; ++q) s0 += li[q] * lp[q];
                const double s = wi - ((s0 + s1) + (s2 + s3));
                l = s * inv;
                l = fma(inv, fma(-l, piv, s), l);  // s / piv
                d[i] -= l * l;
            }
            Lc[(int64_t)(k0 + j) * n + i] = l;
            Lp[(int64_t)i * pitch + j] = l;
        }
    }
    __syncthreads();
    const bool stop = j < b || k0 + j >= maxr;
    int bad = 0;
    for (int i = tid, m = 0; i < n; i += T, ++m) {
        const bool u = taken(i, m);
        if (!WIDE) {
            dg[i] = d[i];
            used[i] = u;
        }
        // indefinite if a remaining diagonal entry is clearly negative
        if (stop && !u && d[i] < -1e3 * tol * dmax0) bad = 1;
    }
    if (bad) s_bad = 1;
    // the panel for the trailing update; columns past its last pivot add nothing to it
    if (!stop)
        for (int e = tid; e < n * width; e += T) {
            const int i = e / width, c = e - i * width;
            Lg[e] = c < j ? Lp[(int64_t)i * pitch + c] : 0.0;
        }
    __syncthreads();
    if (tid == 0) {
        st->dmax0 = dmax0;
        st->k = k0 + j;
        st->stop = stop ? 1 : 0;
        st->bad = s_bad;
        st->active = stop ? 0 : 1;
        if (host) *host = *st;
    }
}

// Ct[i][mu] = Lc[i][mu] for i < rank and mu < n (rank = info[2 c]), else 0;
// sign[i] = 1 when sign is given (single cluster).
__global__ void k_factor_pad(const double* __restrict__ Lc, int64_t strideL, int64_t n, const int* __restrict__ info,
                             double* __restrict__ Ct, int64_t strideCt, int64_t npad, int64_t opad,
                             double* __restrict__ sign, const int* __restrict__ active, int64_t known_rank) {
    const int cl = blockIdx.y;
    if (active && active[cl] == 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= opad * npad) return;
    const int64_t rank = info ? info[2 * cl] : known_rank;
    const int64_t i = e / npad, mu = e % npad;
    Ct[cl * strideCt + e] = (i < rank && mu < n) ? Lc[cl * strideL + i * n + mu] : 0.0;
    if (sign && mu == 0) sign[i] = 1.0;
}

// Kp[c][e] += sum_s P[c][s][e] in split order (deterministic split-K reduction).
__global__ void k_sum_splits(const double* __restrict__ P, int splits, int64_t nn, double* __restrict__ Kp,
                             const int* __restrict__ active) {
    const int c = blockIdx.y;
    if (active && active[c] == 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nn) return;
    const double* src = P + (int64_t)c * splits * nn + e;
    double s = 0.0;
    for (int k = 0; k < splits; ++k) s += src[(int64_t)k * nn];
    Kp[(int64_t)c * nn + e] += s;
}

// K of one chunk of rows straight from its partial products: K[mu][nu] = K[nu][mu] =
// sum_s P[c][s][min][max] in split order, eight loads at a time.
__global__ void k_sum_splits_symmetric(const double* __restrict__ P, int splits, int64_t ldk, int64_t n,
                                       double* __restrict__ K, int64_t strideK, const int* __restrict__ active) {
    const int c = blockIdx.y;
    if (active && active[c] == 0) return;
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * n) return;
    const int64_t mu = e / n, nu = e % n;
    if (mu > nu) return;
    const double* src = P + (int64_t)c * splits * ldk * ldk + mu * ldk + nu;
    double s = 0.0;
#pragma unroll 8
    for (int k = 0; k < splits; ++k) s += src[(int64_t)k * ldk * ldk];
    K[c * strideK + e] = s;
    K[c * strideK + nu * n + mu] = s;
}

constexpr int kMaxDevices = 64;
constexpr int kPivotSmem = 200 * 1024;
std::mutex g_jk_mutex;
bool g_jk_configured[kMaxDevices] = {};

__global__ void k_scale_columns(const double* __restrict__ X, double* __restrict__ Xs, int64_t rows, int64_t ld,
                                int opad, const double* __restrict__ sign) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= rows * ld) return;
    Xs[e] = X[e] * sign[(e % ld) % opad];
}

}  // namespace

cudaError_t coulomb_build(const JkPlan& p, const double* D, int64_t strideD, double scale, double* J, int64_t strideJ,
                          double* work, cudaStream_t stream) {
    // work per cluster: Dw (ntiles*4096) | c (naux) | Jt (ntiles*4096)
    const int64_t nelem = p.ntiles * 4096;
    const int64_t sw = coulomb_work_doubles(p);
    double* Dw = work;
    double* c = work + nelem;
    double* Jt = c + ((p.naux + 1) / 2) * 2;
    const unsigned cnt = (unsigned)p.count;
    k_pack_density<<<dim3((unsigned)((nelem + 255) / 256), cnt), 256, 0, stream>>>(D, strideD, scale, p.n, p.nt, Dw, sw,
                                                                                   p.active);
    k_coulomb_charges<<<dim3(p.naux, cnt), 512, 0, stream>>>(p.Btab, p.B, p.ldb, nelem, Dw, c, sw, p.active);
    if (p.count == 1) {
        cudaMemsetAsync(Jt, 0, sizeof(double) * nelem, stream);
    } else {
        cudaMemset2DAsync(Jt, sizeof(double) * sw, 0, sizeof(double) * nelem, p.count, stream);
    }
    dim3 grid((unsigned)((nelem / 2 + 255) / 256), (p.naux + kJSlab - 1) / kJSlab, cnt);
    k_coulomb_assemble<<<grid, 256, 0, stream>>>(p.Btab, p.B, p.ldb, nelem, p.naux, c, Jt, sw, p.active);
    const int64_t nn = p.n * p.n;
    k_unpack_tiles<<<dim3((unsigned)((nn + 255) / 256), cnt), 256, 0, stream>>>(Jt, sw, p.n, p.nt, J, strideJ, p.active);
    return cudaGetLastError();
}

int64_t coulomb_work_doubles(const JkPlan& p) { return 2 * p.ntiles * 4096 + ((p.naux + 1) / 2) * 2; }

cudaError_t fitted_charges(const JkPlan& p, const double* D, double* d, double* work, cudaStream_t stream) {
    const int64_t nelem = p.ntiles * 4096;
    k_pack_density<<<dim3((unsigned)((nelem + 255) / 256), 1), 256, 0, stream>>>(D, 0, 1.0, p.n, p.nt, work, 0,
                                                                                 nullptr);
    k_coulomb_charges<<<dim3(p.naux, 1), 512, 0, stream>>>(nullptr, p.B, p.ldb, nelem, work, d, 0, nullptr);
    return cudaGetLastError();
}

// The SYRK's CTA tile: 64 x 64 with 2 stages of 32-wide k slices (tile 5).
constexpr int kSyrkTile = 5;

int syrk_splits(int64_t npad, int count) {
    const int bm = kTileShapes[kSyrkTile][0], bn = kTileShapes[kSyrkTile][1];
    const int64_t mt = (npad + bm - 1) / bm, nt = (npad + bn - 1) / bn;
    int64_t upper = 0;
    for (int64_t i = 0; i < mt; ++i)
        for (int64_t j = 0; j < nt; ++j)
            if (i * bm <= j * bn + bn - 1) ++upper;
    const int64_t ctas = upper * std::max(1, count);
    // enough CTAs for many waves: the tail of a last partial wave cost up to 13 %
    // of an FP64 K build at (H2O)64 with two splits
    const int64_t want = 12 * 148;
    int s = (int)std::min<int64_t>(32, (want + ctas - 1) / ctas);
    while (s > 1 && (int64_t)s * std::max(1, count) > 65535) --s;
    return std::max(1, s);
}

int64_t syrk_partial_doubles(int64_t npad, int count) {
    const int s = syrk_splits(npad, count);
    return s > 1 ? (int64_t)s * std::max(1, count) * npad * npad : 0;
}

namespace {
template <int XBN>
cudaError_t launch_half_as(const JkPlan& p, int q0, int qc, const double* Ct, int64_t strideCt, int64_t npad, double* X,
                           int64_t ldx, int64_t strideX, int opad, int transposed, cudaStream_t stream) {
    dim3 grid((opad + XBN - 1) / XBN, (unsigned)(((npad + XBM - 1) / XBM) * p.count), qc);
    k_exchange_half<XBN><<<grid, HalfShape<XBN>::THREADS, HalfShape<XBN>::SMEM, stream>>>(
        p.Btab, p.B, p.ldb, q0, p.nt, Ct, npad, strideCt, (int)p.n, (int)npad, X, ldx, strideX, opad, p.active, transposed);
    return cudaGetLastError();
}

cudaError_t launch_half(const JkPlan& p, int q0, int qc, const double* Ct, int64_t strideCt, int64_t npad, double* X,
                        int64_t ldx, int64_t strideX, int opad, int transposed, cudaStream_t stream) {
    // the least padded width; on a tie the wider of 64 and 32, then 80 and 48
    int best = 64;
    for (int w : {32, 80, 48})
        if ((opad + w - 1) / w * w < (opad + best - 1) / best * best) best = w;
    auto run = best == 32 ? launch_half_as<32> : best == 48 ? launch_half_as<48> : best == 80 ? launch_half_as<80>
                                                                                             : launch_half_as<64>;
    return run(p, q0, qc, Ct, strideCt, npad, X, ldx, strideX, opad, transposed, stream);
}
}  // namespace

cudaError_t exchange_build_fp64(const JkPlan& p, const double* Ct, int64_t strideCt, int opad, const double* sign,
                                double* K, int64_t strideK, double* Kp, double* X, double* Xs, double* partial,
                                int qchunk, cudaStream_t stream) {
    const int64_t npad = (int64_t)p.nt * 64;
    if (sign != nullptr && p.count != 1) return cudaErrorInvalidValue;
    cudaError_t e = jk_configure();
    if (e != cudaSuccess) return e;
    const int splits_wanted = partial ? syrk_splits(npad, p.count) : 1;
    const bool direct = qchunk >= p.naux && splits_wanted > 1;  // one chunk: no running sum in Kp
    if (!direct) cudaMemsetAsync(Kp, 0, sizeof(double) * npad * npad * p.count, stream);
    const int64_t strideX = npad * (int64_t)qchunk * opad;
    for (int q0 = 0; q0 < p.naux; q0 += qchunk) {
        const int qc = (p.naux - q0 < qchunk) ? p.naux - q0 : qchunk;
        const int64_t ldx = (int64_t)qc * opad;
        e = launch_half(p, q0, qc, Ct, strideCt, npad, X, ldx, strideX, opad, 0, stream);
        if (e != cudaSuccess) return e;
        const double* Xb = X;
        if (sign != nullptr) {
            const int64_t tot = npad * ldx;
            k_scale_columns<<<(unsigned)((tot + 255) / 256), 256, 0, stream>>>(X, Xs, npad, ldx, opad, sign);
            Xb = Xs;
        }
        GemmArgs g{};
        g.M = g.N = (int)p.n;
        g.K = (int)ldx;
        g.A = X;
        g.lda = ldx;
        g.B = Xb;
        g.ldb = ldx;
        g.C = Kp;
        g.ldc = npad;
        g.alpha = 1.0;
        g.beta = 1.0;
        g.kmode = 0;
        g.epi = 3;
        g.tile = kSyrkTile;
        g.strideA = g.strideB = strideX;
        g.strideC = npad * npad;
        g.active = p.active;
        const int splits = splits_wanted;
        if (splits > 1) {
            // partial products per split, then a fixed-order sum into Kp
            g.C = partial;
            g.beta = 0.0;
            g.splits = splits;
            e = dgemm_nt(g, p.count, stream);
            if (e != cudaSuccess) return e;
            if (direct) {
                k_sum_splits_symmetric<<<dim3((unsigned)((p.n * p.n + 255) / 256), (unsigned)p.count), 256, 0, stream>>>(
                    partial, splits, npad, p.n, K, strideK, p.active);
                return cudaGetLastError();
            }
            const int64_t nn2 = npad * npad;
            k_sum_splits<<<dim3((unsigned)((nn2 + 255) / 256), (unsigned)p.count), 256, 0, stream>>>(
                partial, splits, nn2, Kp, p.active);
        } else {
            e = dgemm_nt(g, p.count, stream);
        }
        if (e != cudaSuccess) return e;
    }
    const int64_t nn = p.n * p.n;
    k_symmetrize_upper<<<dim3((unsigned)((nn + 255) / 256), (unsigned)p.count), 256, 0, stream>>>(Kp, npad, p.n, K,
                                                                                                 strideK, p.active);
    return cudaGetLastError();
}

cudaError_t pivoted_cholesky(const double* D, int64_t strideD, int n, double tol, int maxr, double* Lc,
                             int64_t strideL, int* info, int count, const int* active, cudaStream_t stream) {
    const size_t smem = sizeof(double) * n + n + 16;
    if (smem > kPivotSmem) return cudaErrorInvalidValue;
    cudaError_t e = jk_configure();
    if (e != cudaSuccess) return e;
    k_pivoted_cholesky<<<count, 1024, smem, stream>>>(D, strideD, n, tol, maxr, Lc, strideL, info, active);
    return cudaGetLastError();
}

namespace {
// Pivots per panel and the pitch of its rows in shared memory (odd: rows of
// consecutive threads in different banks); in_smem 0: rows in global memory.
void pivot_panel(int n, int& width, int& pitch, int& in_smem) {
    if (n > kPivotThreads * kPivotRows) {
        width = pitch = 32;
        in_smem = 0;
        return;
    }
    const int room = (int)((kPivotSmem - sizeof(double) * (size_t)n) / (sizeof(double) * (size_t)n));
    in_smem = room >= 9;
    pitch = in_smem ? std::min((room & 1) ? room : room - 1, n | 1) : 32;
    width = in_smem ? std::max(1, std::min(pitch - 1, 256)) : 32;
    if (n == 1) width = 1;
}
}  // namespace

static_assert(sizeof(PivotState) <= kPivotMapped, "the mapped state's room");

size_t pivoted_cholesky_work_doubles(int n) {
    int width, pitch, in_smem;
    pivot_panel(n, width, pitch, in_smem);
    return (size_t)n * n + (size_t)n * std::max(width, pitch) + n + (n + 7) / 8 + 4;
}

cudaError_t pivoted_cholesky_blocked(const double* D, int n, double tol, int maxr, double* Lc, double* work,
                                     int64_t* rank, int* indefinite, cudaStream_t stream, void* mapped) {
    if (n < 1 || maxr < 1 || n > 1 << 20) return cudaErrorInvalidValue;
    cudaError_t e = jk_configure();
    if (e != cudaSuccess) return e;
    int width, pitch, in_smem;
    pivot_panel(n, width, pitch, in_smem);
    double* W = work;
    double* Lg = W + (size_t)n * n;
    double* d = Lg + (size_t)n * std::max(width, pitch);
    unsigned char* used = reinterpret_cast<unsigned char*>(d + n);
    PivotState* st = reinterpret_cast<PivotState*>(d + n + (n + 7) / 8);
    const bool wide = n > kPivotThreads * kPivotRows;
    const size_t smem = wide ? 0 : sizeof(double) * ((size_t)n + (in_smem ? (size_t)n * pitch : 0));
    const int threads = std::min(kPivotThreads, std::max(128, (n + 31) / 32 * 32));
    const int panels = (maxr + width - 1) / width;
    // A density's rank is its occupied orbitals, about a fifth of n: panels for 0.3 n are queued
    // before the first look at the state, the rest only when it has not stopped by then.
    int queued = 0, until = std::max(1, std::min(panels, (int)(0.3 * n / width) + 1));
    PivotState host{};
    for (;;) {
        for (; queued < until; ++queued) {
            if (queued > 0) {
                if (queued == 1) {
                    e = cudaMemcpyAsync(W, D, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, stream);
                    if (e != cudaSuccess) return e;
                }
                // W -= Lp Lp^T (skipped, CTA by CTA, once the factorisation has stopped)
                GemmArgs g{};
                g.M = g.N = n;
                g.K = width;
                g.A = g.B = Lg;
                g.lda = g.ldb = width;
                g.C = W;
                g.ldc = n;
                g.alpha = -1.0;
                g.beta = 1.0;
                g.kmode = 0;
                g.epi = 0;
                g.tile = 5;
                g.active = &st->active;
                e = dgemm_nt(g, 1, stream);
                if (e != cudaSuccess) return e;
            }
            (wide ? k_pc_panel<true> : k_pc_panel<false>)<<<1, threads, smem, stream>>>(
                queued == 0 ? D : W, n, tol, maxr, Lc, Lg, width, pitch, in_smem, d, used, queued == 0 ? 1 : 0, st,
                queued + 1 == until ? static_cast<PivotState*>(mapped) : nullptr);
        }
        e = mapped ? cudaSuccess : cudaMemcpyAsync(&host, st, sizeof(host), cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return e;
        if (mapped) std::memcpy(&host, mapped, sizeof(host));
        if (host.stop || queued >= panels) break;
        until = panels;
    }
    *rank = host.k;
    *indefinite = host.bad;
    return cudaGetLastError();
}

cudaError_t factor_pad(const double* Lc, int64_t strideL, int64_t n, const int* info, double* Ct, int64_t strideCt,
                       int64_t npad, int64_t opad, double* sign, int count, const int* active, cudaStream_t stream,
                       int64_t rank) {
    k_factor_pad<<<dim3((unsigned)((opad * npad + 255) / 256), (unsigned)count), 256, 0, stream>>>(
        Lc, strideL, n, info, Ct, strideCt, npad, opad, sign, active, rank);
    return cudaGetLastError();
}

cudaError_t half_transform_t(const JkPlan& p, const double* Ct, int opad, int q0, int qc, double* Xt,
                             cudaStream_t stream) {
    if (p.count != 1) return cudaErrorInvalidValue;
    cudaError_t e = jk_configure();
    if (e != cudaSuccess) return e;
    JkPlan all = p;
    all.active = nullptr;
    return launch_half(all, q0, qc, Ct, 0, (int64_t)p.nt * 64, Xt, 0, 0, opad, 1, stream);
}

cudaError_t jk_configure() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_jk_mutex);
    if (g_jk_configured[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(k_exchange_half<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, HalfShape<32>::SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_exchange_half<48>, cudaFuncAttributeMaxDynamicSharedMemorySize, HalfShape<48>::SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_exchange_half<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, HalfShape<64>::SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_exchange_half<80>, cudaFuncAttributeMaxDynamicSharedMemorySize, HalfShape<80>::SMEM);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_pivoted_cholesky, cudaFuncAttributeMaxDynamicSharedMemorySize, kPivotSmem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_pc_panel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPivotSmem);
    if (e != cudaSuccess) return e;
    g_jk_configured[dev] = true;
    return dgemm_configure();
}

}  // namespace hf
