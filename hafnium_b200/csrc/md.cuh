// Device McMurchie–Davidson building blocks, FP64 throughout.
//
// Boys function: Taylor expansion about the nearest point of a 0.05-spaced grid
// on [0, 36) (8 terms, |dT| <= 0.025, truncation below 4e-18 relative), then the
// downward recursion F_{n-1} = (2T F_n + e^{-T}) / (2n - 1); above the grid,
// F_0 = sqrt(pi/T)/2 and the upward recursion, as the reference's special.rs:34-51
// does above max(35, 2n). The grid values come from the reference's series
// (special.rs:67-81) evaluated on the host.
//
// Hermite Coulomb integrals R_tuv (coulomb.rs:162-215): the downward recursion
// in n is done in place in one tetrahedral array, updating total orders from
// the highest down, so R^{n+1} values are still present when R^n needs them.
//
// Spherical functions use the sphere-normalised real solid harmonics of
// cartesian.rs:93-110 (p ordered x, y, z). An auxiliary primitive
// S_lm(r) exp(-q r^2) expands into Hermite Gaussians of degree exactly l with
// coefficients (2q)^-l times the Cartesian coefficients of S_lm (Hobson's
// theorem), so its side of the contraction needs no E-coefficients.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hf {

constexpr int kMaxOrbL = 2;   // cc-pVDZ / def2-SVP / STO-3G for H-Ne
constexpr int kMaxAuxL = 4;   // def2-universal-jkfit for H-Ne
constexpr int kMaxOrbContr[3] = {3, 2, 1};  // general contractions per l (cc-pVDZ O)
constexpr int kBoysTerms = 8;
// one order more than the integrals need, for their first derivatives
constexpr int kBoysOrders = 2 * kMaxOrbL + kMaxAuxL + 1 + kBoysTerms;  // 17
constexpr double kBoysStep = 0.05;
constexpr double kBoysTmax = 36.0;
constexpr int kBoysGrid = 721;  // T = 0 .. 36 inclusive

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int nsph(int l) { return 2 * l + 1; }
// Number of (t,u,v) with t+u+v <= L.
__host__ __device__ constexpr int ntet(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
// Tetrahedral index of (t,u,v): shells of total order s, then u+v, then v.
__host__ __device__ constexpr int tet(int t, int u, int v) {
    return (t + u + v) * (t + u + v + 1) * (t + u + v + 2) / 6 + (u + v) * (u + v + 1) / 2 + v;
}
// Cartesian component c of angular momentum l (x^l first, z^l last): exponents.
__host__ __device__ constexpr int cart_x(int l, int c) {
    int i = l, k = 0;
    for (; i >= 0; --i) {
        if (c < k + (l - i + 1)) return i;
        k += l - i + 1;
    }
    return 0;
}
__host__ __device__ constexpr int cart_y(int l, int c) {
    int i = l, k = 0;
    for (; i >= 0; --i) {
        if (c < k + (l - i + 1)) return (l - i) - (c - k);
        k += l - i + 1;
    }
    return 0;
}
__host__ __device__ constexpr int cart_z(int l, int c) { return l - cart_x(l, c) - cart_y(l, c); }

// Cartesian-to-spherical matrices for l = 0..4, row-major [2l+1][ncart(l)],
// concatenated; offsets c2s_offset(l).
__host__ __device__ constexpr int c2s_offset(int l) {
    int o = 0;
    for (int k = 0; k < l; ++k) o += nsph(k) * ncart(k);
    return o;
}
constexpr int kC2sSize = 1 + 9 + 30 + 70 + 135;

// Primitive pairs whose |c_a c_b| exp(-mu R_AB^2) falls below this contribute
// less than ~1e-15 to any (P|ab) and are skipped (the reference evaluates every
// primitive triple; the difference is far below its 1e-12 integral tolerance).
constexpr double kPairScreen = 1e-22;
constexpr int kMaxPrimPairs = 256;
constexpr double kPi = 3.14159265358979323846;
constexpr double kTwoPi52 = 34.98683665524972;  // 2 pi^(5/2)
// The matrices live in __constant__ memory of the translation unit that uses them.

// x / D, correctly rounded, by a multiplication with the rounded reciprocal and one correction
// (Markstein, IBM J. Res. Dev. 34, 111 (1990)): the residual x - q D of the first quotient is exact in
// one fused operation.
template <int D>
__device__ __forceinline__ double divide_by(double x) {
    if constexpr ((D & (D - 1)) == 0) {
        return x * (1.0 / D);
    } else {
        constexpr double r = 1.0 / D;
        const double q = __dmul_rn(x, r);
        return __fma_rn(__fma_rn(-q, (double)D, x), r, q);
    }
}
// The same with a divisor known at run time and its rounded reciprocal r = 1 / d.
__device__ __forceinline__ double divide_by(double x, double d, double r) {
    const double q = __dmul_rn(x, r);
    return __fma_rn(__fma_rn(-q, d, x), r, q);
}

template <int N>
struct BoysSteps {
    // v <- c_(N-1) + v d / N, N = from .. 1
    static __device__ __forceinline__ double taylor(const double* __restrict__ row, double v, double d) {
        if constexpr (N == 0) {
            return v;
        } else {
            const double c = __ldg(row + N - 1);
            const double w = N == 1 ? __fma_rn(v, d, c) : __dadd_rn(c, divide_by<N>(__dmul_rn(v, d)));
            return BoysSteps<N - 1>::taylor(row, w, d);
        }
    }
    // F[n - 1] = (2 T F[n] + e^-T) / (2 n - 1), n = N .. 1
    static __device__ __forceinline__ void down(double* F, double two_t, double et) {
        if constexpr (N > 0) {
            F[N - 1] = divide_by<2 * N - 1>(__fma_rn(two_t, F[N], et));
            BoysSteps<N - 1>::down(F, two_t, et);
        }
    }
};

// F_0..F_L at T. `table` is [kBoysGrid][kBoysOrders]. The serial chain is what bounds it: its
// divisions by constants are three operations each with the same rounding as a division (as divisions,
// seven in the Taylor sum and L in the recursion were most of a primitive triple's time). The metric's
// condition amplifies an ulp here to 1e-12 in J, so the values stay what they were, bit for bit.
// DIVIDE keeps the divisions in the source: with alpha r^2 inlined, the nuclear attraction's T is
// contracted into what surrounds it, and only the same source gave the same h.
template <int L, bool DIVIDE = false>
__device__ __forceinline__ void boys(double T, const double* __restrict__ table, double* F) {
    const double et = exp(-T);
    if (T < kBoysTmax) {
        const int j = __double2int_rn(T * (1.0 / kBoysStep));
        const double d = j * kBoysStep - T;  // T0 - T
        const double* row = table + j * kBoysOrders + L;
        // F_L(T) = sum_k F_{L+k}(T0) (T0 - T)^k / k!
        if constexpr (DIVIDE) {
            double v = __ldg(row + kBoysTerms - 1);
#pragma unroll
            for (int k = kBoysTerms - 1; k >= 1; --k) v = __ldg(row + k - 1) + v * d / k;
            F[L] = v;
#pragma unroll
            for (int n = L; n >= 1; --n) F[n - 1] = (2.0 * T * F[n] + et) / (2 * n - 1);
        } else {
            F[L] = BoysSteps<kBoysTerms - 1>::taylor(row, __ldg(row + kBoysTerms - 1), d);
            BoysSteps<L>::down(F, 2.0 * T, et);
        }
    } else {
        F[0] = 0.5 * sqrt(3.14159265358979323846 / T);
        const double inv2T = 0.5 / T;
#pragma unroll
        for (int n = 0; n < L; ++n) F[n + 1] = ((2 * n + 1) * F[n] - et) * inv2T;
    }
}

// 1 / (p + q) and 1 / sqrt(p + q) from one reciprocal square root: its square, corrected by one
// Newton step (the step's residual is one fused operation), is as good as a division (the derivative
// kernels; the integrals behind the fit keep their division's and root's exact rounding).
__device__ __forceinline__ void inverse_sum(double p, double q, double& inv, double& inv_sqrt) {
    const double s = p + q;
    inv_sqrt = rsqrt(s);
    inv = inv_sqrt * inv_sqrt;
    inv = fma(inv, fma(-s, inv, 1.0), inv);
}

// (2q)^-L from 1 / q.
template <int L>
__device__ __forceinline__ double half_power(double inv_q) {
    double v = 1.0;
#pragma unroll
    for (int k = 0; k < L; ++k) v *= 0.5 * inv_q;
    return v;
}

// R^0_tuv(alpha, X, Y, Z) for t+u+v <= L into R[tet(t,u,v)]. Up to L = 4 the
// recursion is unrolled so the table stays in registers; above, the loops are
// left rolled (the table lives in L1-resident local memory), which keeps the
// kernels compact and their compile time short.
template <int L, bool DIVIDE = false>
__device__ __forceinline__ void hermite_r(double alpha, double X, double Y, double Z,
                                          const double* __restrict__ btable, double* R) {
    double F[L + 1];
    boys<L, DIVIDE>(alpha * (X * X + Y * Y + Z * Z), btable, F);
    const double m2a = -2.0 * alpha;
    double pw[L + 1];
    pw[0] = 1.0;
#pragma unroll
    for (int k = 1; k <= L; ++k) pw[k] = pw[k - 1] * m2a;
    R[0] = pw[L] * F[L];
    if constexpr (L <= 4) {
#pragma unroll
        for (int n = L - 1; n >= 0; --n) {
#pragma unroll
            for (int s = L - n; s >= 1; --s)
#pragma unroll
                for (int t = s; t >= 0; --t)
#pragma unroll
                    for (int v = 0; v <= s - t; ++v) {
                        const int u = s - t - v;
                        double val;
                        if (t > 0) {
                            val = X * R[tet(t - 1, u, v)];
                            if (t > 1) val += (t - 1) * R[tet(t - 2, u, v)];
                        } else if (u > 0) {
                            val = Y * R[tet(t, u - 1, v)];
                            if (u > 1) val += (u - 1) * R[tet(t, u - 2, v)];
                        } else {
                            val = Z * R[tet(t, u, v - 1)];
                            if (v > 1) val += (v - 1) * R[tet(t, u, v - 2)];
                        }
                        R[tet(t, u, v)] = val;
                    }
            R[0] = pw[n] * F[n];
        }
    } else {
#pragma unroll 1
        for (int n = L - 1; n >= 0; --n) {
#pragma unroll 1
            for (int s = L - n; s >= 1; --s) {
                const int idx = s * (s + 1) * (s + 2) / 6;  // tet(s, 0, 0)
#pragma unroll 1
                for (int t = s; t >= 0; --t) {
                    const int r = s - t;  // u + v
#pragma unroll 1
                    for (int v = 0; v <= r; ++v) {
                        const int u = r - v;
                        double val;
                        if (t > 0) {
                            val = X * R[tet(t - 1, u, v)];
                            if (t > 1) val += (t - 1) * R[tet(t - 2, u, v)];
                        } else if (u > 0) {
                            val = Y * R[tet(t, u - 1, v)];
                            if (u > 1) val += (u - 1) * R[tet(t, u - 2, v)];
                        } else {
                            val = Z * R[tet(t, u, v - 1)];
                            if (v > 1) val += (v - 1) * R[tet(t, u, v - 2)];
                        }
                        R[idx + r * (r + 1) / 2 + v] = val;
                    }
                }
            }
            R[0] = pw[n] * F[n];
        }
    }
}

// One axis of the Hermite expansion of a primitive pair: E[i][j][t] for i<=LA,
// j<=LB+X, t<=i+j (hermite.rs:23-61, Helgaker 9.5.6/9.5.7).
template <int LA, int LB>
struct Hermite1D {
    double e[LA + 1][LB + 1][LA + LB + 1];
    __device__ __forceinline__ void build(double p, double e00, double xpa, double xpb) {
        const double h = 0.5 / p;
#pragma unroll
        for (int i = 0; i <= LA; ++i)
#pragma unroll
            for (int j = 0; j <= LB; ++j)
#pragma unroll
                for (int t = 0; t <= LA + LB; ++t) e[i][j][t] = 0.0;
        e[0][0][0] = e00;
#pragma unroll
        for (int i = 0; i < LA; ++i)
#pragma unroll
            for (int t = 0; t <= i + 1; ++t)
                e[i + 1][0][t] = (t > 0 ? h * e[i][0][t - 1] : 0.0) + xpa * (t <= i ? e[i][0][t] : 0.0) +
                                 (t + 1 <= i ? (t + 1) * e[i][0][t + 1] : 0.0);
#pragma unroll
        for (int i = 0; i <= LA; ++i)
#pragma unroll
            for (int j = 0; j < LB; ++j)
#pragma unroll
                for (int t = 0; t <= i + j + 1; ++t)
                    e[i][j + 1][t] = (t > 0 ? h * e[i][j][t - 1] : 0.0) +
                                     xpb * (t <= i + j ? e[i][j][t] : 0.0) +
                                     (t + 1 <= i + j ? (t + 1) * e[i][j][t + 1] : 0.0);
    }
};

}  // namespace hf
