// The {111}<110> slip family in crystal axes.
//
// In crystal axes the Schmid tensor of each of the 12 FCC systems is
// 1/sqrt(6) times a diagonal difference plus or minus the two shears that
// share the index z left out of that difference (z is the zero of the slip
// direction b).  With the deviatoric stress s written as
//   y = (s0/sqrt12, s1/2, s2/sqrt12, s3/sqrt12, s4/sqrt12)
// (s in the 6-vector basis, crystal axes) every resolved shear is a sum of
// entries of y with coefficients 0, +-1, +-2, and for each z there are four:
//   D_z +- (a + b),  D_z +- (a - b),
//   z = 0: D = y0 - y1,  a = y4, b = y3     (shears 01, 02)
//   z = 1: D = -y0 - y1, a = y4, b = y2     (shears 01, 12)
//   z = 2: D = -2 y0,    a = y3, b = y2     (shears 02, 12)
// The 12 resolved shears take 21 additions instead of 60 multiply-adds with
// stored Schmid vectors, the strain rate 32 operations instead of 60, and the
// 5 x 5 tangent about 40 additions instead of 240 multiply-adds, with nothing
// to load.
//
// The Newton step runs on y.  U maps it to sample axes (s_sample = U y: the
// rotation's deviatoric block with its columns scaled), and the residual and
// the matrices are transformed by the same U:
//   x_y = U^T x,  P_y = U^T (S_g + S0) U,  S0_y = U^T S0 U,
// so that M_y dy = x_y is the sample-axes Newton step in other variables.
// The crystal is cubic (three elastic constants), so its pressure part
// decouples: it is carried as the scalar s5 with the constant P55.
//
// Norms: |s|^2 = 12 (y0^2 + y2^2 + y3^2 + y4^2) + 4 y1^2 + s5^2, and for a
// dual vector x_y the reciprocal weights.
//
// An RVE whose slip table is this family (in any order and with any signs)
// and whose exponent is integral runs this form (RveDesc::fcc).  Its array
// `sch` then holds, instead of the 60 Schmid components, the 60 columns
//   0..24  U[i][c] at 5 i + c      25..39 P_y   (packed upper triangle)
//   40..54 S0_y                    55..59 y of the current stress,
// `sigp` the penultimate stress as (y, s5), and `itau` the reciprocal CRSS
// in canonical order: column 2 c + (resolved shear < 0) of canonical system
// c = 4 z + {0: D + (a + b), 1: D - (a + b), 2: D + (a - b), 3: D - (a - b)}.
#pragma once
#include "voce_dev.cuh"

#define FCC_U 0
#define FCC_P 25
#define FCC_S0 40
#define FCC_Y 55

// packed upper-triangle index of a symmetric 5x5
__host__ __device__ __forceinline__ constexpr int sym5(int i, int j)
{
    return i <= j ? i * 5 - (i * (i - 1)) / 2 + (j - i) : j * 5 - (j * (j - 1)) / 2 + (i - j);
}

// weight of y_c^2 in |s|^2
__host__ __device__ __forceinline__ constexpr double fcc_w2(int c) { return c == 1 ? 4.0 : 12.0; }

// |s|^2 of a deviatoric y
template <typename T>
__device__ __forceinline__ T fcc_norm2(const T (&y)[5])
{
    const T a = y[0] * y[0] + y[2] * y[2] + y[3] * y[3] + y[4] * y[4];
    return T(12) * a + T(4) * (y[1] * y[1]);
}

// |x|^2 of a dual vector
template <typename T>
__device__ __forceinline__ T fcc_dual2(const T (&x)[5])
{
    const T a = x[0] * x[0] + x[2] * x[2] + x[3] * x[3] + x[4] * x[4];
    return T(1.0 / 12.0) * a + T(0.25) * (x[1] * x[1]);
}

// the four resolved shears of family Z
template <int Z, typename T>
__device__ __forceinline__ void fcc_rss(const T (&y)[5], T (&c)[4])
{
    const T D = Z == 0 ? y[0] - y[1] : Z == 1 ? -y[0] - y[1] : T(-2) * y[0];
    const T a = Z == 2 ? y[3] : y[4], b = Z == 0 ? y[3] : y[2];
    const T u = a + b, w = a - b;
    c[0] = D + u;
    c[1] = D - u;
    c[2] = D + w;
    c[3] = D - w;
}

// E += sum over family Z of g_k A_k (dual vector)
template <int Z, typename T>
__device__ __forceinline__ void fcc_edot(const T (&g)[4], T (&E)[5])
{
    const T G = (g[0] + g[1]) + (g[2] + g[3]);
    const T gu = g[0] - g[1], gw = g[2] - g[3];
    const T a = gu + gw, b = gu - gw;
    if (Z == 0) {
        E[0] = G;
        E[1] = -G;
        E[4] = a;
        E[3] = b;
    } else if (Z == 1) {
        E[0] -= G;
        E[1] -= G;
        E[4] += a;
        E[2] = b;
    } else {
        E[0] = fma(T(-2), G, E[0]);
        E[3] += a;
        E[2] += b;
    }
}

// J += sum over family Z of h_k A_k A_k^T (packed upper triangle); the
// families in order 0, 1, 2
template <int Z, typename T>
__device__ __forceinline__ void fcc_tangent(const T (&h)[4], T (&J)[15])
{
    const T pu = h[0] + h[1], pw = h[2] + h[3], mu = h[0] - h[1], mw = h[2] - h[3];
    const T s = pu + pw, dl = pu - pw, a = mu + mw, b = mu - mw;   // DD = aa = bb, ab, Da, Db
    if (Z == 0) {
        J[sym5(0, 0)] = s;
        J[sym5(0, 1)] = -s;
        J[sym5(3, 3)] = s;
        J[sym5(4, 4)] = s;
        J[sym5(0, 4)] = a;
        J[sym5(1, 4)] = -a;
        J[sym5(0, 3)] = b;
        J[sym5(1, 3)] = -b;
        J[sym5(3, 4)] = dl;
    } else if (Z == 1) {
        J[sym5(0, 0)] += s;
        J[sym5(0, 1)] += s;
        J[sym5(1, 1)] = J[sym5(0, 0)];
        J[sym5(4, 4)] += s;
        J[sym5(2, 2)] = s;
        J[sym5(0, 4)] -= a;
        J[sym5(1, 4)] -= a;
        J[sym5(0, 2)] = -b;
        J[sym5(1, 2)] = -b;
        J[sym5(2, 4)] = dl;
    } else {
        J[sym5(0, 0)] = fma(T(4), s, J[sym5(0, 0)]);
        J[sym5(3, 3)] += s;
        J[sym5(2, 2)] += s;
        J[sym5(0, 3)] = fma(T(-2), a, J[sym5(0, 3)]);
        J[sym5(0, 2)] = fma(T(-2), b, J[sym5(0, 2)]);
        J[sym5(2, 3)] = dl;
    }
}

// One family of the flow rule (constitutive.c:126-194) in FP64, without
// gam0: g_k = |r|^n sign(r), and with JAC the tangent's h_k = |r|^(n-1)/tau
// (times gam0 n it is d gdot/d rss).
template <int Z, bool JAC>
__device__ __forceinline__ void fcc_flow_family(const RveDesc &d, long long v, const double (&y)[5],
                                                double (&E)[5], double (&J)[15])
{
    double c[4], g[4], h[4];
    fcc_rss<Z, double>(y, c);
    const int e = d.ipow_n - 1;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int neg = __double2hiint(c[k]) < 0;
        const double it = __ldg(d.itau + (long long)(2 * (4 * Z + k) + neg) * d.nv + v);
        const double r = c[k] * it;
        const double p = pow_abs_e(fabs(r), e);
        g[k] = p * r;
        if (JAC) h[k] = p * it;
    }
    fcc_edot<Z, double>(g, E);
    if (JAC) fcc_tangent<Z, double>(h, J);
}

template <bool JAC>
__device__ __forceinline__ void fcc_flow(const RveDesc &d, long long v, const double (&y)[5], double (&E)[5],
                                         double (&J)[15])
{
    fcc_flow_family<0, JAC>(d, v, y, E, J);
    fcc_flow_family<1, JAC>(d, v, y, E, J);
    fcc_flow_family<2, JAC>(d, v, y, E, J);
}

// LDL^T of the symmetric positive definite 5x5 M (packed upper triangle, in
// place): M(j, i) becomes L(i, j) for i > j, M(j, j) the pivot's reciprocal
__device__ __forceinline__ void fcc_factor(double (&M)[15])
{
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const double di = rcp_nr(M[sym5(j, j)]);
        double w[5];
#pragma unroll
        for (int i = j + 1; i < 5; ++i) {
            w[i] = M[sym5(j, i)];
            M[sym5(j, i)] = w[i] * di;
        }
#pragma unroll
        for (int i = j + 1; i < 5; ++i)
#pragma unroll
            for (int k = i; k < 5; ++k) M[sym5(i, k)] = fma(-M[sym5(j, i)], w[k], M[sym5(i, k)]);
        M[sym5(j, j)] = di;
    }
}

template <typename T>
__device__ __forceinline__ void fcc_solve(const T (&M)[15], T (&b)[5])
{
#pragma unroll
    for (int i = 1; i < 5; ++i)
#pragma unroll
        for (int k = 0; k < i; ++k) b[i] = fma(-M[sym5(k, i)], b[k], b[i]);
#pragma unroll
    for (int i = 0; i < 5; ++i) b[i] *= M[sym5(i, i)];
#pragma unroll
    for (int i = 3; i >= 0; --i)
#pragma unroll
        for (int k = i + 1; k < 5; ++k) b[i] = fma(-M[sym5(i, k)], b[k], b[i]);
}

// a column read the compiler may not merge with an earlier one of the same
// address: reading again (from L1) where keeping the value would cost registers
__device__ __forceinline__ double reread(const double *a)
{
    double x;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(x) : "l"(a));
    return x;
}

// itau column of system k (file order), direction f
__device__ __forceinline__ int itau_col(const RveDesc &d, int k, int f)
{
    return d.fcc ? 2 * d.canon[k] + (f ^ d.flip[k]) : 2 * k + f;
}
