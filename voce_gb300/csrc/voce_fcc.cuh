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
// c = 4 z + {0: D + (a + b), 1: D - (a + b), 2: D + (a - b), 3: D - (a - b)}
// (so do its float pairs); sgp32 and sgp_lo hold P_y's 15 float pairs, and in
// the mixed_nr32 form sch32 the 15 floats of S0_y.  The other arrays of the
// general Newton forms (sch_lo, sgp) stay allocated, because the footprint of
// an RVE does not depend on its slip table, but are not used.
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

// all three families: canonical system 4 z + k
template <typename T>
__device__ __forceinline__ void fcc_rss12(const T (&y)[5], T (&c)[12])
{
    T q[4];
    fcc_rss<0, T>(y, q);
    c[0] = q[0]; c[1] = q[1]; c[2] = q[2]; c[3] = q[3];
    fcc_rss<1, T>(y, q);
    c[4] = q[0]; c[5] = q[1]; c[6] = q[2]; c[7] = q[3];
    fcc_rss<2, T>(y, q);
    c[8] = q[0]; c[9] = q[1]; c[10] = q[2]; c[11] = q[3];
}
template <typename T>
__device__ __forceinline__ void fcc_edot12(const T (&g)[12], T (&E)[5])
{
    fcc_edot<0, T>({g[0], g[1], g[2], g[3]}, E);
    fcc_edot<1, T>({g[4], g[5], g[6], g[7]}, E);
    fcc_edot<2, T>({g[8], g[9], g[10], g[11]}, E);
}
template <typename T>
__device__ __forceinline__ void fcc_tangent12(const T (&h)[12], T (&J)[15])
{
    fcc_tangent<0, T>({h[0], h[1], h[2], h[3]}, J);
    fcc_tangent<1, T>({h[4], h[5], h[6], h[7]}, J);
    fcc_tangent<2, T>({h[8], h[9], h[10], h[11]}, J);
}

// |r[k]|^e by binary powering, out of line and through local memory: the
// loops of the twelve systems would sit between the hot instructions of e = 19
// (n = 20, the exponent of the inputs at hand; in line, its Newton kernels
// took 359 instead of 354 us in FP64, 216 instead of 213 in mixed_ir).  Other
// exponents pay for it and stay ahead of the general kernel: us per launch at
// 64^3, first 40 Green iterations, kb_nr -> this one, n = 10: FP64 1141 -> 498,
// mixed_ir 518 -> 300, mixed_nr32 131 -> 121; n = 20: 1047 -> 403, 428 -> 224,
// 121 -> 103; n = 25: 1258 -> 924 (FP64 solves its correction in FP64 above
// 20), 552 -> 318, 133 -> 124.
template <int N, typename T>
__device__ __noinline__ void fcc_pow_any(const T *r, int e, T *p)
{
    for (int k = 0; k < N; ++k) {
        T b = sizeof(T) == 4 ? (T)fabsf((float)r[k]) : (T)fabs((double)r[k]), q = T(1);
        for (int x = e; x; x >>= 1) {
            if (x & 1) q *= b;
            b *= b;
        }
        p[k] = q;
    }
}

// p[k] = |r[k]|^e, e = n - 1.  The exponent is tested once for all N, so that
// their loads and products stay in one straight run of instructions.
template <int N, typename T>
__device__ __forceinline__ void fcc_pow(const T (&r)[N], int e, T (&p)[N])
{
    if (e == 19) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const T a2 = r[k] * r[k], a4 = a2 * a2, a8 = a4 * a4, a16 = a8 * a8;
            p[k] = (a16 * a2) * (sizeof(T) == 4 ? (T)fabsf((float)r[k]) : (T)fabs((double)r[k]));
        }
    } else {
        T a[N], q[N];
#pragma unroll
        for (int k = 0; k < N; ++k) a[k] = r[k];
        fcc_pow_any<N, T>(a, e, q);
#pragma unroll
        for (int k = 0; k < N; ++k) p[k] = q[k];
    }
}

// One family of the flow rule (constitutive.c:126-194) in FP64, without
// gam0: g = |r|^n sign(r), and with JAC the tangent's h = |r|^(n-1)/tau
// (times gam0 n it is d gdot / d rss).
template <int Z, bool JAC>
__device__ __forceinline__ void fcc_flow_family(const RveDesc &d, long long v, const double (&y)[5],
                                                double (&E)[5], double (&J)[15])
{
    double r[4], it[4], p[4];
    fcc_rss<Z, double>(y, r);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int neg = __double2hiint(r[k]) < 0;
        it[k] = __ldg(d.itau + (long long)(2 * (4 * Z + k) + neg) * d.nv + v);
        r[k] *= it[k];
    }
    fcc_pow<4, double>(r, d.ipow_n - 1, p);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        r[k] *= p[k];
        if (JAC) p[k] *= it[k];
    }
    fcc_edot<Z, double>(r, E);
    if (JAC) fcc_tangent<Z, double>(p, J);
}

template <bool JAC>
__device__ __forceinline__ void fcc_flow(const RveDesc &d, long long v, const double (&y)[5], double (&E)[5],
                                         double (&J)[15])
{
    fcc_flow_family<0, JAC>(d, v, y, E, J);
    fcc_flow_family<1, JAC>(d, v, y, E, J);
    fcc_flow_family<2, JAC>(d, v, y, E, J);
}

// The strain rate of the mixed_ir form's FP64 steps (without gam0): fcc_flow
// without the tangent, |r|^20 by five products and the sign put on the high
// word.  Returns whether a ratio |r| reaches 60 (tested on the high word),
// where the float tangent could overflow.
__device__ __forceinline__ bool fcc_edot_fp64(const RveDesc &d, long long v, const double (&y)[5], double (&E)[5])
{
    double r[12], it[12];
    fcc_rss12<double>(y, r);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        const int neg = __double2hiint(r[k]) < 0;
        it[k] = __ldg(d.itau + (long long)(2 * k + neg) * d.nv + v);
    }
#pragma unroll
    for (int k = 0; k < 12; ++k) r[k] *= it[k];
    bool big = false;
#pragma unroll
    for (int k = 0; k < 12; ++k) big = big || (__double2hiint(r[k]) & 0x7fffffff) >= 0x404E0000;
    if (d.ipow_n == 20) {
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const double a2 = r[k] * r[k], a4 = a2 * a2, a5 = a4 * fabs(r[k]), a10 = a5 * a5, a20 = a10 * a10;
            r[k] = __hiloint2double(__double2hiint(a20) | (__double2hiint(r[k]) & (int)0x80000000), __double2loint(a20));
        }
    } else {
        double p[12];
        fcc_pow<12, double>(r, d.ipow_n - 1, p);
#pragma unroll
        for (int k = 0; k < 12; ++k) r[k] *= p[k];
    }
    fcc_edot12<double>(r, E);
    return big;
}

// The same family by family in one loop body, for the FP64 form, whose Newton
// loop is long: fewer instructions to wait for (128^3 3.94 -> 3.79 ms per
// launch; the mixed_ir form at 64^3 213 -> 218 us, so it keeps the run above)
__device__ __forceinline__ bool fcc_edot_fp64_loop(const RveDesc &d, long long v, const double (&y)[5], double (&E)[5])
{
    bool big = false;
#pragma unroll
    for (int c = 0; c < 5; ++c) E[c] = 0.0;
#pragma unroll 1
    for (int z = 0; z < 3; ++z) {
        const double D = (z == 0 ? y[0] : -y[0]) - (z == 2 ? y[0] : y[1]);
        const double a = z == 2 ? y[3] : y[4], b = z == 0 ? y[3] : y[2], u = a + b, w = a - b;
        double r[4] = {D + u, D - u, D + w, D - w};
        const double *tau = d.itau + (long long)(8 * z) * d.nv + v;
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] *= __ldg(tau + (long long)(2 * k + (__double2hiint(r[k]) < 0)) * d.nv);
#pragma unroll
        for (int k = 0; k < 4; ++k) big = big || (__double2hiint(r[k]) & 0x7fffffff) >= 0x404E0000;
        if (d.ipow_n == 20) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double a2 = r[k] * r[k], a4 = a2 * a2, a5 = a4 * fabs(r[k]), a10 = a5 * a5, a20 = a10 * a10;
                r[k] = __hiloint2double(__double2hiint(a20) | (__double2hiint(r[k]) & (int)0x80000000), __double2loint(a20));
            }
        } else {
            double p[4];
            fcc_pow<4, double>(r, d.ipow_n - 1, p);
#pragma unroll
            for (int k = 0; k < 4; ++k) r[k] *= p[k];
        }
        const double G = (r[0] + r[1]) + (r[2] + r[3]), gu = r[0] - r[1], gw = r[2] - r[3];
        const double ea = gu + gw, eb = gu - gw;
        if (z == 0) { E[0] = G; E[1] = -G; E[4] = ea; E[3] = eb; }
        else if (z == 1) { E[0] -= G; E[1] -= G; E[4] += ea; E[2] = eb; }
        else { E[0] = fma(-2.0, G, E[0]); E[3] += ea; E[2] += eb; }
    }
    return big;
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

// x = h + l, h rounded to nearest and l the signed remainder's 28 bits rounded
// to a float, so to 2^-49 of x while l is a normal float (|x| >= 2^-74).
// |x| < 2^128 (the callers' residual and ratio tests see to it).  With h
// truncated, to 2^-47, the Newton kernels took 1 % less (128^3 FP64 3836
// against 3789 us, 96^3 mixed_nr32 313 against 310), but h is also used alone,
// as the matrix of the single-precision steps.
__device__ __forceinline__ ff32 d2ff(double x)
{
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    ff32 r;
    r.h = d2f_rn(x);
    // 2^(exponent of x - 52) as a float, zero where that is below the floats
    const int e = (int)((hi >> 20) & 0x7ffu) - (1023 - 127) - 52;
    const float s = __uint_as_float((e > 0 ? (unsigned)e << 23 : 0u) | (hi & 0x80000000u));
    r.l = (float)((int)(lo << 3) >> 3) * s;
    return r;
}

// ---------------------------------------------------------------------------
// The same family in single precision and in float pairs, for the forms whose
// Newton runs on the FP32 pipe (VOCE_PREC_MIXED_IR's start, VOCE_PREC_MIXED_NR32)
// ---------------------------------------------------------------------------

// fcc_flow in single precision; false when a resolved-shear ratio is too large
// for |r|^n in single precision, or not a number
__device__ __forceinline__ bool fcc_flow_f32(const RveDesc &d, long long v, const float (&y)[5], float (&E)[5],
                                             float (&J)[15])
{
    float r[12], it[12], p[12];
    fcc_rss12<float>(y, r);
#pragma unroll
    for (int k = 0; k < 12; ++k) it[k] = __ldg(d.itau32 + (long long)(2 * k + (r[k] < 0.0f)) * d.nv + v);
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        r[k] *= it[k];
        ok = ok && fabsf(r[k]) < 60.0f;
    }
    fcc_pow<12, float>(r, d.ipow_n - 1, p);
#pragma unroll
    for (int k = 0; k < 12; ++k) { r[k] *= p[k]; p[k] *= it[k]; }
    fcc_edot12<float>(r, E);
    fcc_tangent12<float>(p, J);
    return ok;
}

// single-precision fcc_factor, the pivots' reciprocals as in ldlt_solve6f
__device__ __forceinline__ void fcc_factor(float (&M)[15])
{
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        float di, w[5];
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(di) : "f"(M[sym5(j, j)]));
#pragma unroll
        for (int i = j + 1; i < 5; ++i) {
            w[i] = M[sym5(j, i)];
            M[sym5(j, i)] = w[i] * di;
        }
#pragma unroll
        for (int i = j + 1; i < 5; ++i)
#pragma unroll
            for (int k = i; k < 5; ++k) M[sym5(i, k)] = fmaf(-M[sym5(j, i)], w[k], M[sym5(i, k)]);
        M[sym5(j, j)] = di;
    }
}

// sums of float pairs that stay unnormalised (a product renormalises first)
__device__ __forceinline__ ff32 ffs_add(ff32 a, ff32 b)
{
    ff32 r;
    float e;
    two_sum(a.h, b.h, r.h, e);
    r.l = e + (a.l + b.l);
    return r;
}
__device__ __forceinline__ ff32 ffs_neg(ff32 a)
{
    a.h = -a.h;
    a.l = -a.l;
    return a;
}
__device__ __forceinline__ ff32 ffs_sub(ff32 a, ff32 b) { return ffs_add(a, ffs_neg(b)); }
__device__ __forceinline__ ff32 ffs_sum(float a, float b)
{
    ff32 r;
    two_sum(a, b, r.h, r.l);
    return r;
}

// E += the strain-rate sums of family Z (as fcc_edot)
template <int Z>
__device__ __forceinline__ void fcc_edot_ff(const ff32 *g, ff32 (&E)[5])
{
    const ff32 G = ffs_add(ffs_add(g[0], g[1]), ffs_add(g[2], g[3]));
    const ff32 gu = ffs_sub(g[0], g[1]), gw = ffs_sub(g[2], g[3]);
    const ff32 ea = ffs_add(gu, gw), eb = ffs_sub(gu, gw);
    if (Z == 0) {
        E[0] = G;
        E[1] = ffs_neg(G);
        E[4] = ea;
        E[3] = eb;
    } else if (Z == 1) {
        E[0] = ffs_sub(E[0], G);
        E[1] = ffs_sub(E[1], G);
        E[4] = ffs_add(E[4], ea);
        E[2] = eb;
    } else {
        ff32 G2;
        G2.h = 2.0f * G.h;
        G2.l = 2.0f * G.l;
        E[0] = ffs_sub(E[0], G2);
        E[3] = ffs_add(E[3], ea);
        E[2] = ffs_add(E[2], eb);
    }
}

// a[k] := |a[k]|^e for n float pairs, out of line like fcc_pow_any
__device__ __noinline__ void fcc_ipow_any(ff32 *a, int n, int e)
{
    for (int k = 0; k < n; ++k) a[k] = ff_ipow(a[k].h < 0.0f ? ffs_neg(a[k]) : a[k], e);
}

// the strain rate (without gam0) as float pairs at the single-precision point
// y (the families in one loop body, as in fcc_jac_ff); false when a ratio
// leaves the float range
__device__ __forceinline__ bool fcc_flow_ff(const RveDesc &d, long long v, const float (&y)[5], ff32 (&E)[5])
{
    bool ok = true;
    const ff32 zero = {0.0f, 0.0f};
#pragma unroll
    for (int c = 0; c < 5; ++c) E[c] = zero;
#pragma unroll 1
    for (int z = 0; z < 3; ++z) {
        const ff32 D = ffs_sum(z == 0 ? y[0] : -y[0], z == 2 ? -y[0] : -y[1]);
        const float a = z == 2 ? y[3] : y[4], b = z == 0 ? y[3] : y[2];
        const ff32 u = ffs_sum(a, b), w = ffs_sum(a, -b);
        ff32 r[4] = {ffs_add(D, u), ffs_sub(D, u), ffs_add(D, w), ffs_sub(D, w)};
        float ih[4], il[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const long long col = (long long)(2 * (4 * z + k) + (r[k].h < 0.0f)) * d.nv + v;
            ih[k] = __ldg(d.itau32 + col);
            il[k] = __ldg(d.itau_lo + col);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            r[k] = ff_mul(ff_norm(r[k].h, r[k].l), ih[k], il[k]);
            ok = ok && fabsf(r[k].h) < 60.0f;
        }
        if (d.ipow_n == 20) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ff32 a2 = ff_mul(r[k], r[k].h, r[k].l), a4 = ff_mul(a2, a2.h, a2.l), a8 = ff_mul(a4, a4.h, a4.l);
                const ff32 a16 = ff_mul(a8, a8.h, a8.l), a20 = ff_mul(a16, a4.h, a4.l);
                r[k] = r[k].h < 0.0f ? ffs_neg(a20) : a20;
            }
        } else {
            ff32 q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = r[k];
            fcc_ipow_any(q, 4, d.ipow_n);
#pragma unroll
            for (int k = 0; k < 4; ++k) r[k] = r[k].h < 0.0f ? ffs_neg(q[k]) : q[k];
        }
        if (z == 0) fcc_edot_ff<0>(r, E);
        else if (z == 1) fcc_edot_ff<1>(r, E);
        else fcc_edot_ff<2>(r, E);
    }
    return ok;
}

// Single-precision Newton from the Green iterate y: steps down to a relative
// update of sqrt(tol) (at most `most`), the last step's factored matrix left
// in L.  False when a ratio leaves the float range, a value is not finite or
// the steps run out.
__device__ __forceinline__ bool fcc_newton_f32(const RveDesc &d, long long v, const float (&cc)[5], float thr,
                                               int most, float (&y)[5], const float (&P)[15], float (&L)[15], int &it)
{
    const float dtg = (float)d.dt * d.gam0f[0], dtgn = dtg * d.nrsf[0];
    for (int p = 0; p < most; ++p) {
        float E[5], x[5];
        if (!fcc_flow_f32(d, v, y, E, L)) return false;
#pragma unroll
        for (int c = 0; c < 5; ++c) x[c] = fmaf(dtg, E[c], cc[c]);
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = i; j < 5; ++j) {
                const float q = P[sym5(i, j)];
                x[i] = fmaf(q, y[j], x[i]);
                if (i != j) x[j] = fmaf(q, y[i], x[j]);
                L[sym5(i, j)] = fmaf(dtgn, L[sym5(i, j)], q);
            }
        fcc_factor(L);
        fcc_solve<float>(L, x);
        const float dn = fcc_norm2<float>(x);
#pragma unroll
        for (int c = 0; c < 5; ++c) y[c] -= x[c];
        ++it;
        if (!(dn <= 3.0e38f)) return false;   // not finite
        if (dn < thr) return true;
    }
    return false;
}

// One step on the float-float residual (residual_ff's accuracy, about 48
// bits) from the single-precision point y with the factors L; x receives the
// correction.  False when a ratio leaves the float range or the correction is
// not finite.
__device__ __forceinline__ bool fcc_step_ff(const RveDesc &d, long long v, const float (&y)[5], const double (&cc)[5],
                                            const float (&P)[15], const float (&L)[15], float dtgh, float dtgl,
                                            float (&x)[5])
{
    ff32 E[5], t[5];
    if (!fcc_flow_ff(d, v, y, E)) return false;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const ff32 c = d2ff(cc[i]);
        t[i] = ffs_add(c, ff_mul(ff_norm(E[i].h, E[i].l), dtgh, dtgl));
    }
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = i; j < 5; ++j) {
            const float q = P[sym5(i, j)], ql = __ldg(d.sgp_lo + (long long)sym5(i, j) * d.nv + v);
            ff_acc(t[i], q, ql, y[j]);
            if (i != j) ff_acc(t[j], q, ql, y[i]);
        }
#pragma unroll
    for (int i = 0; i < 5; ++i) x[i] = t[i].h + t[i].l;
    fcc_solve<float>(L, x);
    return finite_f((x[0] + x[1]) + (x[2] + x[3]) + x[4]);
}

// ---------------------------------------------------------------------------
// The correction of the FP64 Newton step, M dy = x with the exact tangent, in
// float pairs.  Its operands come in to 2^-49 (d2ff), a product or a step of
// the elimination rounds to about 2^-44, and the solve multiplies that by the
// condition of M, which the power law makes large: the correction is less
// accurate than an FP64 solve.  It only chooses the next iterate.  The
// residual that the iterate is measured by, the flow rule, the stop test and
// the iterate are FP64, so a correction off by a part in 10^9 moves the next
// iterate by 10^-9 of a step, and the last step is below 10^-7 of the stress.
// Against a 64-bit solve over the measured cases the stresses are no further
// off than with the FP64 solve (4.2e-15, 4.5e-15).
// ---------------------------------------------------------------------------
__device__ __forceinline__ ff32 ffs_norm(ff32 a) { return ff_norm(a.h, a.l); }
__device__ __forceinline__ ff32 ffs_mul(ff32 a, ff32 b) { return ff_mul(a, b.h, b.l); }

// 1 / a: the hardware's approximate reciprocal and one Newton-Raphson step
__device__ __forceinline__ ff32 ff_rcp(ff32 a)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a.h));
    const float e = fmaf(-a.l, r, fmaf(-a.h, r, 1.0f));
    return ff_norm(r, r * e);
}

// J += the tangent of family z from its four h (see fcc_tangent)
__device__ __forceinline__ void fcc_tangent_ff(int z, const ff32 (&h)[4], ff32 (&J)[15])
{
    const ff32 pu = ffs_add(h[0], h[1]), pw = ffs_add(h[2], h[3]);
    const ff32 mu = ffs_sub(h[0], h[1]), mw = ffs_sub(h[2], h[3]);
    const ff32 s = ffs_add(pu, pw), dl = ffs_sub(pu, pw), a = ffs_add(mu, mw), b = ffs_sub(mu, mw);
    auto twice = [](ff32 x) { x.h *= 2.0f; x.l *= 2.0f; return x; };
    auto add = [&](int i, int j, ff32 x) { J[sym5(i, j)] = ffs_add(J[sym5(i, j)], x); };
    auto sub = [&](int i, int j, ff32 x) { J[sym5(i, j)] = ffs_sub(J[sym5(i, j)], x); };
    if (z == 0) {
        add(0, 0, s);
        sub(0, 1, s);
        add(1, 1, s);
        add(3, 3, s);
        add(4, 4, s);
        add(0, 4, a);
        sub(1, 4, a);
        add(0, 3, b);
        sub(1, 3, b);
        add(3, 4, dl);
    } else if (z == 1) {
        add(0, 0, s);
        add(0, 1, s);
        add(1, 1, s);
        add(4, 4, s);
        add(2, 2, s);
        sub(0, 4, a);
        sub(1, 4, a);
        sub(0, 2, b);
        sub(1, 2, b);
        add(2, 4, dl);
    } else {
        add(0, 0, twice(twice(s)));
        add(3, 3, s);
        add(2, 2, s);
        sub(0, 3, twice(a));
        sub(0, 2, twice(b));
        add(2, 3, dl);
    }
}

// h = dtgn |r|^(n-1) / tau of every system at y (float pairs), into the
// tangent.  One loop body serves the three families (their inputs selected by
// z): unrolled, the instructions of this part alone were three times as many,
// and the warps, each in another place of the Newton loop, waited for them.
__device__ __forceinline__ void fcc_jac_ff(const RveDesc &d, long long v, const ff32 (&y)[5], ff32 dtgn, ff32 (&J)[15])
{
    const int e = d.ipow_n - 1;
#pragma unroll 1
    for (int z = 0; z < 3; ++z) {
        // D = y0 - y1, -y0 - y1, -2 y0
        const ff32 D = ffs_sub(z == 0 ? y[0] : ffs_neg(y[0]), z == 2 ? y[0] : y[1]);
        const ff32 a = z == 2 ? y[3] : y[4], b = z == 0 ? y[3] : y[2];
        const ff32 u = ffs_add(a, b), w = ffs_sub(a, b);
        ff32 r[4] = {ffs_add(D, u), ffs_sub(D, u), ffs_add(D, w), ffs_sub(D, w)}, h[4];
        const double *tau = d.itau + (long long)(8 * z) * d.nv + v;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int neg = r[k].h < 0.0f;
            const ff32 it = d2ff(__ldg(tau + (long long)(2 * k + neg) * d.nv));
            r[k] = ffs_mul(ffs_norm(r[k]), it);
            if (neg) r[k] = ffs_neg(r[k]);
            h[k] = ffs_mul(it, dtgn);
        }
        if (e == 19) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const ff32 a2 = ffs_mul(r[k], r[k]), a4 = ffs_mul(a2, a2), a8 = ffs_mul(a4, a4), a16 = ffs_mul(a8, a8);
                h[k] = ffs_mul(ffs_mul(ffs_mul(a16, a2), r[k]), h[k]);
            }
        } else if (e > 0) {
            ff32 q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = r[k];
            fcc_ipow_any(q, 4, e);
#pragma unroll
            for (int k = 0; k < 4; ++k) h[k] = ffs_mul(q[k], h[k]);
        }
        fcc_tangent_ff(z, h, J);
    }
}

// x := M^-1 x at the stress y.  False when a value left the float range (the
// caller then takes the FP64 solve).
__device__ __forceinline__ bool fcc_solve_ff(const RveDesc &d, long long v, const double (&yd)[5], double (&xd)[5],
                                             ff32 dtgn)
{
    ff32 M[15];
    {
        ff32 y[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) y[c] = d2ff(yd[c]);
#pragma unroll
        for (int q = 0; q < 15; ++q) M[q] = d2ff(__ldg(d.sch + (FCC_P + q) * d.nv + v));
        fcc_jac_ff(d, v, y, dtgn, M);
    }
    auto fms = [](ff32 &acc, ff32 a, ff32 b) { ff_acc2(acc, -a.h, -a.l, b.h, b.l); };
    // LDL^T in place, as fcc_factor
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const ff32 di = ff_rcp(ffs_norm(M[sym5(j, j)]));
        ff32 w[5];
#pragma unroll
        for (int i = j + 1; i < 5; ++i) {
            w[i] = ffs_norm(M[sym5(j, i)]);
            M[sym5(j, i)] = ffs_mul(w[i], di);
        }
#pragma unroll
        for (int i = j + 1; i < 5; ++i)
#pragma unroll
            for (int k = i; k < 5; ++k) fms(M[sym5(i, k)], M[sym5(j, i)], w[k]);
        M[sym5(j, j)] = di;
    }
    ff32 b[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) b[c] = d2ff(xd[c]);
#pragma unroll
    for (int i = 0; i < 5; ++i) {
#pragma unroll
        for (int k = 0; k < i; ++k) fms(b[i], M[sym5(k, i)], b[k]);
        b[i] = ffs_norm(b[i]);
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) b[i] = ffs_mul(b[i], M[sym5(i, i)]);
#pragma unroll
    for (int i = 3; i >= 0; --i) {
#pragma unroll
        for (int k = i + 1; k < 5; ++k) fms(b[i], M[sym5(i, k)], b[k]);
        b[i] = ffs_norm(b[i]);
    }
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        ok = ok && fabsf(b[c].h) < 1e30f;
        xd[c] = f2d(b[c].h) + f2d(b[c].l);   // (finite, or not taken)
    }
    return ok;
}
