// sm_103a kernels of the EVP-FFT solver step.  See voce_dev.cuh for the
// data layout.  One Green-operator iteration is
//   kb_fft_z_fwd -> kb_fft_y(-1) -> kb_fft_x_green -> kb_fft_y(+1) ->
//   kb_fft_z_inv(update) -> kb_nr / kb_nr_fcc -> kb_finalize
// and an increment, opened by kb_prelude, ends with
//   kb_fft_x_aacc -> kb_fft_y(+1,aacc) -> kb_fft_z_inv(rotl) ->
//   kb_incr_end / kb_incr_end_fcc -> kb_finalize
// The spectrum passes are in voce_fft.cuh; the Newton kernels and the increment
// epilogue of the {111}<110> slip family use voce_fcc.cuh.
#include "voce_dev.cuh"
#include "voce_fcc.cuh"
#include "voce_fft.cuh"

#include <math.h>

#include <algorithm>
#include <atomic>

namespace voce {

// ---------------------------------------------------------------------------
// deterministic block reduction of VOCE_NPART partial sums (entry 15 is a max)
// ---------------------------------------------------------------------------
__device__ void block_partials(double (&acc)[VOCE_NPART], double *out)
{
    __shared__ double red[32][VOCE_NPART];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < VOCE_NPART; ++q) {
        double x = acc[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double y = __shfl_down_sync(0xffffffffu, x, o);
            x = (q == VOCE_NPART - 1) ? fmax(x, y) : x + y;
        }
        if (lane == 0) red[warp][q] = x;
    }
    __syncthreads();
    if (threadIdx.x < VOCE_NPART) {
        const int q = threadIdx.x, nw = (blockDim.x + 31) >> 5;
        double s = red[0][q];
        for (int w = 1; w < nw; ++w) s = (q == VOCE_NPART - 1) ? fmax(s, red[w][q]) : s + red[w][q];
        out[q] = s;
    }
    __syncthreads();
}

// Sum the per-block partials of one kernel in a fixed order (one block of 256
// threads) into tot, in shared memory.  A thread takes one quantity over one
// stripe, a run of consecutive blocks, with up to 32 loads in flight and a
// pairwise tree over them; the stripe sums are then added pairwise too.  Entry
// 15 is a max (of non-negative counts, so 0 is its identity as for the sums).
// With one phase (all1) the phase-1 sums 8..13 are those of 2..7, and the
// threads are shared out over the ten others (25 stripes instead of 16).
__device__ void reduce_partials(const double *part, int npart, int all1, double (&tot)[VOCE_NPART])
{
    __shared__ double red[25][VOCE_NPART];
    const int t = threadIdx.x;  // blockDim.x == 256
    const int nq = all1 ? 10 : VOCE_NPART, ns = all1 ? 25 : 16;
    const int stripe = t / nq, k0 = t - stripe * nq;
    const int q = all1 && k0 >= 8 ? k0 + 6 : k0;
    const bool mx = q == VOCE_NPART - 1;
    const int chunk = (npart + ns - 1) / ns;
    const int b0 = stripe * chunk, b1 = stripe < ns ? min(npart, b0 + chunk) : 0;
    double s = 0.0;
    for (int b = b0; b < b1; b += 32) {
        double x[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) x[k] = (b + k < b1) ? part[(long long)(b + k) * VOCE_NPART + q] : 0.0;
#pragma unroll
        for (int w = 16; w >= 1; w >>= 1) {
            if (w >= b1 - b) continue;   // (nothing but zeros beyond)
#pragma unroll
            for (int k = 0; k < w; ++k) x[k] = mx ? fmax(x[k], x[k + w]) : x[k] + x[k + w];
        }
        s = mx ? fmax(s, x[0]) : s + x[0];
    }
    if (stripe < ns) red[stripe][q] = s;
    __syncthreads();
    // quantity q by the lanes of one warp's half: 16 lanes, then 8, 4, 2, 1
    {
        const int lane16 = t & 15, q2 = t >> 4;
        const bool on = !(all1 && q2 >= 8 && q2 < 14), mx2 = q2 == VOCE_NPART - 1;
        double v = on ? red[lane16][q2] : 0.0;
        if (on && lane16 + 16 < ns) v = mx2 ? fmax(v, red[lane16 + 16][q2]) : v + red[lane16 + 16][q2];
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) {
            const double y = __shfl_down_sync(0xffffffffu, v, o, 16);
            v = mx2 ? fmax(v, y) : v + y;
        }
        if (lane16 == 0 && on) {
            tot[q2] = v;
            if (all1 && q2 >= 2 && q2 < 8) tot[q2 + 6] = v;
        }
    }
    __syncthreads();
}

// rotation of the 6-vector basis: x_sample = Mr * x_crystal for the
// tensor map X -> a^T X a (a = sample->crystal matrix, TranMat = a^T):
// Mr[b][c] = <B_b, a^T B_c a>
__device__ void rotation_B(const double (&a)[3][3], double (&Mr)[6][6])
{
    for (int c = 0; c < 6; ++c) {
        double bc6[6] = {0, 0, 0, 0, 0, 0};
        bc6[c] = 1.0;
        double t6[6];
        b_to_t6<double>(bc6, t6);
        double X[3][3] = {{t6[0], t6[5], t6[4]}, {t6[5], t6[1], t6[3]}, {t6[4], t6[3], t6[2]}};
        double Y[3][3], Z[3][3];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double s = 0.0;
                for (int m = 0; m < 3; ++m) s += X[i][m] * a[m][j];
                Y[i][j] = s;  // X a
            }
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) {
                double s = 0.0;
                for (int m = 0; m < 3; ++m) s += a[m][i] * Y[m][j];
                Z[i][j] = s;  // a^T X a
            }
        double z6[6] = {Z[0][0], Z[1][1], Z[2][2], 0.5 * (Z[1][2] + Z[2][1]),
                        0.5 * (Z[0][2] + Z[2][0]), 0.5 * (Z[0][1] + Z[1][0])};
        double col[6];
        t6_to_b<double>(z6, col);
        for (int b = 0; b < 6; ++b) Mr[b][c] = col[b];
    }
}

// EulerToTransMatrix opt 2 (kinematics.c:529-545)
__device__ void euler_a(double t1, double ph, double t2, double (&a)[3][3])
{
    double ct1 = cos(t1), st1 = sin(t1), cph = cos(ph), sph = sin(ph), ct2 = cos(t2), st2 = sin(t2);
    a[0][0] = ct1 * ct2 - st1 * st2 * cph;
    a[0][1] = st1 * ct2 + ct1 * st2 * cph;
    a[0][2] = st2 * sph;
    a[1][0] = -1.0 * ct1 * st2 - st1 * ct2 * cph;
    a[1][1] = -1.0 * st1 * st2 + ct1 * ct2 * cph;
    a[1][2] = ct2 * sph;
    a[2][0] = st1 * sph;
    a[2][1] = -1.0 * ct1 * sph;
    a[2][2] = cph;
}

__device__ void schmid_from_tm(const RveDesc &d, long long v, const double (&T)[3][3])
{
    double a[3][3], Mr[6][6];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) a[i][j] = T[j][i];
    rotation_B(a, Mr);
    for (int s = 0; s < d.nsys; ++s)
        for (int i = 0; i < 5; ++i) {
            double acc = 0.0;
            for (int c = 0; c < 5; ++c) acc += Mr[i][c] * d.schxt[5 * s + c];
            d.sch[(long long)(5 * s + i) * d.nv + v] = acc;
            if (d.sch32) put_pair(d.sch32, d.sch_lo, (long long)(5 * s + i) * d.nv + v, acc);
        }
}

// put_pair through the integer pipe
__device__ __forceinline__ void put_ff(float *hi, float *lo, long long i, double x)
{
    const ff32 p = d2ff(x);
    hi[i] = p.h;
    lo[i] = p.l;
}

// Column c < 5 of the rotation of the 6-vector basis from crystal to sample
// axes: the deviatoric part of T B_c T^T, written out tensor by tensor (its
// entries are products of two columns of T)
__device__ __forceinline__ void rotated_basis(const double (&T)[3][3], int c, double (&q)[5])
{
    const int I6[6] = {0, 1, 2, 1, 0, 0}, J6[6] = {0, 1, 2, 2, 2, 1};
    double z[6], b6[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int i = I6[k], j = J6[k];
        if (c == 0) z[k] = RSQ2 * (T[i][1] * T[j][1] - T[i][0] * T[j][0]);
        else if (c == 1) z[k] = RSQ6 * (2.0 * T[i][2] * T[j][2] - T[i][0] * T[j][0] - T[i][1] * T[j][1]);
        else {
            const int p = c == 2 ? 1 : 0, r = c == 4 ? 1 : 2;
            z[k] = RSQ2 * (T[i][p] * T[j][r] + T[i][r] * T[j][p]);
        }
    }
    t6_to_b<double>(z, b6);
#pragma unroll
    for (int i = 0; i < 5; ++i) q[i] = b6[i];
}

// The crystal-axes columns of voxel v (voce_fcc.cuh) for the orientation T
// (crystal -> sample): U, P_y, S0_y, and y of the stress the voxel has
__device__ __forceinline__ void fcc_frame(const RveDesc &d, long long v, const double (&T)[3][3])
{
    const long long nv = d.nv;
    double *fx = d.sch + v;
    double U[5][5];
    double s[5], t[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < 5; ++i) s[i] = d.sig[i * nv + v];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        double q[5];
        rotated_basis(T, c, q);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            U[i][c] = q[i] * (c == 1 ? 2.0 : 3.4641016151377545871);   // sqrt 12
            fx[(FCC_U + 5 * i + c) * nv] = U[i][c];
            t[c] = fma(U[i][c], s[i], t[c]);
        }
        fx[(FCC_Y + c) * nv] = t[c] * (1.0 / fcc_w2(c));
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        double p0[5], p1[5];   // columns k of S0 U and S_g U
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            p0[i] = p1[i] = 0.0;
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                p0[i] = fma(d.S0[i * 6 + j], U[j][k], p0[i]);
                p1[i] = fma(__ldg(d.sg + (long long)sym6(i, j) * nv + v), U[j][k], p1[i]);
            }
        }
#pragma unroll
        for (int c = 0; c <= k; ++c) {
            double a0 = 0.0, a1 = 0.0;
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                a0 = fma(U[i][c], p0[i], a0);
                a1 = fma(U[i][c], p1[i], a1);
            }
            fx[(FCC_S0 + sym5(c, k)) * nv] = a0;
            fx[(FCC_P + sym5(c, k)) * nv] = a0 + a1;
            if (d.sgp32) put_ff(d.sgp32, d.sgp_lo, sym5(c, k) * nv + v, a0 + a1);
            if (d.nr32) d.sch32[sym5(c, k) * nv + v] = (float)a0;
        }
    }
}

// ---------------------------------------------------------------------------
// setup: per-voxel rotation, grain stiffness/compliance, Schmid tensors,
// initial stress (InitMicroStruct init.c:393-442, InitFields init.c:486-534,
// update_schmid kinematics.c:426-459 for istep 1).  The crystal is cubic (three
// elastic constants), so its stiffness and compliance are diagonal in the
// 6-vector basis with two deviatoric values x1 (components 0, 1) and x2 and the
// pressure apart, and a grain's are x2 I + (x1 - x2) (q0 q0^T + q1 q1^T), q0
// and q1 the rotated first two basis tensors: 60 FP64 operations instead of
// the 3000 of two 6x6 triple products (creation of a 96^3 mixed_nr32 RVE 13.2
// -> 6.5 ms, a 64^3 mixed_ir one 5.1 -> 3.1 ms).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_setup(RveDesc d, SetupConst sc, const double *__restrict__ euler)
{
    double count = 0.0;   // solid voxels
    double cacc[16];      // sums of C_gr: the deviatoric block, packed, and the pressure entry
#pragma unroll
    for (int q = 0; q < 16; ++q) cacc[q] = 0.0;
    const long long nv = d.nv;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv;
         v += (long long)gridDim.x * blockDim.x) {
        const int ph = d.phase[v];
        for (int c = 0; c < 6; ++c) {
            d.eps[c < 5 ? c * nv + v : v] = 0.0;
            d.dgs[c * nv + v] = 0.0;
        }
        for (int c = 0; c < 3; ++c) d.dga[c * nv + v] = 0.0;
        d.gamacum[v] = 0.0;
        for (int k = 0; k < VOCE_NS; ++k) {
            d.gtot[k * nv + v] = 0.0;
            d.gamdot[k * nv + v] = 0.0;
            d.taux[k * nv + v] = 0.0;
        }
        for (int c = 0; c < 5; ++c) d.edot[c * nv + v] = 0.0;
        d.svm[v] = 0.0;
        d.evm[v] = 0.0;
        for (int c = 0; c < 3; ++c) d.diag[c * nv + v] = 0.0;
        if (!d.solid[ph]) {
            for (int c = 0; c < 6; ++c) { d.sig[c * nv + v] = 0.0; d.sigp[c * nv + v] = 0.0; }
            for (int c = 0; c < 9; ++c) d.tm[c * nv + v] = (c % 4 == 0) ? 1.0 : 0.0;
            for (int c = 0; c < 21; ++c) d.sg[c * nv + v] = 0.0;
            for (int c = 0; c < 60; ++c) d.sch[c * nv + v] = 0.0;
            if (d.sch32)
                for (int c = 0; c < 60; ++c) put_pair(d.sch32, d.sch_lo, c * nv + v, 0.0);
            for (int c = 0; c < 24; ++c) { d.crss[c * nv + v] = 0.0; d.itau[c * nv + v] = 0.0; }
            if (d.itau32)
                for (int c = 0; c < 24; ++c) put_pair(d.itau32, d.itau_lo, c * nv + v, 0.0);
            continue;
        }
        count += 1.0;
        double a[3][3], T[3][3], q0[5], q1[5];
        const double f = VOCE_PI_REF / 180.;
        euler_a(euler[3 * v] * f, euler[3 * v + 1] * f, euler[3 * v + 2] * f, a);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                T[i][j] = a[j][i];
                d.tm[(3 * i + j) * nv + v] = a[j][i];
            }
        rotated_basis(T, 0, q0);
        rotated_basis(T, 1, q1);
        const double c2 = sc.cxt[14], c12 = sc.cxt[0] - c2, c5 = sc.cxt[35];
        const double s2 = sc.sxt[14], s12 = sc.sxt[0] - s2;
        // C_gr's deviatoric block (packed) and C_gr : DisGradAvg (+ Scauchy under creep)
        double sg6[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) sg6[i] = d.creep ? sc.sc6[i] : 0.0;
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = i; j < 5; ++j) {
                const double p = fma(q0[i], q0[j], q1[i] * q1[j]);
                const double cg = fma(c12, p, i == j ? c2 : 0.0);
                cacc[sym5(i, j)] += cg;
                sg6[i] = fma(cg, sc.d6[j], sg6[i]);
                if (i != j) sg6[j] = fma(cg, sc.d6[i], sg6[j]);
                d.sg[(long long)sym6(i, j) * nv + v] = fma(s12, p, i == j ? s2 : 0.0);
            }
        cacc[15] += c5;
        sg6[5] = fma(c5, sc.d6[5], sg6[5]);
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            d.sg[(long long)sym6(i, 5) * nv + v] = i == 5 ? sc.sxt[35] : 0.0;
            d.sig[i * nv + v] = sg6[i];
            d.sigp[i * nv + v] = sg6[i];
        }
        for (int k = 0; k < d.nsys; ++k) {
            d.crss[(2 * k) * nv + v] = d.tau0[k];
            d.crss[(2 * k + 1) * nv + v] = d.tau0b[k];
            d.itau[itau_col(d, k, 0) * nv + v] = 1.0 / d.tau0[k];
            d.itau[itau_col(d, k, 1) * nv + v] = 1.0 / d.tau0b[k];
            if (d.itau32) {
                put_pair(d.itau32, d.itau_lo, itau_col(d, k, 0) * nv + v, 1.0 / d.tau0[k]);
                put_pair(d.itau32, d.itau_lo, itau_col(d, k, 1) * nv + v, 1.0 / d.tau0b[k]);
            }
        }
        if (!d.fcc) schmid_from_tm(d, v, T);   // (the crystal-axes columns wait for S0: k_fill_fcc)
    }
    // voxel count and C066 partial sums in two passes of 15 (the 16th slot of
    // block_partials is a max and stays unused): the count and entries 0..13 of
    // cacc, then its last two
    double tmp[VOCE_NPART];
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int q = 0; q < VOCE_NPART; ++q) tmp[q] = 0.0;
        if (pass == 0) {
            tmp[0] = count;
#pragma unroll
            for (int q = 0; q < 14; ++q) tmp[1 + q] = cacc[q];
        } else {
            tmp[0] = cacc[14];
            tmp[1] = cacc[15];
        }
        block_partials(tmp, d.part + ((long long)pass * gridDim.x + blockIdx.x) * VOCE_NPART);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// per-voxel Newton-Raphson stress update (UpdateStress, evolution.c:3-168),
// solved in the equivalent symmetric form
//   (S0 + S_g + dt dEdot) dsig = S0 R
// where R is the reference's residual (evolution.c:78-83) and S0 = C0^-1.
// NR32 (the VOCE_PREC_MIXED_NR32 form): see mixed_newton below; otherwise
// the FP64 Newton of the reference, for the FP64 and VOCE_PREC_MIXED forms.
// ---------------------------------------------------------------------------

// P = S_g + S0 (packed upper triangle) of voxel v
__device__ __forceinline__ void load_P(const RveDesc &d, long long v, double (&P)[21])
{
#pragma unroll
    for (int q = 0; q < 21; ++q) P[q] = __ldg(d.sg + (long long)q * d.nv + v);
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = i; j < 6; ++j) P[sym6(i, j)] += d.S0[i * 6 + j];
}

// The same, with loads the compiler may not merge with earlier ones: a
// reload where keeping P live would cost registers.
__device__ __forceinline__ void reload_P(const RveDesc &d, long long v, double (&P)[21])
{
#pragma unroll
    for (int q = 0; q < 21; ++q) {
        const double *a = d.sg + (long long)q * d.nv + v;
        double x;
        asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(x) : "l"(a));
        P[q] = x;
    }
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = i; j < 6; ++j) P[sym6(i, j)] += d.S0[i * 6 + j];
}

// Newton steps on the FP64 residual with the stop test of evolution.c:112.
// NR32 (fallback of the single-precision form only): the Jacobian and its
// solve in FP32, an inexact Newton step converging to the same FP64 fixed
// point; otherwise all FP64.  With d.chord (the VOCE_PREC_MIXED form), an
// FP64 step whose predecessor moved the stress by less than 1e-4 relative
// reuses that predecessor's factored Jacobian (a chord step: the residual,
// the flow rule's strain rate and the stop test are evaluated as always, the
// Jacobian and its LDL^T factorisation are not).  Near the root the Jacobian
// then differs by about n x 1e-4 relative, so each chord step still divides
// the error by ~500; the converged stress moves by ~1e-14 relative against
// the exact-Jacobian Newton of the reference (evolution.c:85-110), the point
// before the last update (where the strain rate is evaluated) by up to 1e-8
// when the step count changes.
template <bool NR32, bool CHORD = false>
__device__ __forceinline__ void newton_fp64(const RveDesc &d, long long v, const double (&P)[21],
                                           const double (&cc)[6], double thr, double (&sig)[6],
                                           double (&sp)[6], double (&Rl)[6], int &it)
{
    const double dt = d.dt;
    bool go = true;
    // FP64 Jacobian factors, kept for chord steps (CHORD instances only)
    double L[6][6], dinv[6];
    bool fresh = true;
    (void)L; (void)dinv; (void)fresh;
    while (go && it < 100) {
        ++it;
        double ed[5];
#pragma unroll
        for (int c = 0; c < 6; ++c) sp[c] = sig[c];
        double R[6];
        if (NR32) {
            float D[15];
            flow_rule<true, false, float>(d, v, sig, ed, D, nullptr, nullptr);
            float M[6][6], x[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                double s = cc[i] + (i < 5 ? dt * ed[i] : 0.0);
#pragma unroll
                for (int j = 0; j < 6; ++j) s = fma(P[sym6(i, j)], sig[j], s);
                R[i] = s;
                Rl[i] = s;
                x[i] = (float)s;
            }
            const float dtf = (float)dt;
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    float m = (float)P[sym6(i, j)];
                    if (i < 5 && j < 5) m = fmaf(dtf, D[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
                    M[i][j] = m;
                }
            ldlt_solve6f(M, x);
#pragma unroll
            for (int i = 0; i < 6; ++i) R[i] = (double)x[i];
        } else if (!CHORD) {
            double D[15];
            flow_rule<true, false, double>(d, v, sig, ed, D, nullptr, nullptr);
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                double s = cc[i] + (i < 5 ? dt * ed[i] : 0.0);
#pragma unroll
                for (int j = 0; j < 6; ++j) s = fma(P[sym6(i, j)], sig[j], s);
                R[i] = s;
                Rl[i] = s;
            }
            double M[6][6];
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    double m = P[sym6(i, j)];
                    if (i < 5 && j < 5) m = fma(dt, D[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
                    M[i][j] = m;
                }
            ldlt_solve6(M, R);
        } else {
            if (fresh) {
                double D[15];
                flow_rule<true, false, double>(d, v, sig, ed, D, nullptr, nullptr);
                double M[6][6];
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int j = 0; j <= i; ++j) {
                        double m = P[sym6(i, j)];
                        if (i < 5 && j < 5) m = fma(dt, D[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
                        M[i][j] = m;
                    }
                ldlt_factor6(M, L, dinv);
            } else {
                flow_rule<false, false, double>(d, v, sig, ed, (double *)nullptr, nullptr, nullptr);
            }
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                double s = cc[i] + (i < 5 ? dt * ed[i] : 0.0);
#pragma unroll
                for (int j = 0; j < 6; ++j) s = fma(P[sym6(i, j)], sig[j], s);
                R[i] = s;
                Rl[i] = s;
            }
            ldlt_apply6(L, dinv, R);
        }
        double cnr = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const double sn = sig[c] - R[c];
            const double dd = sn - sig[c];
            cnr = fma(dd, dd, cnr);
            sig[c] = sn;
        }
        go = cnr > thr;
        // the next step reuses this Jacobian (a chord step) once the update
        // is below 1e-4 relative (cnr <= 1e-8 sn2 = 1e6 thr)
        if (CHORD) fresh = !d.chord || cnr > 1e6 * thr;
    }
}

// Mixed form: Newton in single precision (residual, Jacobian and solve) down
// to a relative update of 1e-4, then one Newton step on the double-precision
// residual with the last single-precision matrix.  That residual is evaluated
// in float-float on the FP32 pipe (residual_ff), from float pairs of the
// model data: the double-precision model to about 2^-48, at a fraction of the
// cost of FP64 arithmetic on this part.  That step is accepted when
// its relative update is below 1e-5: Newton's quadratic term then puts the
// next update near 1e-9, under the 1e-7 test of the FP64 form, so the
// accepted stress is taken as the converged point (zero residual, and the
// point the strain rate is later evaluated at).  Anything else continues with
// newton_fp64 from where it stands.  Without polish (Green iterations whose
// predecessor's error is above VOCE_POLISH_ERR, and the first of an
// increment) the single-precision Newton runs down to 1e-5 and its point is
// taken as converged: its error, a few 1e-6 relative, is far below the
// change such an iteration makes.
__device__ __forceinline__ void mixed_newton(const RveDesc &d, long long v, const float *st,
                                             const double (&lam)[6], const double (&cc)[6], double sn2,
                                             bool polish, double (&sig)[6], double (&sp)[6],
                                             double (&Rl)[6], int &it)
{
    const double dt = d.dt;
    bool done = false;
    if (d.ipow_n >= 1) {
        float sf[6], Mf[6][6], Pf[21];
#pragma unroll
        for (int q = 0; q < 21; ++q) Pf[q] = __ldg(d.sgp32 + (long long)q * d.nv + v);
        float ccf[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) { sf[c] = (float)lam[c]; ccf[c] = (float)cc[c]; }
        // single precision alone stops at a relative update of 1e-5, before a
        // polish step at 1e-4
        const float thr32 = (float)((polish ? 1e-8 : 1e-10) * sn2);
        const float dtf = (float)dt;
        bool ok = true, conv = false;
        cp_async_wait_all();   // the staged column of this voxel
        while (it < 24) {
            ++it;
            float ed[5], D[15], x[6];
            if (!flow_rule_f32(d, st, sf, ed, D)) { ok = false; break; }
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                float t = ccf[i] + (i < 5 ? dtf * ed[i] : 0.0f);
#pragma unroll
                for (int j = 0; j < 6; ++j) t = fmaf(Pf[sym6(i, j)], sf[j], t);
                x[i] = t;
            }
#pragma unroll
            for (int i = 0; i < 6; ++i)
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    float m = Pf[sym6(i, j)];
                    if (i < 5 && j < 5) m = fmaf(dtf, D[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
                    Mf[i][j] = m;
                }
            ldlt_solve6f(Mf, x);
            float dn = 0.0f;
#pragma unroll
            for (int c = 0; c < 6; ++c) { dn = fmaf(x[c], x[c], dn); sf[c] -= x[c]; }
            if (!(dn <= 3.0e38f)) { ok = false; break; }   // not finite
            if (dn < thr32) { conv = true; break; }
        }
        if (ok && conv && !polish) {
            done = true;
#pragma unroll
            for (int c = 0; c < 6; ++c) { sig[c] = (double)sf[c]; sp[c] = sig[c]; Rl[c] = 0.0; }
        } else if (ok && conv) {
            ++it;
            float x[6];
            if (residual_ff(d, v, st, sf, cc, Pf, x)) {
                ldlt_solve6f(Mf, x);
                float dn = 0.0f;
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    dn = fmaf(x[c], x[c], dn);
                    sig[c] = (double)sf[c] - (double)x[c];
                }
                if (dn <= (float)(1e-10 * sn2)) {
                    done = true;
#pragma unroll
                    for (int c = 0; c < 6; ++c) { sp[c] = sig[c]; Rl[c] = 0.0; }
                }
            } else {
#pragma unroll
                for (int c = 0; c < 6; ++c) sig[c] = (double)sf[c];
            }
        } else {
#pragma unroll
            for (int c = 0; c < 6; ++c) sig[c] = lam[c];
        }
    }
    if (!done) {
        double P[21];
        reload_P(d, v, P);
        newton_fp64<true>(d, v, P, cc, 1e-14 * sn2, sig, sp, Rl, it);
    }
}

// Newton iterations of the VOCE_PREC_MIXED_IR form: every iteration
// evaluates the reference's residual (evolution.c:78-83, in the symmetric
// form x = cc + dt edot(s) + (S_g + S0) s) and the flow rule
// (constitutive.c:126-194: resolved shears, |r|^n, strain rate) in FP64, and
// takes the stop test of evolution.c:112 in FP64; only the correction -- the
// Jacobian dt dEdot/ds + S_g + S0 and its LDL^T solve -- is assembled and
// solved in FP32, from float copies of the Schmid vectors, 1/CRSS and
// S_g + S0.  This is iterative refinement: each step solves for the FP64
// residual with an approximate matrix (relative error ~1e-7 times its
// condition number), so the iteration converges to the root of the FP64
// residual, near the root nearly as fast as the exact Newton.  A resolved
// shear ratio |r| >= 60 (where |r|^(n-1) could leave the float range) makes
// that iteration take the FP64 Jacobian instead.  gam0 is one value for all
// systems (one slip mode), so it is applied once to the strain-rate sums.
//
// With d.ir_pred the FP64 iterations start from a point computed on the FP32
// pipe (ir_start): single-precision Newton steps down to a relative update of
// 1e-4, then one step on the float-float residual (residual_ff, the model
// data as float pairs, about 48 bits) with the last single-precision matrix.
// That point lies within about 1e-9 relative of the FP64 residual's root, so
// the first FP64 step's update is already below the 1e-7 stop test: one FP64
// residual evaluation per voxel accepts it, against two to seven from the
// Green iterate.  The start never decides the result -- the accepted stress
// and the stop decision come from the FP64 steps.  A start that does not
// converge in single precision, meets a resolved-shear ratio too large for
// |r|^n in FP32 or a non-finite value is dropped (the FP64 steps then start
// from the Green iterate).  st is the voxel's staged column of float Schmid
// vectors and 1/CRSS (as in the single-precision Newton form).  The last
// single-precision matrix goes to the column mout (lower triangle packed,
// stride VOCE_NR_THREADS), where the FP64 steps read it.
__device__ __forceinline__ bool ir_start(const RveDesc &d, long long v, const float *st,
                                         const double (&lam)[6], const double (&cc)[6], double sn2,
                                         double (&sig)[6], int &it, float *mout)
{
    float sf[6], ccf[6], Pf[21], Mf[6][6];
#pragma unroll
    for (int q = 0; q < 21; ++q) Pf[q] = __ldg(d.sgp32 + (long long)q * d.nv + v);
#pragma unroll
    for (int c = 0; c < 6; ++c) { sf[c] = (float)lam[c]; ccf[c] = (float)cc[c]; }
    // single precision stops at a relative update of 1e-4 (its rounding
    // floor can lie near 1e-5); the float-float step then takes the point to
    // within Newton's quadratic term of that update (~1e-9)
    const float thr32 = 1e-8f * (float)sn2;
    const float dtf = d.dth;
    bool conv = false;
    cp_async_wait_all();   // the staged column of this voxel
    for (int p = 0; p < 12; ++p) {
        float ed[5], D[15], x[6];
        if (!flow_rule_f32(d, st, sf, ed, D)) return false;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            float t = ccf[i] + (i < 5 ? dtf * ed[i] : 0.0f);
#pragma unroll
            for (int j = 0; j < 6; ++j) t = fmaf(Pf[sym6(i, j)], sf[j], t);
            x[i] = t;
#pragma unroll
            for (int j = 0; j <= i; ++j) {
                float m = Pf[sym6(i, j)];
                if (i < 5 && j < 5) m = fmaf(dtf, D[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
                Mf[i][j] = m;
            }
        }
        ldlt_solve6f(Mf, x);
        float dn = 0.0f;
#pragma unroll
        for (int c = 0; c < 6; ++c) { dn = fmaf(x[c], x[c], dn); sf[c] -= x[c]; }
        ++it;
        if (!(dn <= 3.0e38f)) return false;   // not finite
        if (dn < thr32) { conv = true; break; }
    }
    if (!conv) return false;
    float x[6];
    if (!residual_ff(d, v, st, sf, cc, Pf, x)) return false;
    ldlt_solve6f(Mf, x);
    ++it;
#pragma unroll
    for (int c = 0; c < 6; ++c) sig[c] = (double)sf[c] - (double)x[c];
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) mout[sym6(i, j) * VOCE_NR_THREADS] = Mf[i][j];
    return true;
}

// One FP64-Jacobian step of newton_ir, for the rare iteration whose
// resolved-shear ratio leaves the float range; kept out of line so that its
// registers do not weigh on the common path.
__device__ __noinline__ void ir_fp64_step(const RveDesc &d, long long v, const double *sig, double *R)
{
    double P[21], Dd[15], edd[5];
    for (int q = 0; q < 21; ++q) P[q] = d.sgp[(long long)q * d.nv + v];
    flow_rule<true, false, double>(d, v, sig, edd, Dd, nullptr, nullptr);
    double M[6][6], b[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        b[i] = R[i];
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            double m = P[sym6(i, j)];
            if (i < 5 && j < 5) m = fma(d.dt, Dd[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
            M[i][j] = m;
        }
    }
    ldlt_solve6(M, b);
#pragma unroll
    for (int i = 0; i < 6; ++i) R[i] = b[i];
}

// mst (with START): the single-precision matrix of the start's last step,
// lower triangle packed, in the voxel's staged column; the FP64 steps solve
// with it instead of assembling the Jacobian again (near the root it is the
// Jacobian to about n x 1e-4 relative, so each step still divides the error
// by ~500 -- and from the start one step is usually the last).  S_g + S0 is
// read from d.sgp (FP64, stored at setup) where the residual needs it, rather
// than kept in registers across the iterations.
template <bool START>
__device__ __forceinline__ void newton_ir(const RveDesc &d, long long v, const double (&cc)[6],
                                          double thr, double (&sig)[6], double (&sp)[6],
                                          double (&Rl)[6], int &it, const float *mst)
{
    const long long nv = d.nv;
    const double dtg = d.dt * d.gam0[0];
    const float dtf = d.dth;
    const float g1c = d.gam0f[0] * d.nrsf[0];   // gam0 n
    const int e = d.ipow_n - 1;
    bool go = true;
    while (go && it < 100) {
        ++it;
#pragma unroll
        for (int c = 0; c < 6; ++c) sp[c] = sig[c];
        double ed[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        float D[15];
#pragma unroll
        for (int q = 0; q < 15; ++q) D[q] = 0.0f;
        bool big = false;
#pragma unroll 2
        for (int k = 0; k < d.nsys; ++k) {
            double sc[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) sc[i] = __ldg(d.sch + (long long)(5 * k + i) * nv + v);
            const double rss = sc[0] * sig[0] + sc[1] * sig[1] + sc[2] * sig[2] + sc[3] * sig[3] + sc[4] * sig[4];
            const int neg = __double2hiint(rss) < 0;
            const long long ti = (long long)(2 * k + neg) * nv + v;
            const double it0 = __ldg(d.itau + (long long)(2 * k) * nv + v);
            const double it1 = __ldg(d.itau + (long long)(2 * k + 1) * nv + v);
            const double r = rss * (neg ? it1 : it0);
            // |r| >= 60 (or not finite), tested on the high word: an
            // integer comparison instead of one on the FP64 pipe
            big = big || (__double2hiint(r) & 0x7fffffff) >= 0x404E0000;
            double g2;                                // |r|^n sign(r) / gam0
            float aef;                                // |r|^(n-1), for the float Jacobian
            if (e == 19) {
                // |r|^20 = ((r^2)^2 |r|)^2)^2: five products, the sign of r
                // put on the high word
                const double a2 = r * r, a4 = a2 * a2, a5 = a4 * fabs(r), a10 = a5 * a5, a20 = a10 * a10;
                g2 = __hiloint2double(__double2hiint(a20) | (__double2hiint(r) & (int)0x80000000),
                                      __double2loint(a20));
                if (!START) {
                    const float af = fabsf((float)r), af2 = af * af, af4 = af2 * af2, af8 = af4 * af4;
                    aef = af8 * af8 * af2 * af;
                }
            } else {
                const double ae = pow_abs_e(fabs(r), e);   // |r|^(n-1)
                g2 = ae * r;
                aef = (float)ae;
            }
#pragma unroll
            for (int i = 0; i < 5; ++i) ed[i] = fma(sc[i], g2, ed[i]);
            if (START) continue;
            // Jacobian term gam0 n |r|^(n-1) / tau m m^T, in single precision
            const float g1 = g1c * aef * __ldg(d.itau32 + ti);
            float sf[5], t[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                sf[i] = __ldg(d.sch32 + (long long)(5 * k + i) * nv + v);
                t[i] = g1 * sf[i];
            }
            int q = 0;
#pragma unroll
            for (int i = 0; i < 5; ++i)
#pragma unroll
                for (int j = i; j < 5; ++j) { D[q] = fmaf(t[i], sf[j], D[q]); ++q; }
        }
        double R[6];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            double s = (i < 5) ? fma(dtg, ed[i], cc[i]) : cc[i];
#pragma unroll
            for (int j = 0; j < 6; ++j) s = fma(__ldg(d.sgp + (long long)sym6(i, j) * nv + v), sig[j], s);
            R[i] = s;
            Rl[i] = s;
        }
        if (!big) {
            float M[6][6], x[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                x[i] = (float)R[i];
#pragma unroll
                for (int j = 0; j <= i; ++j) {
                    float m;
                    if (START) {
                        m = mst[sym6(i, j) * VOCE_NR_THREADS];
                    } else {
                        m = __ldg(d.sgp32 + (long long)sym6(i, j) * nv + v);
                        if (i < 5 && j < 5) m = fmaf(dtf, D[j * 5 - (j * (j - 1)) / 2 + (i - j)], m);
                    }
                    M[i][j] = m;
                }
            }
            ldlt_solve6f(M, x);
#pragma unroll
            for (int i = 0; i < 6; ++i) R[i] = (double)x[i];
        } else {
            ir_fp64_step(d, v, sig, R);
        }
        // the stop test of evolution.c:112 on the update itself (the
        // reference's |sig_new - sig_old|^2 up to the rounding of one
        // subtraction)
        double cnr = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            cnr = fma(R[c], R[c], cnr);
            sig[c] -= R[c];
        }
        go = cnr > thr;
    }
}

template <bool NR32, bool CHORD = false, bool IR = false>
__device__ void nr_unit(const RveDesc &d, int unit, int nunits)
{
    // per-thread sums in shared memory (one slot per thread, the same
    // additions in the same order as register accumulators) keep them out of
    // the registers the Newton loop needs
    __shared__ double s_acc[VOCE_NPART][VOCE_NR_THREADS];
    // Newton iteration count (sum, max) as integers; entries 14 and 15 of
    // the partials receive them converted, the same values
    __shared__ int s_it[2][VOCE_NR_THREADS];
    const int tid = threadIdx.x;
    // NR32: this thread's column of the staged float model data
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *st = reinterpret_cast<float *>(smem_raw) + tid;
    bool polish = true;
    if (NR32) {
        const MacroDev *m = d.macro;
        polish = !m->first_iter && fmax(fabs(m->Err_e), fabs(m->Err_s)) <= VOCE_POLISH_ERR;
    }
#pragma unroll
    for (int q = 0; q < VOCE_NPART; ++q) s_acc[q][tid] = 0.0;
    s_it[0][tid] = 0;
    s_it[1][tid] = 0;
    const long long nv = d.nv;
    for (long long v = (long long)unit * blockDim.x + threadIdx.x; v < nv;
         v += (long long)nunits * blockDim.x) {
        if (NR32 || IR) {
            // asynchronous copies of the voxel's float Schmid vectors and
            // 1/CRSS; every path below waits for them before the next voxel
#pragma unroll
            for (int c = 0; c < VOCE_STAGE_ITAU; ++c) cp_async4(st + c * VOCE_NR_THREADS, d.sch32 + c * nv + v);
#pragma unroll
            for (int c = 0; c < 24; ++c)
                cp_async4(st + (VOCE_STAGE_ITAU + c) * VOCE_NR_THREADS, d.itau32 + c * nv + v);
        }
        if ((IR && d.ir_pred) || (NR32 && polish)) {
            // the low halves the float-float step reads (the mixed_ir start's,
            // the mixed_nr32 acceptance step's), brought to L2 while the
            // single-precision steps run: one 128-byte line per row of the
            // warp's 32 voxels, the 105 rows shared out over the lanes (the
            // FP64 rows or the next voxel's rows as well: measured slower)
            const int lane = tid & 31;
            const long long vw = v - lane;
            for (int r = lane; r < 105; r += 32) {
                const float *b = r < 60 ? d.sch_lo + (long long)r * nv
                               : r < 84 ? d.itau_lo + (long long)(r - 60) * nv : d.sgp_lo + (long long)(r - 84) * nv;
                asm volatile("prefetch.global.L2 [%0];" ::"l"(b + vw));
            }
        }
        const int ph = d.phase[v];
        if (!d.solid[ph]) {
#pragma unroll
            for (int c = 0; c < 6; ++c) { d.sig[c * nv + v] = 0.0; d.sigp[c * nv + v] = 0.0; }
            if (NR32 || IR) cp_async_wait_all();
            continue;
        }
        double lam[6], cc[6];
        {
            double e6[6], ep[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) {
                lam[c] = d.sig[c * nv + v];
                e6[c] = d.dgs[c * nv + v];
            }
#pragma unroll
            for (int c = 0; c < 5; ++c) ep[c] = d.eps[c * nv + v];
            ep[5] = 0.0;
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                double s = ep[i] - e6[i];
#pragma unroll
                for (int j = 0; j < 6; ++j) s = fma(-d.S0[i * 6 + j], lam[j], s);
                cc[i] = s;
            }
        }
        double sn2 = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) sn2 = fma(lam[c], lam[c], sn2);
        double sig[6], sp[6], Rl[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) { sig[c] = lam[c]; sp[c] = lam[c]; Rl[c] = 0.0; }
        int it = 0;
        if (NR32) {
            mixed_newton(d, v, st, lam, cc, sn2, polish, sig, sp, Rl, it);
            cp_async_wait_all();   // (already done unless the float phase was skipped)
        } else if (IR && d.ipow_n >= 1) {
            // sqrt(cnr)/signorm > 1e-7 (evolution.c:112) tested as cnr > 1e-14 signorm^2
            bool started = false;
            if (d.ir_pred) {
                int it0 = it;
                // the staged column is read no more once the start ends: it
                // keeps the last matrix for the FP64 steps (st is this
                // thread's own column)
                started = ir_start(d, v, st, lam, cc, sn2, sig, it, const_cast<float *>(st));
                if (!started) {
#pragma unroll
                    for (int c = 0; c < 6; ++c) sig[c] = lam[c];
                    it = it0;
                }
            }
            if (started) newton_ir<true>(d, v, cc, 1e-14 * sn2, sig, sp, Rl, it, st);
            else newton_ir<false>(d, v, cc, 1e-14 * sn2, sig, sp, Rl, it, nullptr);
            cp_async_wait_all();
        } else {
            double P[21];
            load_P(d, v, P);
            // sqrt(cnr)/signorm > 1e-7 (evolution.c:112) tested as cnr > 1e-14 signorm^2
            newton_fp64<IR, CHORD>(d, v, P, cc, 1e-14 * sn2, sig, sp, Rl, it);
            if (IR) cp_async_wait_all();
        }
        double ncs, nce;   // |sig - lam| and the strain-compatibility norm (evolution.c:118-123)
        if (NR32) {
            // error norms in single precision: they only steer the Green
            // iteration's stop test at 1e-5
            float ds[6], dp[6], cs = 0.0f, ce = 0.0f;
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                ds[i] = (float)(sig[i] - lam[i]);
                dp[i] = (float)(sp[i] - lam[i]);
                cs = fmaf(ds[i], ds[i], cs);
            }
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                float te = (float)Rl[i];
#pragma unroll
                for (int j = 0; j < 6; ++j) te = fmaf(-d.S0f[i * 6 + j], dp[j], te);
                ce = fmaf(te, te, ce);
            }
            ncs = (double)sqrtf(cs);
            nce = (double)sqrtf(ce);
        } else {
            double cs = 0.0, ce = 0.0;
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const double ds = sig[i] - lam[i];
                cs = fma(ds, ds, cs);
                double te = Rl[i];
#pragma unroll
                for (int j = 0; j < 6; ++j) te = fma(-d.S0[i * 6 + j], sp[j] - lam[j], te);
                ce = fma(te, te, ce);
            }
            // the mixed_ir form's norms by a Newton-Raphson square root
            // (about 1e-13 relative); the other forms' correctly rounded
            ncs = IR ? sqrt_nr(cs) : sqrt(cs);
            nce = IR ? sqrt_nr(ce) : sqrt(ce);
        }
#pragma unroll
        for (int c = 0; c < 6; ++c) { d.sig[c * nv + v] = sig[c]; d.sigp[c * nv + v] = sp[c]; }
        s_acc[0][tid] += ncs;
        s_acc[1][tid] += nce;
#pragma unroll
        for (int c = 0; c < 6; ++c) s_acc[2 + c][tid] += sig[c];
        // phase-1 sums; when every voxel is phase 1 they would repeat the
        // sums above addition for addition, and are copied from them below
        if (ph == 1 && !d.all_ph1) {
#pragma unroll
            for (int c = 0; c < 6; ++c) s_acc[8 + c][tid] += sig[c];
        }
        s_it[0][tid] += it;
        s_it[1][tid] = max(s_it[1][tid], it);
    }
    double acc[VOCE_NPART];
#pragma unroll
    for (int q = 0; q < VOCE_NPART; ++q) acc[q] = s_acc[q][tid];
    if (d.all_ph1) {
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[8 + c] = acc[2 + c];
    }
    acc[14] = (double)s_it[0][tid];
    acc[15] = (double)s_it[1][tid];
    block_partials(acc, d.part + (long long)unit * VOCE_NPART);
}


// ---------------------------------------------------------------------------
// UpdateStress (evolution.c:3-168) for an RVE of the {111}<110> family in
// crystal axes (voce_fcc.cuh), one kernel instance per form.
//
// FCC_FP64 (the FP64 form and VOCE_PREC_MIXED): the Newton iteration of
// newton_fp64 -- the exact Jacobian, the stop test of evolution.c:112, the
// strain rate and the norms at the stress before the last update -- in the
// variables y, so its iterates agree to rounding.  Bound: the FP64 pipe (64
// cycles of an SM quarter's pipe per warp instruction).  A Newton iteration
// takes about 170 FP64 operations instead of about 680 in sample axes: 21
// instead of 60 for the resolved shears, 27 instead of 60 for the strain rate,
// 72 for the powers, 25 for P y (the pressure decouples); the tangent and the
// 5x5 solve, 240 + 125 there, run in float pairs on the FP32 pipe beside it.
// Measured per launch against kb_nr (FP64 form, first increment): 64^3 879 ->
// 347 us (477 with the solve in FP64), 128^3 10.4 -> 3.8 ms, 16^3 (a grain
// per voxel) 86 -> 46 us.
// With the solve off the FP64 pipe a chord step saves nothing, so d.chord is
// not looked at here.
//
// FCC_IR (VOCE_PREC_MIXED_IR): newton_ir in the same variables: the start in
// single precision and float pairs, then steps whose residual, flow rule and
// stop test are FP64 and whose correction is solved in FP32 with the start's
// last matrix; 64^3 363 -> 214 us, 256^3 29.9 -> 14.8 ms.  FCC_NR32
// (VOCE_PREC_MIXED_NR32): mixed_newton; 96^3 394 -> 315 us.  Nothing is staged
// in shared memory: the single-precision steps read 15 + 12 floats per voxel
// instead of 21 + 72.  Conversions go through the integer pipe (d2f_rn, f2d:
// with the hardware's, 239 and 331 us).
//
// kb_nr stays for every other slip table and for non-integral exponents.
// ---------------------------------------------------------------------------
enum { FCC_FP64 = 0, FCC_IR = 1, FCC_NR32 = 2 };

// x += P y with P_y of voxel v in FP64
__device__ __forceinline__ void fcc_add_Py(const double *fx, long long nv, const double (&y)[5], double (&x)[5])
{
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = i; j < 5; ++j) {
            const double q = __ldg(fx + (FCC_P + sym5(i, j)) * nv);
            x[i] = fma(q, y[j], x[i]);
            if (i != j) x[j] = fma(q, y[i], x[j]);
        }
}

// x := M^-1 x with the FP64 Jacobian at y, for the rare step whose
// resolved-shear ratio leaves the float range; out of line so that its
// registers do not weigh on the common path
__device__ __noinline__ void fcc_fp64_step(const RveDesc &d, long long v, const double *yp, double *xp)
{
    double y[5], x[5], E[5], J[15];
    for (int c = 0; c < 5; ++c) { y[c] = yp[c]; x[c] = xp[c]; }
    fcc_flow<true>(d, v, y, E, J);
    const double dtgn = d.dt * d.gam0[0] * d.nrs[0];
#pragma unroll
    for (int q = 0; q < 15; ++q) J[q] = fma(dtgn, J[q], d.sch[(FCC_P + q) * d.nv + v]);
    fcc_factor(J);
    fcc_solve<double>(J, x);
    for (int c = 0; c < 5; ++c) xp[c] = x[c];
}

// the same from registers: the copies keep y and x out of local memory
__device__ __forceinline__ void fcc_rare_step(const RveDesc &d, long long v, const double (&y)[5], double (&x)[5])
{
    double yt[5], xt[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) { yt[c] = y[c]; xt[c] = x[c]; }
    fcc_fp64_step(d, v, yt, xt);
#pragma unroll
    for (int c = 0; c < 5; ++c) x[c] = xt[c];
}

// The FP64 Newton steps with the exact Jacobian from y (s5 its pressure
// part): y, s5 the new stress, yp, s5p the stress before the last update, Rl,
// R5 the residual there.  The correction is solved in float pairs on the FP32
// pipe (fcc_solve_ff), except where a ratio |r| or the residual leaves the
// float range.
__device__ __forceinline__ void fcc_newton(const RveDesc &d, long long v, const double (&cc)[5], double cc5,
                                           double thr, double (&y)[5], double &s5, double (&yp)[5], double &s5p,
                                           double (&Rl)[5], double &R5, int &it)
{
    const long long nv = d.nv;
    const double *fx = d.sch + v;
    const double dtg = d.dt * d.gam0[0];
    const ff32 dtgn = d2ff(dtg * d.nrs[0]);
    bool go = true;
    while (go && it < 100) {
        ++it;
        double E[5], x[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) yp[c] = y[c];
        s5p = s5;
        bool fp64 = fcc_edot_fp64_loop(d, v, y, E) || d.ipow_n > 20;
#pragma unroll
        for (int c = 0; c < 5; ++c) x[c] = fma(dtg, E[c], cc[c]);
        fcc_add_Py(fx, nv, y, x);
        int top = 0;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            Rl[c] = x[c];
            top = max(top, __double2hiint(x[c]) & 0x7fffffff);
        }
        R5 = fma(d.P55, s5, cc5);
        const double x5 = R5 * d.iP55;
        fp64 = fp64 || top >= 0x46000000;   // |x| >= 2^97, or not finite
        if (!fp64) fp64 = !fcc_solve_ff(d, v, y, x, dtgn);
        if (fp64) {
#pragma unroll
            for (int c = 0; c < 5; ++c) x[c] = Rl[c];
            fcc_rare_step(d, v, y, x);
        }
#pragma unroll
        for (int c = 0; c < 5; ++c) y[c] -= x[c];
        s5 -= x5;
        go = fma(x5, x5, fcc_norm2<double>(x)) > thr;
    }
}

// The steps of newton_ir: FP64 residual, flow rule and stop test, the
// correction in FP32 with the factors L (started: the start's last matrix,
// kept for every step; otherwise the Jacobian of each step)
__device__ __forceinline__ void fcc_newton_ir(const RveDesc &d, long long v, bool started, float (&L)[15],
                                              const double (&cc)[5], double cc5, double thr, double (&y)[5],
                                              double &s5, double (&yp)[5], double &s5p, double (&Rl)[5], double &R5,
                                              int &it)
{
    const long long nv = d.nv;
    const double *fx = d.sch + v;
    const double dtg = d.dt * d.gam0[0];
    bool go = true;
    while (go && it < 100) {
        ++it;
        double E[5], x[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) yp[c] = y[c];
        s5p = s5;
        const bool big = fcc_edot_fp64(d, v, y, E);
#pragma unroll
        for (int c = 0; c < 5; ++c) x[c] = fma(dtg, E[c], cc[c]);
        fcc_add_Py(fx, nv, y, x);
#pragma unroll
        for (int c = 0; c < 5; ++c) Rl[c] = x[c];
        R5 = fma(d.P55, s5, cc5);
        const double x5 = R5 * d.iP55;
        bool fp64 = big;
        if (!big) {
            float xf[5];
            if (!started) {
                const float dtgn = (float)d.dt * d.gam0f[0] * d.nrsf[0];
                float yf[5], Ef[5];
#pragma unroll
                for (int c = 0; c < 5; ++c) yf[c] = (float)y[c];
                fp64 = !fcc_flow_f32(d, v, yf, Ef, L);   // (the ratio in float may round up to the limit)
#pragma unroll
                for (int q = 0; q < 15; ++q) L[q] = fmaf(dtgn, L[q], __ldg(d.sgp32 + (long long)q * nv + v));
                fcc_factor(L);
            }
            if (!fp64) {
#pragma unroll
                for (int c = 0; c < 5; ++c) xf[c] = d2f_rn(x[c]);
                fcc_solve<float>(L, xf);
                // a correction that is not finite in float (a residual beyond
                // the floats or broken, or an overflowed Jacobian) is solved
                // in FP64, where it stays what it is
                fp64 = !finite_f((xf[0] + xf[1]) + (xf[2] + xf[3]) + xf[4]);
                if (!fp64)
#pragma unroll
                    for (int c = 0; c < 5; ++c) x[c] = f2d(xf[c]);
            }
        }
        if (fp64) fcc_rare_step(d, v, y, x);
#pragma unroll
        for (int c = 0; c < 5; ++c) y[c] -= x[c];
        s5 -= x5;
        go = fma(x5, x5, fcc_norm2<double>(x)) > thr;
    }
}

template <int FORM>
__device__ void nr_fcc_unit(const RveDesc &d, int unit, int nunits)
{
    __shared__ double s_acc[VOCE_NPART][VOCE_NR_THREADS];
    __shared__ int s_it[2][VOCE_NR_THREADS];
    const int tid = threadIdx.x;
#pragma unroll
    for (int q = 0; q < VOCE_NPART; ++q) s_acc[q][tid] = 0.0;
    s_it[0][tid] = 0;
    s_it[1][tid] = 0;
    bool polish = true;
    if (FORM == FCC_NR32) {
        const MacroDev *m = d.macro;
        polish = !m->first_iter && fmax(fabs(m->Err_e), fabs(m->Err_s)) <= VOCE_POLISH_ERR;
    }
    // dt gam0 as a float pair
    const float dtgh = (float)(d.dt * d.gam0[0]), dtgl = (float)(d.dt * d.gam0[0] - (double)dtgh);
    (void)polish; (void)dtgh; (void)dtgl;
    const long long nv = d.nv;
    for (long long v = (long long)unit * blockDim.x + threadIdx.x; v < nv;
         v += (long long)nunits * blockDim.x) {
        const int ph = d.phase[v];
        if (!d.solid[ph]) {
#pragma unroll
            for (int c = 0; c < 6; ++c) { d.sig[c * nv + v] = 0.0; d.sigp[c * nv + v] = 0.0; }
            continue;
        }
        double *fx = d.sch + v;
        // y of the Green iterate, cc_y = U^T (eps - dg) - S0_y y, and the
        // pressure component of both
        double yl[5], cc[5];
        const double s5l = d.sig[5 * nv + v], g5 = -d.dgs[5 * nv + v];
        {
            double e6[5];
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                yl[c] = fx[(FCC_Y + c) * nv];
                e6[c] = d.eps[c * nv + v] - d.dgs[c * nv + v];
            }
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                double s = 0.0;
#pragma unroll
                for (int i = 0; i < 5; ++i) s = fma(fx[(FCC_U + 5 * i + c) * nv], e6[i], s);
                cc[c] = s;
            }
#pragma unroll
            for (int i = 0; i < 5; ++i)
#pragma unroll
                for (int j = i; j < 5; ++j) {
                    const double q = fx[(FCC_S0 + sym5(i, j)) * nv];
                    cc[i] = fma(-q, yl[j], cc[i]);
                    if (i != j) cc[j] = fma(-q, yl[i], cc[j]);
                }
        }
        const double cc5 = fma(-d.S0[35], s5l, g5);
        const double sn2 = fma(s5l, s5l, fcc_norm2<double>(yl));
        // sqrt(cnr)/signorm > 1e-7 (evolution.c:112) tested as cnr > 1e-14 signorm^2
        const double thr = 1e-14 * sn2;
        double y[5], yp[5], Rl[5], s5 = s5l, s5p = s5l, R5 = 0.0;
#pragma unroll
        for (int c = 0; c < 5; ++c) { y[c] = yl[c]; yp[c] = yl[c]; Rl[c] = 0.0; }
        int it = 0;
        bool converged = false;   // FCC_NR32: the start's point is taken as the solution
        (void)converged;
        if constexpr (FORM == FCC_FP64) {
            fcc_newton(d, v, cc, cc5, thr, y, s5, yp, s5p, Rl, R5, it);
        } else {
            float yf[5], ccf[5], P[15], L[15], xf[5];
            bool ok = false;
            if (FORM == FCC_NR32 || d.ir_pred) {
#pragma unroll
                for (int q = 0; q < 15; ++q) P[q] = __ldg(d.sgp32 + (long long)q * nv + v);
#pragma unroll
                for (int c = 0; c < 5; ++c) { yf[c] = d2f_rn(yl[c]); ccf[c] = d2f_rn(cc[c]); }
                // before a float-float step single precision stops at a
                // relative update of 1e-4 (its rounding floor can lie near
                // 1e-5), alone at 1e-5
                const float thr32 = (FORM == FCC_NR32 && !polish ? 1e-10f : 1e-8f) * (float)sn2;
                ok = fcc_newton_f32(d, v, ccf, thr32, FORM == FCC_NR32 ? 24 : 12, yf, P, L, it);
                if (ok && polish) {
                    ok = fcc_step_ff(d, v, yf, cc, P, L, dtgh, dtgl, xf);
                    ++it;
                } else {
#pragma unroll
                    for (int c = 0; c < 5; ++c) xf[c] = 0.0f;
                }
                if (ok) {
                    // the pressure component is linear: its root at once
                    s5 = -cc5 * d.iP55;
#pragma unroll
                    for (int c = 0; c < 5; ++c) y[c] = f2d(yf[c]) - f2d(xf[c]);
                    if (FORM == FCC_NR32) converged = !polish || fcc_norm2<float>(xf) <= (float)(1e-10 * sn2);
                }
            }
            if constexpr (FORM == FCC_IR) {
                if (!ok) it = 0;
                fcc_newton_ir(d, v, ok, L, cc, cc5, thr, y, s5, yp, s5p, Rl, R5, it);
            } else if (converged) {
                // taken as the converged point: no residual, and the stress
                // the strain rate is later evaluated at
#pragma unroll
                for (int c = 0; c < 5; ++c) yp[c] = y[c];
                s5p = s5;
            } else {
                fcc_newton(d, v, cc, cc5, thr, y, s5, yp, s5p, Rl, R5, it);
            }
        }
        // |sig - lam| and the strain-compatibility norm |Rl - S0 (sp - lam)|
        // (evolution.c:118-123)
        double ncs, nce;
        if constexpr (FORM == FCC_NR32) {
            // in single precision: they only steer the Green iteration's stop
            // test at 1e-5
            float dy[5], te[5] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            float d5 = d2f_rn(s5 - s5l), r5 = 0.0f;
#pragma unroll
            for (int c = 0; c < 5; ++c) dy[c] = d2f_rn(y[c] - yl[c]);
            ncs = (double)sqrtf(fmaf(d5, d5, fcc_norm2<float>(dy)));
            if (!converged) {   // (a point taken as converged: yp = y, no residual)
#pragma unroll
                for (int c = 0; c < 5; ++c) { dy[c] = (float)(yp[c] - yl[c]); te[c] = (float)Rl[c]; }
                d5 = (float)(s5p - s5l);
                r5 = (float)R5;
            }
#pragma unroll
            for (int i = 0; i < 5; ++i)
#pragma unroll
                for (int j = i; j < 5; ++j) {
                    const float q = __ldg(d.sch32 + (long long)sym5(i, j) * nv + v);
                    te[i] = fmaf(-q, dy[j], te[i]);
                    if (i != j) te[j] = fmaf(-q, dy[i], te[j]);
                }
            const float t5 = fmaf(-d.S0f[35], d5, r5);
            nce = (double)sqrtf(fmaf(t5, t5, fcc_dual2<float>(te)));
        } else {
            double dy[5], te[5];
#pragma unroll
            for (int c = 0; c < 5; ++c) { dy[c] = y[c] - yl[c]; te[c] = Rl[c]; }
            const double d5 = s5 - s5l;
            const double cs = fma(d5, d5, fcc_norm2<double>(dy));
#pragma unroll
            for (int c = 0; c < 5; ++c) dy[c] = yp[c] - yl[c];
#pragma unroll
            for (int i = 0; i < 5; ++i)
#pragma unroll
                for (int j = i; j < 5; ++j) {
                    const double q = reread(fx + (FCC_S0 + sym5(i, j)) * nv);
                    te[i] = fma(-q, dy[j], te[i]);
                    if (i != j) te[j] = fma(-q, dy[i], te[j]);
                }
            const double t5 = fma(-d.S0[35], s5p - s5l, R5);
            const double ce = fma(t5, t5, fcc_dual2<double>(te));
            // the mixed_ir form's norms by a Newton-Raphson square root
            // (about 1e-13 relative); the other forms' correctly rounded
            ncs = FORM == FCC_IR ? sqrt_nr(cs) : sqrt(cs);
            nce = FORM == FCC_IR ? sqrt_nr(ce) : sqrt(ce);
        }
        s_acc[0][tid] += ncs;
        s_acc[1][tid] += nce;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            double s = s5;
            if (i < 5) {
                s = 0.0;
#pragma unroll
                for (int c = 0; c < 5; ++c) s = fma(reread(fx + (FCC_U + 5 * i + c) * nv), y[c], s);
                fx[(FCC_Y + i) * nv] = y[i];
            }
            d.sig[i * nv + v] = s;
            d.sigp[i * nv + v] = i < 5 ? yp[i < 5 ? i : 0] : s5p;
            s_acc[2 + i][tid] += s;
            if (ph == 1 && !d.all_ph1) s_acc[8 + i][tid] += s;
        }
        s_it[0][tid] += it;
        s_it[1][tid] = max(s_it[1][tid], it);
    }
    // the block's partial sums: a warp takes every fourth quantity over the 128
    // thread sums (eight additions a quantity; a shuffle tree per thread over
    // all sixteen took eighty).  With one phase the phase-1 sums are the full
    // ones again and are left out.
    __syncthreads();
    const int lane = tid & 31, nq = d.all_ph1 ? 8 : 14;
    double *out = d.part + (long long)unit * VOCE_NPART;
    for (int q = tid >> 5; q < nq; q += VOCE_NR_THREADS / 32) {
        double s = (s_acc[q][lane] + s_acc[q][lane + 32]) + (s_acc[q][lane + 64] + s_acc[q][lane + 96]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) out[q] = s;
    }
    if (tid < 32) {
        const int n = s_it[0][lane] + s_it[0][lane + 32] + s_it[0][lane + 64] + s_it[0][lane + 96];
        const int m = max(max(s_it[1][lane], s_it[1][lane + 32]), max(s_it[1][lane + 64], s_it[1][lane + 96]));
        const int sn = __reduce_add_sync(0xffffffffu, n), sm = __reduce_max_sync(0xffffffffu, m);
        if (lane < 2) out[14 + lane] = (double)(lane ? sm : sn);
    }
    __syncthreads();
}


__device__ double vm_strain(const double *t)  // VonMises, evolution.c:243-262
{
    double tr = t[0] + t[4] + t[8], vm = 0.0;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            double x = (t[3 * a + b] + t[3 * b + a]) / 2. - (double)(a == b) * tr / 3.0;
            vm += x * x;
        }
    return sqrt(2. / 3. * vm);
}

// Component p of (00, 11, 22, 12, 02, 01) of a 6-vector b: b_to_t6 with the
// lane's coefficients, three products whatever p is
__device__ __forceinline__ double t6_component(int p, const double *b)
{
    const double ca = p == 0 ? -RSQ2 : p == 2 ? 0.0 : RSQ2;
    const double cb = p < 2 ? -RSQ6 : p == 2 ? 2.0 * RSQ6 : 0.0, cc = p < 3 ? RSQ3 : 0.0;
    return fma(cc, b[5], fma(cb, b[1], ca * b[p < 3 ? 0 : p - 1]));
}

// Errors, volume averages, mixed-BC macro correction and the convergence
// decision (evolution.c:401-431, get_smacro :170-241), from the reduced
// partial sums tot.  One SM runs this and waits for its slow FP64 operations
// (64 cycles of a quarter's pipe each, at any number of lanes), so what counts
// is the number of instructions on the longest chain: warp 0 takes the error
// norms (the von Mises norm straight from the 6-vector, one reciprocal square
// root for it and for the strain normalisation, no division), warp 1 the
// averages and the mixed-BC correction, a value per lane with lane-wise
// coefficients.  Measured by events at 16^3 / 64^3 (32 / 456 partial sums):
// 18.4 / 20.5 -> 8.9 / 14.3 us.  m is the block's shared-memory copy.
__device__ void finalize_iter_body(const RveDesc &d, MacroDev *m, const double *tot)
{
    __shared__ double s_dg[9], s_t6[6], s_act[2][9];
    __shared__ int s_more;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int it = m->iter, istep = m->istep;
    if (warp == 0) {
        // lane 0: s_vm and Err_s, lane 1: s_vm1, lane 2: Err_e
        const double e_vm = m->e_vm;
        // the mixed form's Newton ran in single precision alone this iteration
        // (the predicate nr_unit used): it may not end the increment
        const bool fp32_only = d.nr32 && (m->first_iter || fmax(fabs(m->Err_e), fabs(m->Err_s)) > VOCE_POLISH_ERR);
        const double *b = tot + (lane == 1 ? 8 : 2);
        double x = lane == 2 ? (fabs(e_vm) > 1E-5 ? e_vm * e_vm : 1.0)
                             : 1.5 * (((b[0] * b[0] + b[1] * b[1]) + (b[2] * b[2] + b[3] * b[3])) + b[4] * b[4]);
        const double r = rsqrt(x);
        // sum wgt / (wgt sqrt(x)), and sum wgt / e_vm
        const double err = lane == 2 ? (tot[1] * d.wgt) * r : tot[0] * r;
        // sqrt(x) as x / sqrt(x): 0 and infinity are their own roots (x is never
        // negative, NaN stays; tested on the integer pipe)
        const long long xb = __double_as_longlong(x);
        const double root = xb == 0 || xb == 0x7ff0000000000000LL ? x : x * r;
        const double svm = root * (lane == 1 ? d.wgt_ratio : d.wgt);
        const double Err_s = __shfl_sync(0xffffffffu, err, 0), Err_e = __shfl_sync(0xffffffffu, err, 2);
        const double s_vm = __shfl_sync(0xffffffffu, svm, 0);
        const bool more = (it + 1 < d.iter_max) &&
                          (fp32_only || fmax(fabs(Err_s), fabs(Err_e)) > fabs(d.err_tol));
        if (lane == 1) m->s_vm1 = svm;
        if (lane == 0) {
            m->s_vm = svm;
            m->Err_e = Err_e;
            m->Err_s = Err_s;
            m->iter = it + 1;
            m->iter_total += 1;
            m->nr_total += tot[14];
            m->nr_max = max(m->nr_max, (int)tot[15]);
            m->first_iter = 0;
            m->pending_prelude = 0;
            m->converged = more ? 0 : 1;
            s_more = more;
        }
        if (it < d.iter_max && lane < VOCE_ITLOG) {
            const int slot = (istep - 1) % d.incr_cap;
            double *lg = d.itlog + ((long long)slot * d.iter_max + it) * VOCE_ITLOG;
            // Err_e, Err_s, s_vm, Newton steps, the raw sums of the strain-compatibility and
            // stress-change norms, the sum of sigma (basis)
            const int from[VOCE_ITLOG] = {0, 0, 0, 14, 1, 0, 2, 3, 4, 5, 6, 7};
            lg[lane] = lane == 0 ? Err_e : lane == 1 ? Err_s : lane == 2 ? s_vm : tot[from[lane]];
        }
    } else if (warp == 1) {
        // lane q < 9: SigAvg[q]; lane 9 + q: SigAvg1[q] (phase 1)
        if (lane < 18) {
            const int q = lane < 9 ? lane : lane - 9;
            const int p6[9] = {0, 5, 4, 5, 1, 3, 4, 3, 2};
            const double v = t6_component(p6[q], tot + (lane < 9 ? 2 : 8)) * (lane < 9 ? d.wgt : d.wgt_ratio);
            if (lane < 9) m->SigAvg[q] = v;
            else m->SigAvg1[q] = v;
        }
        // entries get_smacro leaves alone keep their value
        if (lane < 9) s_dg[lane] = m->dDisGradAvg[lane];
        __syncwarp();
        const int I6[6] = {0, 1, 2, 1, 0, 0}, J6[6] = {0, 1, 2, 2, 2, 1};
        // lane i < 6: dDisGradAvg at component i (get_smacro); the stress flags are 0 or 1
        if (lane < 6) {
            const int ii = I6[lane], jj = J6[lane];
            double s = 0.0;
            if (d.vflag[lane] == 0)
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    const int kk = I6[k], ll = J6[k];
                    if (d.sflag[k])
                        s = fma(d.S0t[((ii * 3 + jj) * 3 + kk) * 3 + ll], d.Scauchy[kk * 3 + ll] - m->SigAvg[kk * 3 + ll], s);
                }
            s_dg[ii * 3 + jj] = s;
        }
        __syncwarp();
        if (lane < 9) {
            const double dg = s_dg[lane];
            m->dDisGradAvg[lane] = dg;
            m->dDisGradAvg_acum[lane] += dg;
        }
        // its symmetric part in the 6-vector basis, for the next update
        if (lane < 6) s_t6[lane] = 0.5 * (s_dg[I6[lane] * 3 + J6[lane]] + s_dg[J6[lane] * 3 + I6[lane]]);
        __syncwarp();
        if (lane < 6) {
            const double k0 = lane == 0 ? -RSQ2 : lane == 1 ? -RSQ6 : lane == 5 ? RSQ3 : 0.0;
            const double k1 = lane == 0 ? RSQ2 : k0, k2 = lane == 1 ? 2.0 * RSQ6 : lane == 5 ? RSQ3 : 0.0;
            const bool shear = lane >= 2 && lane < 5;
            m->ddg6[lane] = shear ? 2.0 * RSQ2 * s_t6[lane + 1] : fma(k2, s_t6[2], fma(k1, s_t6[1], k0 * s_t6[0]));
        }
    }
    __syncthreads();
    if (s_more || warp != 0) return;
    // epilogue macro bookkeeping (evolution.c:438-461); lane q < 9 entry q
    if (lane < 9) {
        const int q = lane;
        const double act = m->DisGradAvg[q] + m->dDisGradAvg_acum[q];
        const double vga = (act - m->DisGradAvg_t[q]) / d.dt;
        s_act[0][q] = act;
        s_act[1][q] = vga;
        m->VelGradAvg[q] = vga;
        m->DisGradAvg_t[q] = act;
        m->DisGradAvg[q] = act + d.Udot[q] * d.dt;
        // the prelude of this increment used the previous DisGradAvg_actual
        m->DGA_prev[q] = m->DisGradAvg_actual[q];
        m->DisGradAvg_actual[q] = act;
    }
    __syncwarp();
    // lane 0: e_vm of DisGradAvg_actual, lane 1: d_vm of VelGradAvg
    if (lane < 2) {
        const double v = vm_strain(s_act[lane]);
        if (lane == 0) m->e_vm = v;
        else m->d_vm = v;
    }
    if (lane == 0) {
        // the displacement gradient received every dDisGradAvg of this
        // increment except the last one, which get_smacro computes after the
        // final update (evolution.c:391 vs :418): only those enter VelGrad
        double a[9];
        for (int q = 0; q < 9; ++q) a[q] = m->dDisGradAvg_acum[q] - s_dg[q];
        m->acum_a[0] = 0.5 * (a[5] - a[7]);
        m->acum_a[1] = 0.5 * (a[2] - a[6]);
        m->acum_a[2] = 0.5 * (a[1] - a[3]);
    }
    __syncwarp();
}


// Harden one voxel: harden() body (constitutive.c:261-305)
__device__ void harden_voxel(const RveDesc &d, long long v, const double *gd)
{
    const long long nv = d.nv;
    const double dt = d.dt;
    const double gamtot = d.gamacum[v];
    double deltgam = 0.0;
    for (int i = 0; i < d.nsys; ++i) d.gtot[i * nv + v] = d.gtot[i * nv + v] + gd[i] * dt;
    for (int i = 0; i < d.nsys; ++i) deltgam += fabs(gd[i]) * dt;
    for (int i = 0; i < d.nsys; ++i) {
        double dtau = 0.;
        for (int j = 0; j < d.nsys; ++j) dtau += d.hard[i * VOCE_NS + j] * fabs(gd[j]) * dt;
        const double tau0 = d.tau0[i], tau1 = d.tau1[i], th0 = d.thet0[i], th1 = d.thet1[i];
        const double tiny = 1.E-4 * tau0;
        double voce = 0.0;
        if (fabs(th0) > tiny) {
            voce = th1 * deltgam;
            if (fabs(tau1) > tiny) {
                const double fact = fabs(th0 / tau1);
                const double exp_ini = exp(-1.0 * gamtot * fact);
                const double exp_del = exp(-1.0 * deltgam * fact);
                voce += -1. * (fact * tau1 - th1) / fact * exp_ini * (exp_del - 1.0) -
                        th1 / fact * exp_ini * (exp_del * ((gamtot + deltgam) * fact + 1.0) - (gamtot * fact + 1.0));
            }
        }
        const double inc = dtau * voce / deltgam;
        const double c0 = d.crss[(2 * i) * nv + v] + inc;
        const double c1 = d.crss[(2 * i + 1) * nv + v] + inc;
        d.crss[(2 * i) * nv + v] = c0;
        d.crss[(2 * i + 1) * nv + v] = c1;
        d.itau[itau_col(d, i, 0) * nv + v] = 1.0 / c0;
        d.itau[itau_col(d, i, 1) * nv + v] = 1.0 / c1;
        if (d.itau32) {
            put_pair(d.itau32, d.itau_lo, itau_col(d, i, 0) * nv + v, 1.0 / c0);
            put_pair(d.itau32, d.itau_lo, itau_col(d, i, 1) * nv + v, 1.0 / c1);
        }
    }
    d.gamacum[v] = gamtot + deltgam;
}

// Orientation() (constitutive.c:117-169)
__device__ void orientation(double (&tran)[3][3], double (&rot)[3][3])
{
    double w[3] = {rot[2][1], rot[0][2], rot[1][0]};
    double wn = sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    double wt = tan(wn / 2.0);
    if (fabs(wn) < 1E-6) wn = 1.0;
    for (int i = 0; i < 3; ++i) w[i] *= wt / wn;
    const double om[3][3] = {{0., -1. * w[2], w[1]}, {w[2], 0., -1. * w[0]}, {-1. * w[1], w[0], 0.}};
    double om2[3][3], tn[3][3];
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            double s = 0.0;
            for (int i = 0; i < 3; ++i) s += om[a][i] * om[i][b];
            om2[a][b] = s;
        }
    wt = wt * wt;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) rot[a][b] = (double)(a == b) + 2. * (om[a][b] + om2[a][b]) / (1. + wt);
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            double s = 0.0;
            for (int i = 0; i < 3; ++i) s += rot[a][i] * tran[i][b];
            tn[a][b] = s;
        }
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) tran[a][b] = tn[a][b];
}

// increment epilogue (evolution.c:433-530; update_orient constitutive.c:171-248; harden :250-310;
// update_schmid kinematics.c:426-459)
__device__ void incr_end_unit(const RveDesc &d, int unit, int nunits)
{
    double acc[VOCE_NPART];
    for (int q = 0; q < VOCE_NPART; ++q) acc[q] = 0.0;
    const MacroDev *m = d.macro;
    const long long nv = d.nv;
    const double dt = d.dt;
    const int istep = m->istep;
    const bool upd = d.update_flag == 1 && istep > 1;
    const bool hrd = d.hard_flag == 1 && istep > 2;
    // under creep the prelude set DisGrad to the previous DisGradAvg_actual
    double dga_start_c[3];
    {
        const double *p = m->DGA_prev;
        dga_start_c[0] = 0.5 * (p[5] - p[7]);
        dga_start_c[1] = 0.5 * (p[2] - p[6]);
        dga_start_c[2] = 0.5 * (p[1] - p[3]);
    }
    for (long long v = (long long)unit * blockDim.x + threadIdx.x; v < nv;
         v += (long long)nunits * blockDim.x) {
        const int ph = d.phase[v];
        // antisymmetric displacement gradient bookkeeping
        double rl[3];
        for (int c = 0; c < 3; ++c) {
            const double prev = d.dga[c * nv + v];
            const double st = d.creep ? dga_start_c[c] : prev + d.ua[c] * dt;
            const double en = st + m->acum_a[c] + d.rotl[c * nv + v];
            rl[c] = (en - prev) / dt;
            d.dga[c * nv + v] = en;
        }
        double e5[5] = {0, 0, 0, 0, 0}, ed[5] = {0, 0, 0, 0, 0};
        for (int c = 0; c < 5; ++c) e5[c] = d.eps[c * nv + v];
        if (d.solid[ph]) {
            double sp[6], gd[VOCE_NS], tx[VOCE_NS];
            for (int c = 0; c < 6; ++c) sp[c] = d.sigp[c * nv + v];
            flow_rule<false, true, double>(d, v, sp, ed, (double *)nullptr, gd, tx);
            for (int k = 0; k < d.nsys; ++k) {
                d.gamdot[k * nv + v] = gd[k];
                d.taux[k * nv + v] = tx[k];
            }
            for (int c = 0; c < 5; ++c) d.edot[c * nv + v] = ed[c];
            // SVM from the new stress, EVM from the total strain of the last
            // Newton iteration (evolution.c:134-155)
            double s6[6], s9[9], te6[6], t9[9];
            for (int c = 0; c < 6; ++c) s6[c] = d.sig[c * nv + v];
            sym9_from_b(s6, s9);
            {
                double tr = s9[0] + s9[4] + s9[8], acc2 = 0.0;
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) {
                        double x = s9[3 * a + b] - (double)(a == b) * tr / 3.0;
                        acc2 += x * x;
                    }
                d.svm[v] = sqrt(3. / 2. * acc2);
            }
            for (int i = 0; i < 6; ++i) {
                double s = (i < 5 ? e5[i] + ed[i] * dt : 0.0);
                for (int j = 0; j < 6; ++j) s += d.sg[(long long)sym6(i, j) * nv + v] * sp[j];
                te6[i] = s;
            }
            sym9_from_b(te6, t9);
            {
                double tr = t9[0] + t9[4] + t9[8], acc2 = 0.0;
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) {
                        double x = t9[3 * a + b] - (double)(a == b) * tr / 3.0;
                        acc2 += x * x;
                    }
                d.evm[v] = sqrt(2. / 3. * acc2);
            }
            // Eps += Edot dt (evolution.c:464-468)
            for (int c = 0; c < 5; ++c) {
                e5[c] = e5[c] + ed[c] * dt;
                d.eps[c * nv + v] = e5[c];
            }
            // resolved shear stresses for the diagnostics, with the Schmid
            // tensors of this increment (the reorientation below replaces them)
            double rss[VOCE_NS];
            if (hrd)
                for (int k = 0; k < d.nsys; ++k) {
                    const double *sc = d.sch + (long long)(5 * k) * nv + v;
                    rss[k] = sc[0] * s6[0] + sc[nv] * s6[1] + sc[2 * nv] * s6[2] + sc[3 * nv] * s6[3] +
                             sc[4 * nv] * s6[4];
                }
            if (upd) {
                double T[3][3], RL[3][3], Lp[3][3], RS[3][3], Rot[3][3];
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) {
                        T[a][b] = d.tm[(3 * a + b) * nv + v];
                        Lp[a][b] = 0.0;
                    }
                RL[0][0] = RL[1][1] = RL[2][2] = 0.0;
                RL[1][2] = rl[0]; RL[2][1] = -rl[0];
                RL[0][2] = rl[1]; RL[2][0] = -rl[1];
                RL[0][1] = rl[2]; RL[1][0] = -rl[2];
                for (int s = 0; s < d.nsys; ++s) {
                    double bs[3], ns[3];
                    for (int a = 0; a < 3; ++a) {
                        bs[a] = 0.0; ns[a] = 0.0;
                        for (int b = 0; b < 3; ++b) {
                            bs[a] += T[a][b] * d.bb[3 * s + b];
                            ns[a] += T[a][b] * d.bn[3 * s + b];
                        }
                    }
                    for (int a = 0; a < 3; ++a)
                        for (int b = 0; b < 3; ++b) Lp[a][b] += bs[a] * ns[b] * gd[s];
                }
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) RS[a][b] = (Lp[a][b] - Lp[b][a]) / 2.;
                acc[12] += sqrt(RS[2][1] * RS[2][1] + RS[0][2] * RS[0][2] + RS[1][0] * RS[1][0]) * d.wgt;
                acc[13] += sqrt(RL[2][1] * RL[2][1] + RL[0][2] * RL[0][2] + RL[1][0] * RL[1][0]) * d.wgt;
                const double Ua[3][3] = {{0.0, d.ua[2], d.ua[1]}, {-d.ua[2], 0.0, d.ua[0]}, {-d.ua[1], -d.ua[0], 0.0}};
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) Rot[a][b] = (Ua[a][b] + RL[a][b] - RS[a][b]) * dt;
                orientation(T, Rot);
                for (int a = 0; a < 3; ++a)
                    for (int b = 0; b < 3; ++b) d.tm[(3 * a + b) * nv + v] = T[a][b];
                schmid_from_tm(d, v, T);
            }
            if (hrd) {
                harden_voxel(d, v, gd);
                // rho_rss, rho_crss, work_p (evolution.c:509-529)
                const double ref = 0.35 * 47.565 * 0.256;
                double rr = 0.0, rc = 0.0, wp = 0.0;
                for (int k = 0; k < d.nsys; ++k) {
                    const double a = rss[k] / ref, b = d.crss[(2 * k) * nv + v] / ref;
                    rr += a * a;
                    rc += b * b;
                    wp += fabs(d.gtot[k * nv + v] * rss[k]);
                }
                d.diag[v] = rr;
                d.diag[nv + v] = rc;
                d.diag[2 * nv + v] = wp;
            }
        } else {
            for (int c = 0; c < 5; ++c) d.edot[c * nv + v] = 0.0;
        }
        for (int c = 0; c < 5; ++c) { acc[c] += e5[c]; acc[6 + c] += ed[c]; }
    }
    block_partials(acc, d.part + (long long)unit * VOCE_NPART);
}


// tan x to rounding for the small half angles of a reorientation (the Taylor
// series through x^9; the next term is below 1e-20 of x for |x| < 2^-6)
__device__ __forceinline__ double tan_small(double x)
{
    if (fabs(x) >= 0.015625) return tan(x);
    const double q = x * x;
    double p = fma(62.0 / 2835.0, q, 17.0 / 315.0);
    p = fma(p, q, 2.0 / 15.0);
    p = fma(p, q, 1.0 / 3.0);
    return fma(x * q, p, x);
}

// ---------------------------------------------------------------------------
// The increment epilogue of an RVE of the {111}<110> family: incr_end_unit in
// crystal axes, every per-system quantity in canonical order and in registers
// (d.file gives the system's place in the arrays that keep file order).
// Against incr_end_unit, which is bound by the FP64 pipe and by local memory:
// the plastic spin is summed as the 3 components of its axial vector in
// crystal axes and turned once (it was 12 products of 3 x 3 matrices), the
// reorientation works on axial vectors, and the Voce factor, the same for all
// systems of a slip mode, is computed once instead of twelve times.
// Third increment (reorientation and hardening): 35 ms at 256^3 (mixed_ir),
// 4.3 ms at 128^3 (FP64); the whole 256^3 increment of eight Green iterations
// went from 298 to 202 ms.
// ---------------------------------------------------------------------------
__device__ void incr_end_fcc_unit(const RveDesc &d, int unit, int nunits)
{
    __shared__ double s_acc[VOCE_NPART][VOCE_NR_THREADS];
    const int tid = threadIdx.x;
#pragma unroll
    for (int q = 0; q < VOCE_NPART; ++q) s_acc[q][tid] = 0.0;
    const MacroDev *m = d.macro;
    const long long nv = d.nv;
    const double dt = d.dt, idt = 1.0 / dt, wgt = d.wgt;
    const int istep = m->istep;
    const bool upd = d.update_flag == 1 && istep > 1;
    const bool hrd = d.hard_flag == 1 && istep > 2;
    // under creep the prelude set DisGrad to the previous DisGradAvg_actual
    const double *pg = m->DGA_prev;
    const double dga0[3] = {0.5 * (pg[5] - pg[7]), 0.5 * (pg[2] - pg[6]), 0.5 * (pg[1] - pg[3])};
    for (long long v = (long long)unit * blockDim.x + threadIdx.x; v < nv;
         v += (long long)nunits * blockDim.x) {
        // antisymmetric displacement gradient bookkeeping
        double rl[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double prev = d.dga[c * nv + v];
            const double st = d.creep ? dga0[c] : prev + d.ua[c] * dt;
            const double en = st + m->acum_a[c] + d.rotl[c * nv + v];
            rl[c] = (en - prev) * idt;
            d.dga[c * nv + v] = en;
        }
        double e5[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) e5[c] = d.eps[c * nv + v];
        if (!d.solid[d.phase[v]]) {
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                d.edot[c * nv + v] = 0.0;
                s_acc[c][tid] += e5[c];
            }
            continue;
        }
        double *fx = d.sch + v;
        double gd[VOCE_NS];
        {
            double y[5], E[5], it[VOCE_NS], p[VOCE_NS];
#pragma unroll
            for (int c = 0; c < 5; ++c) y[c] = d.sigp[c * nv + v];
            fcc_rss12<double>(y, gd);
#pragma unroll
            for (int k = 0; k < VOCE_NS; ++k) {
                it[k] = d.itau[(long long)(2 * k + (__double2hiint(gd[k]) < 0)) * nv + v];
                gd[k] *= it[k];
            }
            fcc_pow<VOCE_NS, double>(gd, d.ipow_n - 1, p);
            const double g0 = d.gam0[0], n0 = d.nrs[0];
#pragma unroll
            for (int k = 0; k < VOCE_NS; ++k) {
                const double q = g0 * p[k];
                gd[k] *= q;
                const long long o = d.file[k] * nv + v;
                d.gamdot[o] = d.flip[d.file[k]] ? -gd[k] : gd[k];
                d.taux[o] = (q * it[k]) * n0;
            }
            fcc_edot12<double>(gd, E);
            // strain rate and penultimate stress in sample axes, the total
            // strain there (EVM: evolution.c:134-155)
            double sp[5], te[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                double s = 0.0, e = 0.0;
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    const double u = fx[(FCC_U + 5 * i + c) * nv];
                    s = fma(u, y[c], s);
                    e = fma(u, E[c] * (1.0 / fcc_w2(c)), e);
                }
                sp[i] = s;
                d.edot[i * nv + v] = e;
                s_acc[6 + i][tid] += e;
                e5[i] = fma(e, dt, e5[i]);   // Eps += Edot dt (evolution.c:464-468)
                d.eps[i * nv + v] = e5[i];
                s_acc[i][tid] += e5[i];
                te[i] = e5[i];
            }
#pragma unroll
            for (int i = 0; i < 5; ++i)
#pragma unroll
                for (int j = i; j < 5; ++j) {
                    const double q = d.sg[(long long)sym6(i, j) * nv + v];
                    te[i] = fma(q, sp[j], te[i]);
                    if (i != j) te[j] = fma(q, sp[i], te[j]);
                }
            double t2 = 0.0;
#pragma unroll
            for (int i = 0; i < 5; ++i) t2 = fma(te[i], te[i], t2);
            d.evm[v] = sqrt(2. / 3. * t2);
        }
        double rss[VOCE_NS];   // resolved shears of the new stress, for the diagnostics
        {
            double y[5];
#pragma unroll
            for (int c = 0; c < 5; ++c) y[c] = fx[(FCC_Y + c) * nv];
            d.svm[v] = sqrt(3. / 2. * fcc_norm2<double>(y));
            fcc_rss12<double>(y, rss);
        }
        if (upd) {
            // update_orient (constitutive.c:171-248) with axial vectors
            // (w0, w1, w2) = (W21, W02, W10)
            double T[3][3], wc[3] = {0.0, 0.0, 0.0}, w[3];
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) T[a][b] = d.tm[(3 * a + b) * nv + v];
#pragma unroll
            for (int k = 0; k < VOCE_NS; ++k)
#pragma unroll
                for (int a = 0; a < 3; ++a) wc[a] = fma(d.skew[3 * k + a], gd[k], wc[a]);
            const double lw[3] = {-rl[0], rl[1], -rl[2]}, uw[3] = {-d.ua[0], d.ua[1], -d.ua[2]};
            double n2 = 0.0, l2 = 0.0, r2 = 0.0;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const double ws = T[a][0] * wc[0] + T[a][1] * wc[1] + T[a][2] * wc[2];
                n2 = fma(ws, ws, n2);
                l2 = fma(lw[a], lw[a], l2);
                w[a] = ((uw[a] + lw[a]) - ws) * dt;
                r2 = fma(w[a], w[a], r2);
            }
            s_acc[12][tid] += sqrt(n2) * wgt;
            s_acc[13][tid] += sqrt(l2) * wgt;
            // Orientation (constitutive.c:117-169): T := (I + 2 (om + om^2) / (1 + t^2)) T
            const double wn = sqrt(r2), wt = tan_small(0.5 * wn);
            const double f = wn < 1E-6 ? wt : wt / wn, h = 2.0 / fma(wt, wt, 1.0);
#pragma unroll
            for (int a = 0; a < 3; ++a) w[a] *= f;
            const double w2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                // om x = w x x, om^2 x = w (w.x) - x |w|^2
                const double x0 = T[0][b], x1 = T[1][b], x2 = T[2][b];
                const double dot = w[0] * x0 + w[1] * x1 + w[2] * x2;
                T[0][b] = fma(h, (w[1] * x2 - w[2] * x1) + (w[0] * dot - x0 * w2), x0);
                T[1][b] = fma(h, (w[2] * x0 - w[0] * x2) + (w[1] * dot - x1 * w2), x1);
                T[2][b] = fma(h, (w[0] * x1 - w[1] * x0) + (w[2] * dot - x2 * w2), x2);
            }
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) d.tm[(3 * a + b) * nv + v] = T[a][b];
            fcc_frame(d, v, T);
        }
        if (hrd) {
            // harden (constitutive.c:261-305) and rho_rss, rho_crss, work_p
            // (evolution.c:509-529)
            const double gamtot = d.gamacum[v];
            double deltgam = 0.0, rr = 0.0, rc = 0.0, wp = 0.0;
#pragma unroll
            for (int k = 0; k < VOCE_NS; ++k) {
                const int fk = d.file[k];
                const double sg = d.flip[fk] ? -1.0 : 1.0;
                const double gt = fma(sg * gd[k], dt, d.gtot[fk * nv + v]);
                d.gtot[fk * nv + v] = gt;
                gd[k] = fabs(gd[k]) * dt;
                deltgam += gd[k];
                rr = fma(rss[k], rss[k], rr);
                wp += fabs(gt * rss[k]);
            }
            const double tau1 = d.tau1[0], th0 = d.thet0[0], th1 = d.thet1[0];
            const double tiny = 1.E-4 * d.tau0[0];
            double voce = 0.0;
            if (fabs(th0) > tiny) {
                voce = th1 * deltgam;
                if (fabs(tau1) > tiny) {
                    const double fact = fabs(th0 / tau1);
                    const double exp_ini = exp(-1.0 * gamtot * fact);
                    const double exp_del = exp(-1.0 * deltgam * fact);
                    voce += -1. * (fact * tau1 - th1) / fact * exp_ini * (exp_del - 1.0) -
                            th1 / fact * exp_ini * (exp_del * ((gamtot + deltgam) * fact + 1.0) - (gamtot * fact + 1.0));
                }
            }
            const double rate = voce / deltgam;
#pragma unroll
            for (int i = 0; i < VOCE_NS; ++i) {
                const int fi = d.file[i];
                double dtau = 0.0;
#pragma unroll
                for (int j = 0; j < VOCE_NS; ++j) dtau = fma(d.hard[fi * VOCE_NS + d.file[j]], gd[j], dtau);
                const double inc = dtau * rate;
                const double c0 = d.crss[(2 * fi) * nv + v] + inc, c1 = d.crss[(2 * fi + 1) * nv + v] + inc;
                d.crss[(2 * fi) * nv + v] = c0;
                d.crss[(2 * fi + 1) * nv + v] = c1;
                // the two directions' CRSS are mostly one value
                const double i0 = 1.0 / c0, i1 = c1 == c0 ? i0 : 1.0 / c1;
                const int f0 = 2 * i + d.flip[fi], f1 = 2 * i + 1 - d.flip[fi];   // itau_col(fi, 0), (fi, 1)
                d.itau[f0 * nv + v] = i0;
                d.itau[f1 * nv + v] = i1;
                if (d.itau32) {
                    put_ff(d.itau32, d.itau_lo, f0 * nv + v, i0);
                    put_ff(d.itau32, d.itau_lo, f1 * nv + v, i1);
                }
                rc = fma(c0, c0, rc);
            }
            d.gamacum[v] = gamtot + deltgam;
            const double ref = 0.35 * 47.565 * 0.256;
            d.diag[v] = rr * (1.0 / (ref * ref));
            d.diag[nv + v] = rc * (1.0 / (ref * ref));
            d.diag[2 * nv + v] = wp;
        }
    }
    double acc[VOCE_NPART];
#pragma unroll
    for (int q = 0; q < VOCE_NPART; ++q) acc[q] = s_acc[q][tid];
    block_partials(acc, d.part + (long long)unit * VOCE_NPART);
}


// increment prelude (evolution.c:306-318): DisGrad += Udot dt, or, under
// creep, DisGrad := DisGradAvg_actual of the previous increment
__device__ void prelude_unit(const RveDesc &d, int unit, int nunits)
{
    const MacroDev *m = d.macro;
    double set6[6];
    {
        const double *a = m->DisGradAvg_actual;
        double t6[6] = {a[0], a[4], a[8], 0.5 * (a[5] + a[7]), 0.5 * (a[2] + a[6]), 0.5 * (a[1] + a[3])};
        t6_to_b<double>(t6, set6);
    }
    const long long nv = d.nv;
    // component by component, the ones that do not change left out
    for (int c = 0; c < 6; ++c) {
        const double add = d.u6[c] * d.dt, set = set6[c];
        if (!d.creep && add == 0.0) continue;
        double *g = d.dgs + c * nv;
#pragma unroll 4
        for (long long v = (long long)unit * blockDim.x + threadIdx.x; v < nv; v += (long long)nunits * blockDim.x)
            g[v] = d.creep ? set : g[v] + add;
    }
}


__device__ void finalize_incr_body(const RveDesc &d, MacroDev *m, const double *tot)
{
    if (threadIdx.x != 0) return;
    double e6[6] = {tot[0], tot[1], tot[2], tot[3], tot[4], 0.0};
    double d6[6] = {tot[6], tot[7], tot[8], tot[9], tot[10], 0.0};
    double e9[9], d9[9];
    sym9_from_b(e6, e9);
    sym9_from_b(d6, d9);
    double evmp = 0.0, dvmp = 0.0;
    for (int q = 0; q < 9; ++q) {
        m->EpsAvg[q] = e9[q] * d.wgt;
        m->EdotAvg[q] = d9[q] * d.wgt;
        evmp += m->EpsAvg[q] * m->EpsAvg[q];
        dvmp += m->EdotAvg[q] * m->EdotAvg[q];
    }
    m->evmp = sqrt(2. / 3. * evmp);
    m->dvmp = sqrt(2. / 3. * dvmp);
    m->rsl = tot[12];
    m->rlc = tot[13];
    const int k = m->istep - 1;
    if (k >= 0 && d.incr_cap > 0) {
        IncrDev *r = d.incr + (k % d.incr_cap);
        r->istep = m->istep;
        r->iters = m->iter;
        r->iter_total = m->iter_total;
        r->nr_max = m->nr_max;
        r->e_vm = m->e_vm; r->evmp = m->evmp; r->d_vm = m->d_vm; r->dvmp = m->dvmp;
        r->s_vm = m->s_vm; r->s_vm1 = m->s_vm1;
        for (int q = 0; q < 9; ++q) {
            r->sig_avg[q] = m->SigAvg[q];
            r->sig_avg1[q] = m->SigAvg1[q];
            r->eps_avg[q] = m->EpsAvg[q];
            r->edot_avg[q] = m->EdotAvg[q];
            r->disgrad_avg[q] = m->DisGradAvg_actual[q];
        }
        r->err_e = m->Err_e; r->err_s = m->Err_s;
        r->rsl = m->rsl; r->rlc = m->rlc;
        r->nr_total = m->nr_total;
    }
    // reset for the next increment (evolution.c:330-340)
    m->istep += 1;
    if (m->istep > m->target) { m->active = 0; m->pending_prelude = 0; }
    else m->pending_prelude = 1;
    m->iter = 0;
    m->converged = 0;
    m->first_iter = 1;
    m->nr_max = 0;
    m->nr_total = 0.0;
    m->Err_e = 2. * d.err_tol;
    m->Err_s = 2. * d.err_tol;
    for (int q = 0; q < 9; ++q) { m->dDisGradAvg[q] = 0.0; m->dDisGradAvg_acum[q] = 0.0; }
    for (int q = 0; q < 6; ++q) m->ddg6[q] = 0.0;
    for (int q = 0; q < 3; ++q) m->acum_a[q] = 0.0;
}


// fields in the reference's layouts, for download
__global__ void k_field_out(RveDesc d, int field, double *out)
{
    const long long nv = d.nv;
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < nv;
         v += (long long)gridDim.x * blockDim.x) {
        double b6[6] = {0, 0, 0, 0, 0, 0}, t9[9], t6[6];
        switch (field) {
        case 0: case 20:
            for (int c = 0; c < 6; ++c) b6[c] = d.sig[c * nv + v];
            break;
        case 1:
            for (int c = 0; c < 5; ++c) b6[c] = d.eps[c * nv + v];
            break;
        case 2: case 21:
            for (int c = 0; c < 5; ++c) b6[c] = d.edot[c * nv + v];
            break;
        case 3:
            for (int c = 0; c < 6; ++c) b6[c] = d.dgs[c * nv + v];
            break;
        default: break;
        }
        switch (field) {
        case 0: case 1: case 2:
            sym9_from_b(b6, t9);
            for (int q = 0; q < 9; ++q) out[9 * v + q] = t9[q];
            break;
        case 3: {
            sym9_from_b(b6, t9);
            const double a0 = d.dga[v], a1 = d.dga[nv + v], a2 = d.dga[2 * nv + v];
            t9[5] += a0; t9[7] -= a0;
            t9[2] += a1; t9[6] -= a1;
            t9[1] += a2; t9[3] -= a2;
            for (int q = 0; q < 9; ++q) out[9 * v + q] = t9[q];
            break;
        }
        case 4:
            for (int q = 0; q < 9; ++q) out[9 * v + q] = d.tm[q * nv + v];
            break;
        case 5:
            for (int k = 0; k < VOCE_NS; ++k) out[VOCE_NS * v + k] = d.crss[(2 * k) * nv + v];
            break;
        case 6:
            for (int k = 0; k < VOCE_NS; ++k) out[VOCE_NS * v + k] = d.gamdot[k * nv + v];
            break;
        case 7: out[v] = d.gamacum[v]; break;
        case 8: out[v] = d.svm[v]; break;
        case 9: out[v] = d.evm[v]; break;
        case 10:
            for (int k = 0; k < VOCE_NS; ++k) out[VOCE_NS * v + k] = d.gtot[k * nv + v];
            break;
        case 11:
            for (int k = 0; k < VOCE_NS; ++k) out[VOCE_NS * v + k] = d.taux[k * nv + v];
            break;
        case 12: case 13: case 14: out[v] = d.diag[(field - 12) * nv + v]; break;
        case 20: case 21:
            b_to_t6<double>(b6, t6);
            for (int c = 0; c < 6; ++c) out[(long long)c * nv + v] = t6[c];
            break;
        default: break;
        }
    }
}


// resident blocks of 128 threads per SM the single-precision Newton kernel
// (kb_nr<true>) is compiled for (register budget 65536 / (128 x blocks))
#ifndef VOCE_NR_MIXED_BLOCKS
#define VOCE_NR_MIXED_BLOCKS 3
#endif

// CHORD: the FP64 Newton may take chord steps (VOCE_PREC_MIXED plans; each
// RVE's d.chord decides); the FP64 form's instance is the exact-Jacobian one
// IR: the VOCE_PREC_MIXED_IR form (FP64 residual, float Jacobian)
#ifndef VOCE_NR_IR_BLOCKS
#define VOCE_NR_IR_BLOCKS 3
#endif
template <bool NR32, bool CHORD = false, bool IR = false>
__global__ void __launch_bounds__(128, NR32 ? VOCE_NR_MIXED_BLOCKS : IR ? VOCE_NR_IR_BLOCKS : 1)
kb_nr(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_ACTIVE)) continue;
        nr_unit<NR32, CHORD, IR>(d, e.y, d.npart);
    }
}

// blocks of 128 threads per SM (256^3 mixed_ir, third increment: 48 ms at 2, 37 at
// 3, 38 at 4)
constexpr int kIncrEndBlocks = 3;
#ifndef VOCE_NR_FCC_BLOCKS
#define VOCE_NR_FCC_BLOCKS 3
#endif
#ifndef VOCE_NR_FCC32_BLOCKS
#define VOCE_NR_FCC32_BLOCKS 3
#endif
template <int FORM>
__global__ void __launch_bounds__(128, FORM >= FCC_IR ? VOCE_NR_FCC32_BLOCKS : VOCE_NR_FCC_BLOCKS) kb_nr_fcc(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_ACTIVE)) continue;
        nr_fcc_unit<FORM>(d, e.y, d.npart);
    }
}

__global__ void __launch_bounds__(128) kb_incr_end(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_CONVERGED)) continue;
        incr_end_unit(d, e.y, d.npart);
    }
}

__global__ void __launch_bounds__(128, kIncrEndBlocks) kb_incr_end_fcc(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_CONVERGED)) continue;
        incr_end_fcc_unit(d, e.y, d.npart);
    }
}

// threads per block of the prelude: pure memory traffic over the 456 or fewer
// units of an RVE, so wide blocks keep enough of it in flight
constexpr int kPreludeThreads = 512;
__global__ void __launch_bounds__(kPreludeThreads) kb_prelude(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_PRELUDE)) continue;
        prelude_unit(d, e.y, d.npart);
    }
}

// one block per RVE.  With use_cond (a plan of one RVE), the iteration
// finaliser also sets the condition of the graph's WHILE node: continue
// while the RVE has not converged (evolution.c:342).
// The RVE's descriptor and macro state are copied into shared memory by the
// whole block while the partial sums are reduced, so that the finaliser reads
// and updates them at shared-memory latency; the macro state is written back
// once at the end.  The iteration finaliser starts its loads before it knows
// whether the RVE is active (most are), the increment's waits for the flag.
__global__ void __launch_bounds__(256) kb_finalize(const RveDesc *descs, int nrve, int incr_end,
                                                   cudaGraphConditionalHandle cond, int use_cond)
{
    static_assert(sizeof(RveDesc) % 8 == 0 && sizeof(MacroDev) % 8 == 0, "staged as 8-byte words");
    constexpr int kDescWords = (int)(sizeof(RveDesc) / 8), kMacroWords = (int)(sizeof(MacroDev) / 8);
    __shared__ unsigned long long s_desc[kDescWords];
    __shared__ unsigned long long s_macro[kMacroWords];
    __shared__ double s_tot[VOCE_NPART];
    for (int r = blockIdx.x; r < nrve; r += gridDim.x) {
        const RveDesc &dg = descs[r];
        if (incr_end && !unit_on(dg, MASK_CONVERGED)) continue;
        unsigned long long *gm = reinterpret_cast<unsigned long long *>(dg.macro);
        const unsigned long long *gd = reinterpret_cast<const unsigned long long *>(&dg);
        const double *part = dg.part;
        const int npart = dg.npart, all1 = !incr_end && dg.all_ph1;
        for (int i = threadIdx.x; i < kMacroWords; i += blockDim.x) s_macro[i] = gm[i];
        for (int i = threadIdx.x; i < kDescWords; i += blockDim.x) s_desc[i] = gd[i];
        reduce_partials(part, npart, all1, s_tot);   // (synchronises the block)
        const RveDesc &d = *reinterpret_cast<const RveDesc *>(s_desc);
        MacroDev *m = reinterpret_cast<MacroDev *>(s_macro);
        // (the increment's finaliser has tested the flag above, and its thread 0
        // clears it in m below: tested here too, it would be read by the other
        // threads while it changes.  The iteration's leaves it alone.)
        if (!incr_end && !m->active) {
            __syncthreads();
            continue;
        }
        if (incr_end) finalize_incr_body(d, m, s_tot);
        else finalize_iter_body(d, m, s_tot);
        __syncthreads();
        if (use_cond && threadIdx.x == 0) cudaGraphSetConditional(cond, m->converged ? 0u : 1u);
        for (int i = threadIdx.x; i < kMacroWords; i += blockDim.x) gm[i] = s_macro[i];
        __syncthreads();
    }
}

// loop condition of the batch: continue while any RVE is active and the
// tick budget is not spent
__global__ void kb_cond(const RveDesc *descs, int nrve, int *ticks, const int *max_ticks,
                        int *active_out, cudaGraphConditionalHandle cond, int use_cond)
{
    __shared__ int any;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    int a = 0;
    for (int r = threadIdx.x; r < nrve; r += blockDim.x) a += descs[r].macro->active;
    if (a) atomicAdd(&any, a);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int t = *ticks + 1;
        *ticks = t;
        *active_out = any;
        if (use_cond) cudaGraphSetConditional(cond, (any > 0 && t < *max_ticks) ? 1u : 0u);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename R>
void Tiles::choose(const RveDesc &d)
{
    const int budget = (sizeof(R) == 8) ? 2048 : 4096;  // complex elements per buffer
    zrows = pick_div(d.ny, budget / (3 * d.nz));
    yxt = pick_div(d.nx, budget / d.ny);
    xkc = pick_div(d.ny, (budget * 3 / 2) / (6 * d.nx));
    xkc3 = pick_div(d.ny, (budget * 3 / 2) / (3 * d.nx));
    zirows = pick_div(d.ny, budget / (3 * d.nz));
    zirows3 = pick_div(d.ny, budget / (2 * d.nz));
}
template void Tiles::choose<double>(const RveDesc &);
template void Tiles::choose<float>(const RveDesc &);


void batch_units(const RveDesc &d, int u[BP_COUNT])
{
    u[BP_NP] = d.npart;
    u[BP_NG] = d.fcc ? 0 : d.npart;
    u[BP_NF] = d.fcc ? d.npart : 0;
    u[BP_ZF] = d.nx * (d.ny / d.zrows);
    u[BP_Y6] = 6 * d.nzh * (d.nx / d.yxt);
    u[BP_XG] = d.nzh * (d.ny / d.xkc);
    u[BP_ZI] = d.nx * (d.ny / d.zirows);
    u[BP_X3] = d.nzh * (d.ny / d.xkc3);
    u[BP_Y3] = 3 * d.nzh * (d.nx / d.yxt);
    u[BP_Z3] = d.nx * (d.ny / d.zirows3);
}

template <typename R>
static size_t batch_smem_t(const RveDesc &d, int ph)
{
    typedef typename Cx<R>::T C;
    // the register-FFT z and Green passes, the staged single-precision z passes
    // where the tile fits in their layout
    if (ph == BP_ZF && zf_fits<C>(d)) return zf_smem<C>(d.nz, d.plz.n1, d.zrows);
    if (ph == BP_ZI && zi_fits<C>(d)) return zi_smem<C>(d.nz, d.plz.n1, d.zirows);
    if (ph == BP_XG && xg_fits<C>(d)) return xg_smem<C>(d.nx, d.plx.n1, d.xkc);
    // (the single-precision forms' own lengths always had that layout along x:
    // a tile too large for it is refused)
    if (ph == BP_XG && sizeof(R) == 4 && d.plx.n1 > 0 && reg_fft_split(d.nx)) return xg_smem<C>(d.nx, d.plx.n1, d.xkc);
    if (sizeof(R) == 4) {
        if (ph == BP_ZF) return sizeof(float2) * (size_t)zf32_fwd_size(d.nz, d.zrows);
        if (ph == BP_ZI) return sizeof(float2) * (size_t)zi32_size(d.nz, d.nzh, d.zirows);
    }
    switch (ph) {
    case BP_ZF: return smem_lines<R>(d.nz, 3 * d.zrows);
    case BP_Y6: case BP_Y3: return smem_lines<R>(d.ny, d.yxt);
    case BP_XG: return smem_lines<R>(d.nx, 6 * d.xkc);
    case BP_ZI: return smem_lines<R>(d.nz, 3 * d.zirows);
    case BP_X3: return smem_lines<R>(d.nx, 3 * d.xkc3);
    case BP_Z3: return smem_lines<R>(d.nz, 2 * d.zirows3);
    default: return 0;
    }
}

size_t batch_smem(const RveDesc &d, int ph)
{
    return d.mixed ? batch_smem_t<float>(d, ph) : batch_smem_t<double>(d, ph);
}

int plan_smem(const std::vector<RveDesc> &descs, bool mixed, size_t smem[BP_COUNT])
{
    long long S = 0;
    bool all = !descs.empty();
    for (const RveDesc &d : descs) {
        for (int ph = 0; ph < BP_COUNT; ++ph) smem[ph] = std::max(smem[ph], batch_smem(d, ph));
        if (d.ply.n1 <= 0) all = false;
        else S = std::max(S, (long long)d.yxt * (d.ny + d.ply.n1 + 1));
    }
    S = (S + 1) & ~1LL;
    const size_t sm = 2 * (size_t)S * (mixed ? sizeof(float2) : sizeof(double2));
    if (!all || sm > kBlockSmem) return 0;
    smem[BP_Y6] = std::max(smem[BP_Y6], sm);
    smem[BP_Y3] = std::max(smem[BP_Y3], sm);
    return (int)S;
}

cudaError_t set_batch_smem(const BatchPlan &bp)
{
    return bp.mixed ? set_fft_smem<float>(bp) : set_fft_smem<double>(bp);
}

// dynamic shared memory of kb_nr<true>: the staged float model columns
static const int kNrStageBytes = VOCE_STAGE_FLOATS * VOCE_NR_THREADS * (int)sizeof(float);

// Newton-kernel blocks resident per GPU (SMs x blocks per SM): the grid cap
// of kb_nr and the most units an RVE is split into for it.  The first call
// also raises kb_nr<true>'s dynamic shared-memory limit; it is made when an
// RVE is created, before any launch or stream capture.
int nr_resident_blocks(int kind)
{
    // several host threads may ask at once: each computes the same value
    static std::atomic<int> cached[6];
    std::atomic<int> &c = cached[(kind >= 0 && kind < 6) ? kind : 0];
    if (!c.load()) {
        int dev = 0, sms = 152, per = 2;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (kind == 1) {
            cudaFuncSetAttribute(kb_nr<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNrStageBytes);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kb_nr<true>, VOCE_NR_THREADS, kNrStageBytes);
        } else if (kind == 2) {
            cudaFuncSetAttribute(kb_nr<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kNrStageBytes);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kb_nr<false, false, true>, VOCE_NR_THREADS,
                                                          kNrStageBytes);
        } else if (kind == 3) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kb_nr_fcc<FCC_FP64>, VOCE_NR_THREADS, 0);
        } else if (kind == 4) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kb_nr_fcc<FCC_IR>, VOCE_NR_THREADS, 0);
        } else if (kind == 5) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kb_nr_fcc<FCC_NR32>, VOCE_NR_THREADS, 0);
        } else {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kb_nr<false>, VOCE_NR_THREADS, 0);
        }
        c.store(sms * (per > 0 ? per : 1));
    }
    return c.load();
}

template <typename R>
static void plan_prelude_t(const BatchPlan &bp, cudaStream_t s, Prof &pf)
{
    const int NG = 152 * 4;
    pf.begin(K_PRELUDE, s);
    kb_prelude<<<grid_for(bp.total[BP_NP], NG), kPreludeThreads, 0, s>>>(bp.descs, bp.map[BP_NP], bp.total[BP_NP]);
    pf.end(K_PRELUDE, s);
}

template <typename R>
static void plan_iteration_t(const BatchPlan &bp, cudaStream_t s, Prof &pf, cudaGraphConditionalHandle cond,
                             int use_cond)
{
    const RveDesc *D = bp.descs;
    pf.begin(K_FFT_Z_FWD, s);
    launch_fft<R>(bp, FFT_ZF, s);
    pf.end(K_FFT_Z_FWD, s);
    pf.begin(K_FFT_Y_FWD, s);
    launch_fft<R>(bp, FFT_YF, s);
    pf.end(K_FFT_Y_FWD, s);
    pf.begin(K_FFT_X_GREEN, s);
    launch_fft<R>(bp, FFT_XG, s);
    pf.end(K_FFT_X_GREEN, s);
    pf.begin(K_FFT_Y_INV, s);
    launch_fft<R>(bp, FFT_YI, s);
    pf.end(K_FFT_Y_INV, s);
    pf.begin(K_FFT_Z_INV, s);
    launch_fft<R>(bp, FFT_ZI, s);
    pf.end(K_FFT_Z_INV, s);
    // a plan's RVEs of the {111}<110> family and the others: one launch each,
    // where there are any
    pf.begin(K_NR, s);
    int launched = 0;
    if (const int n = bp.total[BP_NF]) {
        const int g = grid_for(n, nr_resident_blocks(bp.nr32 ? 5 : bp.ir ? 4 : 3));
        if (bp.nr32) kb_nr_fcc<FCC_NR32><<<g, VOCE_NR_THREADS, 0, s>>>(D, bp.map[BP_NF], n);
        else if (bp.ir) kb_nr_fcc<FCC_IR><<<g, VOCE_NR_THREADS, 0, s>>>(D, bp.map[BP_NF], n);
        else kb_nr_fcc<FCC_FP64><<<g, VOCE_NR_THREADS, 0, s>>>(D, bp.map[BP_NF], n);
        ++launched;
    }
    if (const int n = bp.total[BP_NG]) {
        const int kind = bp.nr32 ? 1 : bp.ir ? 2 : 0;
        const int g = grid_for(n, nr_resident_blocks(kind));
        if (bp.nr32) kb_nr<true><<<g, VOCE_NR_THREADS, kNrStageBytes, s>>>(D, bp.map[BP_NG], n);
        else if (bp.ir) kb_nr<false, false, true><<<g, VOCE_NR_THREADS, kNrStageBytes, s>>>(D, bp.map[BP_NG], n);
        else if (bp.mixed) kb_nr<false, true><<<g, VOCE_NR_THREADS, 0, s>>>(D, bp.map[BP_NG], n);
        else kb_nr<false><<<g, VOCE_NR_THREADS, 0, s>>>(D, bp.map[BP_NG], n);
        ++launched;
    }
    pf.end(K_NR, s, launched);
    pf.begin(K_FIN_ITER, s);
    kb_finalize<<<grid_for(bp.nrve, 152 * 4), 256, 0, s>>>(D, bp.nrve, 0, cond, use_cond);
    pf.end(K_FIN_ITER, s);
}

template <typename R>
static void plan_incr_end_t(const BatchPlan &bp, cudaStream_t s, Prof &pf)
{
    const int NG = 152 * 2;
    const RveDesc *D = bp.descs;
    pf.begin(K_INC_FFT, s);
    launch_fft<R>(bp, FFT_X3, s);
    launch_fft<R>(bp, FFT_Y3, s);
    launch_fft<R>(bp, FFT_Z3, s);
    pf.end(K_INC_FFT, s, 3);
    pf.begin(K_INCR_END, s);
    if (const int n = bp.total[BP_NF]) kb_incr_end_fcc<<<grid_for(n, 152 * kIncrEndBlocks), 128, 0, s>>>(D, bp.map[BP_NF], n);
    if (const int n = bp.total[BP_NG]) kb_incr_end<<<grid_for(n, NG), 128, 0, s>>>(D, bp.map[BP_NG], n);
    pf.end(K_INCR_END, s, (bp.total[BP_NF] ? 1 : 0) + (bp.total[BP_NG] ? 1 : 0));
    pf.begin(K_FIN_INCR, s);
    kb_finalize<<<grid_for(bp.nrve, 152 * 4), 256, 0, s>>>(D, bp.nrve, 1, 0, 0);
    pf.end(K_FIN_INCR, s);
}

cudaError_t launch_plan_prelude(const BatchPlan &bp, cudaStream_t s, Prof &pf)
{
    if (bp.mixed) plan_prelude_t<float>(bp, s, pf);
    else plan_prelude_t<double>(bp, s, pf);
    return cudaGetLastError();
}

cudaError_t launch_plan_iteration(const BatchPlan &bp, cudaStream_t s, Prof &pf,
                                  cudaGraphConditionalHandle cond, int use_cond)
{
    if (bp.mixed) plan_iteration_t<float>(bp, s, pf, cond, use_cond);
    else plan_iteration_t<double>(bp, s, pf, cond, use_cond);
    return cudaGetLastError();
}

cudaError_t launch_plan_incr_end(const BatchPlan &bp, cudaStream_t s, Prof &pf)
{
    if (bp.mixed) plan_incr_end_t<float>(bp, s, pf);
    else plan_incr_end_t<double>(bp, s, pf);
    return cudaGetLastError();
}

cudaError_t launch_plan_phase(const BatchPlan &bp, int phase, cudaStream_t s)
{
    const FftPass pass = phase == BP_ZF ? FFT_ZF : phase == BP_Y6 ? FFT_YF : phase == BP_XG ? FFT_XG : FFT_ZI;
    if (bp.mixed) launch_fft<float>(bp, pass, s);
    else launch_fft<double>(bp, pass, s);
    return cudaGetLastError();
}

// units of a phase with tile t
static int tile_units(const RveDesc &d, int phase, int t)
{
    switch (phase) {
    case BP_Y6: return 6 * d.nzh * (d.nx / t);
    case BP_XG: return d.nzh * (d.ny / t);
    default: return d.nx * (d.ny / t);
    }
}

// an axis on the register FFT whose tile goes through fft_lines all the same
template <typename C>
static bool off_layout(const RveDesc &d, int phase)
{
    switch (phase) {
    case BP_ZF: return d.plz.n1 > 0 && !zf_fits<C>(d);
    case BP_XG: return d.plx.n1 > 0 && !xg_fits<C>(d);
    case BP_ZI: return d.plz.n1 > 0 && !zi_fits<C>(d);
    default: return false;
    }
}

int tile_candidates(const RveDesc &d, int phase, int *out, int max)
{
    const bool f = d.mixed != 0;
    const int B = f ? 4096 : 2048;
    const size_t smem_max = 200 * 1024;
    int n = 0;
    // from the largest down, and below a quarter of the budget only while a
    // tile gives the phase fewer units than two blocks per SM: a small grid
    // fills the GPU with small tiles (16^3 FP64: x + Green 28 -> 24 us, the
    // Green iteration 113 -> 102 us; 32^3 163 -> 157 us), a large one does
    // not need them
    for (int k = 2; k >= -5 && n < max; --k) {
        const int budget = k < 0 ? (B >> -k) : (B << k);
        if (k < -2 && n > 0 && tile_units(d, phase, out[n - 1]) >= 2 * 152) break;
        int t = 0;
        RveDesc dt = d;
        switch (phase) {
        case BP_ZF: t = dt.zrows = pick_div(d.ny, budget / (3 * d.nz)); break;
        case BP_Y6: t = dt.yxt = pick_div(d.nx, budget / d.ny); break;
        case BP_XG: t = dt.xkc = pick_div(d.ny, (budget * 3 / 2) / (6 * d.nx)); break;
        case BP_ZI: t = dt.zirows = pick_div(d.ny, budget / (3 * d.nz)); break;
        default: return 0;
        }
        if (t < 1 || batch_smem(dt, phase) > smem_max) continue;
        // only in the register FFT's own layout, where the axis has one
        const bool off = f ? off_layout<float2>(dt, phase) : off_layout<double2>(dt, phase);
        if (off) continue;
        bool seen = false;
        for (int i = 0; i < n; ++i) seen = seen || out[i] == t;
        if (!seen) out[n++] = t;
    }
    return n;
}

cudaError_t launch_batch_tick(const BatchPlan &bp, cudaStream_t s, cudaGraphConditionalHandle cond)
{
    Prof none;
    launch_plan_prelude(bp, s, none);
    launch_plan_iteration(bp, s, none, 0, 0);
    launch_plan_incr_end(bp, s, none);
    kb_cond<<<1, 256, 0, s>>>(bp.descs, bp.nrve, bp.ticks, bp.max_ticks, bp.active_out, cond, 1);
    return cudaGetLastError();
}

cudaError_t launch_batch_tick_timed(const BatchPlan &bp, cudaStream_t s, Prof &pf)
{
    launch_plan_prelude(bp, s, pf);
    launch_plan_iteration(bp, s, pf, 0, 0);
    launch_plan_incr_end(bp, s, pf);
    kb_cond<<<1, 256, 0, s>>>(bp.descs, bp.nrve, bp.ticks, bp.max_ticks, bp.active_out, 0, 0);
    pf.launches += 1;
    return cudaGetLastError();
}

// Periodic Voronoi labels: each voxel centre ((x+0.5)/nx, ...) of the unit
// cube takes the nearest seed by minimum-image distance, ties to the lowest
// index.  The arithmetic is that of the host generator's numpy form: the
// image by round-half-to-even (rint), the squared distance summed as
// (d0^2 + d1^2) + d2^2 without contraction, strict < over seeds in order.
__global__ void k_voronoi(int nx, int ny, int nz, int ns, const double *__restrict__ seeds,
                          int *__restrict__ label)
{
    extern __shared__ double s_seed[];   // 3 x VORONOI_TILE
    const long long nv = (long long)nx * ny * nz;
    const long long v0 = (long long)blockIdx.x * blockDim.x;
    const long long v = v0 + threadIdx.x;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    if (v < nv) {
        const int z = (int)(v % nz), y = (int)((v / nz) % ny), x = (int)(v / ((long long)ny * nz));
        p0 = ((double)x + 0.5) / (double)nx;
        p1 = ((double)y + 0.5) / (double)ny;
        p2 = ((double)z + 0.5) / (double)nz;
    }
    double best = 1e300;
    int bi = 0;
    for (int t0 = 0; t0 < ns; t0 += VORONOI_TILE) {
        const int tn = min(VORONOI_TILE, ns - t0);
        __syncthreads();
        for (int i = threadIdx.x; i < 3 * tn; i += blockDim.x) s_seed[i] = seeds[3 * t0 + i];
        __syncthreads();
        for (int j = 0; j < tn; ++j) {
            double d0 = __dsub_rn(p0, s_seed[3 * j]);
            double d1 = __dsub_rn(p1, s_seed[3 * j + 1]);
            double d2 = __dsub_rn(p2, s_seed[3 * j + 2]);
            d0 = __dsub_rn(d0, rint(d0));
            d1 = __dsub_rn(d1, rint(d1));
            d2 = __dsub_rn(d2, rint(d2));
            const double dd = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
            if (dd < best) {
                best = dd;
                bi = t0 + j;
            }
        }
    }
    if (v < nv) label[v] = bi;
}

cudaError_t launch_voronoi(int nx, int ny, int nz, int ns, const double *seeds, int *label, cudaStream_t s)
{
    const long long nv = (long long)nx * ny * nz;
    const int blocks = (int)((nv + 255) / 256);
    k_voronoi<<<blocks, 256, 3 * VORONOI_TILE * sizeof(double), s>>>(nx, ny, nz, ns, seeds, label);
    return cudaGetLastError();
}

// gstore: n and omega of every frequency of the half spectrum (FP64 form),
// with the arithmetic green_apply uses when it computes them
__global__ void k_fill_green(RveDesc d)
{
    const long long ns = d.nspec, plane = (long long)d.nx * d.ny;
    for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < ns;
         o += (long long)gridDim.x * blockDim.x) {
        const int iz = (int)(o / plane), ix = (int)((o % plane) / d.ny), iy = (int)(o % d.ny);
        double n[3] = {0.0, 0.0, 0.0}, w[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if ((ix | iy | iz) != 0) {
            unit_freq(d, ix, iy, iz, n);
            green_omega<double>(d.Kq, n, w);
        }
        for (int q = 0; q < 3; ++q) d.gstore[q * ns + o] = n[q];
        for (int q = 0; q < 6; ++q) d.gstore[(3 + q) * ns + o] = w[q];
    }
}

cudaError_t launch_fill_green(const RveDesc &d, cudaStream_t s)
{
    if (!d.gstore) return cudaSuccess;
    int blocks = (int)((d.nspec + 255) / 256);
    if (blocks > 152 * 8) blocks = 152 * 8;
    k_fill_green<<<blocks, 256, 0, s>>>(d);
    return cudaGetLastError();
}

// sgp32 + sgp_lo = S_g + S0 once S0 is known (mixed form)
__global__ void k_fill_p32(RveDesc d)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < d.nv;
         v += (long long)gridDim.x * blockDim.x) {
        double P[21];
        load_P(d, v, P);
        const bool solid = d.solid[d.phase[v]] != 0;
        for (int q = 0; q < 21; ++q) put_pair(d.sgp32, d.sgp_lo, (long long)q * d.nv + v, solid ? P[q] : 0.0);
        if (d.sgp)
            for (int q = 0; q < 21; ++q) d.sgp[(long long)q * d.nv + v] = solid ? P[q] : 0.0;
    }
}

cudaError_t launch_fill_p32(const RveDesc &d, cudaStream_t s)
{
    int blocks = (int)((d.nv + 255) / 256);
    if (blocks > 152 * 8) blocks = 152 * 8;
    k_fill_p32<<<blocks, 256, 0, s>>>(d);
    return cudaGetLastError();
}

// the crystal-axes columns of every solid voxel, once S0 is known; gas voxels,
// which nothing reads but a snapshot, hold zeros (k_setup writes theirs in the
// other arrays)
__global__ void __launch_bounds__(128) k_fill_fcc(RveDesc d)
{
    for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < d.nv;
         v += (long long)gridDim.x * blockDim.x) {
        if (!d.solid[d.phase[v]]) {
            if (d.sgp32)
                for (int q = 0; q < 15; ++q) put_ff(d.sgp32, d.sgp_lo, q * d.nv + v, 0.0);
            continue;
        }
        double T[3][3];
        for (int i = 0; i < 3; ++i)
            for (int j = 0; j < 3; ++j) T[i][j] = d.tm[(3 * i + j) * d.nv + v];
        fcc_frame(d, v, T);
    }
}

cudaError_t launch_fill_fcc(const RveDesc &d, cudaStream_t s)
{
    if (!d.fcc) return cudaSuccess;
    int blocks = (int)((d.nv + 127) / 128);
    if (blocks > 152 * 8) blocks = 152 * 8;
    k_fill_fcc<<<blocks, 128, 0, s>>>(d);
    return cudaGetLastError();
}

cudaError_t launch_setup(const RveDesc &d, const SetupConst &sc, const double *euler, int npart,
                         cudaStream_t s)
{
    k_setup<<<npart, 128, 0, s>>>(d, sc, euler);
    return cudaGetLastError();
}


// writes n doubles: evicts the L2 between timed steps
__global__ void k_flush(double *buf, long long n)
{
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        buf[i] = (double)i;
}

cudaError_t launch_flush(double *buf, long long n, cudaStream_t s)
{
    k_flush<<<152 * 8, 256, 0, s>>>(buf, n);
    return cudaGetLastError();
}

// rcp_nr on n doubles (a check of the Newton step's reciprocal against 1/x)
__global__ void k_rcp_probe(const double *__restrict__ x, double *__restrict__ out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = rcp_nr(x[i]);
}

cudaError_t launch_rcp_probe(const double *x, double *out, int n, cudaStream_t s)
{
    if (n > 0) k_rcp_probe<<<(n + 255) / 256, 256, 0, s>>>(x, out, n);
    return cudaGetLastError();
}

__global__ void k_sqrt_probe(const double *__restrict__ x, double *__restrict__ out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = sqrt_nr(x[i]);
}

cudaError_t launch_sqrt_probe(const double *x, double *out, int n, cudaStream_t s)
{
    if (n > 0) k_sqrt_probe<<<(n + 255) / 256, 256, 0, s>>>(x, out, n);
    return cudaGetLastError();
}

// out[0..n): d2f_rn, out[n..2n): f2d of (float)x where that is finite, (float)x
// itself where it is not, out[2n..3n): the sum and out[3n..4n): the first
// part of the float pair d2ff
__global__ void k_convert_probe(const double *__restrict__ x, double *__restrict__ out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float f = (float)x[i];
        const ff32 p = d2ff(x[i]);
        out[i] = (double)d2f_rn(x[i]);
        out[n + i] = finite_f(f) ? f2d(f) : (double)f;
        out[2 * n + i] = (double)p.h + (double)p.l;
        out[3 * n + i] = (double)p.h;
    }
}

cudaError_t launch_convert_probe(const double *x, double *out, int n, cudaStream_t s)
{
    if (n > 0) k_convert_probe<<<(n + 255) / 256, 256, 0, s>>>(x, out, n);
    return cudaGetLastError();
}

// FP64 FMA throughput: 8 independent FMA chains per thread
__global__ void k_fp64_fma(double *out, int iters, double a, double b)
{
    double x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = threadIdx.x * 1e-9 + k;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = fma(x[k], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += x[k];
    if (s == 12345.678) out[0] = s;   // keeps the chains live; never true
}

double measure_fp64_tflops()
{
    double *out = nullptr;
    if (cudaMalloc(&out, sizeof(double)) != cudaSuccess) return -1.0;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int blocks = sms * 8, threads = 256, iters = 8192;
    k_fp64_fma<<<blocks, threads>>>(out, 64, 0.999999, 1e-7);   // warm-up
    cudaEventRecord(e0);
    k_fp64_fma<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    const double flops = 2.0 * 8.0 * (double)iters * blocks * threads;
    return ms > 0.f ? flops / (ms * 1e-3) / 1e12 : -1.0;
}

cudaError_t launch_field_out(const RveDesc &d, int field, double *out, cudaStream_t s)
{
    int blocks = (int)((d.nv + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    k_field_out<<<blocks, 256, 0, s>>>(d, field, out);
    return cudaGetLastError();
}

}  // namespace voce
