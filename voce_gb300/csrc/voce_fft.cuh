// The spectrum passes: tile copies, the transforms along z, y and x with the
// Green operator, and their kernels.  A translation unit instantiates one
// precision (voce_fft32.cu, voce_fft64.cu) through VOCE_FFT_INSTANCE; the
// displacement fluctuation (voce_disp.cu) uses the unit functions.
#pragma once
#include "voce_dev.cuh"
#include "voce_kernels.h"

#include <algorithm>

namespace voce {

// ---------------------------------------------------------------------------
// Asynchronous global -> shared copies (cp.async): the data lands in shared
// memory without passing through registers, so a thread can have every
// element of its share of a tile in flight at once; cp_async_wait_all waits
// for all of this thread's outstanding copies (a __syncthreads then makes
// them visible to the block).  4 and 8 bytes are cached in L1 and L2, 16
// bytes in L2 only; both addresses aligned to the size.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async4(float *smem, const float *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(__cvta_generic_to_global(gmem)) : "memory");
}

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(__cvta_generic_to_global(gmem)) : "memory");
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(__cvta_generic_to_global(gmem)) : "memory");
}

// one complex number
__device__ __forceinline__ void cp_asyncc(float2 *smem, const float2 *gmem) { cp_async8(smem, gmem); }
__device__ __forceinline__ void cp_asyncc(double2 *smem, const double2 *gmem) { cp_async16(smem, gmem); }

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---------------------------------------------------------------------------
// FFT passes
// ---------------------------------------------------------------------------
// Position (a0, a1, a2) of a flat tile index i = a0 + n0 (a1 + n1 a2),
// carried from one element of a thread to its next (i += step) by additions
// and compares: a tile loop pays the integer divisions by the run-time tile
// extents once per thread instead of once per element (those divisions were
// most of the instructions of the FFT passes' load and store loops).
struct Idx3 {
    int a0, a1, a2, d0, d1, d2, n0, n1;
    __device__ __forceinline__ Idx3(int i, int step, int n0_, int n1_) : n0(n0_), n1(n1_)
    {
        int t = i / n0;
        a0 = i - t * n0;
        a1 = t % n1;
        a2 = t / n1;
        t = step / n0;
        d0 = step - t * n0;
        d1 = t % n1;
        d2 = t / n1;
    }
    __device__ __forceinline__ void next()
    {
        a0 += d0;
        int c = a0 >= n0;
        if (c) a0 -= n0;
        a1 += d1 + c;
        c = a1 >= n1;
        if (c) a1 -= n1;
        a2 += d2 + c;
    }
};
constexpr int kIdxUnbounded = 1 << 30;   // n1 of a two-level index (a2 stays 0)

// Tile copy of n elements by the block over a carried index: each thread
// first loads U elements (its i, i + nthr, ...) into registers, then stores
// them, so that U global loads per thread are in flight at once.
// ld(a0, a1, a2) returns an element, st(a0, a1, a2, value) places it.
template <int U, typename T, class LD, class ST>
__device__ __forceinline__ void staged_copy3(int n, int n0, int n1, LD ld, ST st)
{
    const int nt = blockDim.x;
    Idx3 il(threadIdx.x, nt, n0, n1), is = il;
    for (int b = threadIdx.x; b < n; b += U * nt) {
        T v[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (b + j * nt < n) v[j] = ld(il.a0, il.a1, il.a2);
            il.next();
        }
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (b + j * nt < n) st(is.a0, is.a1, is.a2, v[j]);
            is.next();
        }
    }
}

// loads in flight per thread: the single-precision passes wait on memory, the
// double-precision ones on the FP64 pipe (there one at a time, as before,
// keeps their registers and occupancy)
template <typename R> struct CopyDepth { static constexpr int v = 8; };
template <> struct CopyDepth<double> { static constexpr int v = 1; };
// the z passes gather strided columns and convert: measured slower with
// deeper copies (more registers, fewer resident blocks), so one at a time
constexpr int kZCopyDepth = 1;

// the stress's six components into the spectrum (evolution.c:350-361)
template <typename R>
__device__ void fft_z_fwd_unit(const RveDesc &d, int rows, int unit)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bufA = reinterpret_cast<C *>(smem_raw);
    const int nx = d.nx, ny = d.ny, nz = d.nz, nzh = d.nzh;
    const long long nv = d.nv;
    const int NL = 3 * rows, ldl = NL | 1;
    C *bufB = bufA + nz * ldl;
    const int ytiles = ny / rows;
    const int x = unit / ytiles, y0 = (unit % ytiles) * rows;
    const long long vb = ((long long)x * ny + y0) * nz;
    if constexpr (sizeof(R) == 4) {
        // rows y0 .. y0 + rows - 1 of a component are one run of rows * nz
        // doubles (z fastest): the six runs are staged behind bufA by
        // 16-byte asynchronous copies, then converted into the line layout
        double *stage = reinterpret_cast<double *>(bufB);
        const int run = rows * nz, half_run = run / 2;   // nz is even
        Idx3 ic(threadIdx.x, blockDim.x, half_run, kIdxUnbounded);
        for (int i = threadIdx.x; i < 6 * half_run; i += blockDim.x, ic.next())
            cp_async16(stage + 2 * i, d.sig + ic.a1 * nv + vb + 2 * ic.a0);
        cp_async_wait_all();
        __syncthreads();
        // element (z, r, p): components 2p and 2p + 1 of row r
        Idx3 ix(threadIdx.x, blockDim.x, nz, rows);
        for (int i = threadIdx.x; i < 3 * run; i += blockDim.x, ix.next()) {
            const int z = ix.a0, r = ix.a1, p = ix.a2, q = r * nz + z;
            bufA[z * ldl + p * rows + r] = make_float2(d2f_rn(stage[2 * p * run + q]), d2f_rn(stage[(2 * p + 1) * run + q]));
        }
    } else {
        // element (z, r, c) is sig[c][vb + r * nz + z]
        staged_copy3<kZCopyDepth, double>(
            6 * rows * nz, nz, rows,
            [&](int z, int r, int c) { return __ldg(d.sig + c * nv + vb + (long long)r * nz + z); },
            [&](int z, int r, int c, double v) {
                C *e = &bufA[z * ldl + (c >> 1) * rows + r];
                if (c & 1) e->y = (R)v; else e->x = (R)v;
            });
    }
    __syncthreads();
    C *res = fft_lines<R>(bufA, bufB, NL, ldl, d.plz, (const C *)d.twz, -1);
    C *spec = (C *)d.spec;
    const long long plane = (long long)nx * ny;
    Idx3 ix(threadIdx.x, blockDim.x, rows, nzh);
    for (int idx = threadIdx.x; idx < 3 * rows * nzh; idx += blockDim.x, ix.next()) {
        const int r = ix.a0, k = ix.a1, p = ix.a2;
        const int l = p * rows + r;
        const C zk = res[k * ldl + l], zm = res[((nz - k) % nz) * ldl + l];
        C A, B;
        A.x = R(0.5) * (zk.x + zm.x);
        A.y = R(0.5) * (zk.y - zm.y);
        B.x = R(0.5) * (zk.y + zm.y);
        B.y = R(-0.5) * (zk.x - zm.x);
        const long long o = (long long)k * plane + (long long)x * ny + y0 + r;
        spec[(long long)(2 * p) * nzh * plane + o] = A;
        spec[(long long)(2 * p + 1) * nzh * plane + o] = B;
    }
}


// forward r2c along z of ncomp real fields src[c][nv] into the half
// spectrum dstp[c][nzh][nx][ny]: two fields per complex line (an odd count
// pads the last line with zeros), split by the Hermitian symmetry of each
template <typename R, int ncomp>
__device__ void fft_z_fwd_src(const RveDesc &d, const double *src, void *dstp, int rows, int unit)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bufA = reinterpret_cast<C *>(smem_raw);
    const int nx = d.nx, ny = d.ny, nz = d.nz, nzh = d.nzh;
    const long long nv = d.nv;
    const int np = (ncomp + 1) / 2;
    const int NL = np * rows, ldl = NL | 1;
    C *bufB = bufA + nz * ldl;
    const int ytiles = ny / rows;
    const int x = unit / ytiles, y0 = (unit % ytiles) * rows;
    const long long vb = ((long long)x * ny + y0) * nz;
    Idx3 iz(threadIdx.x, blockDim.x, nz, rows);
    for (int idx = threadIdx.x; idx < 2 * np * rows * nz; idx += blockDim.x, iz.next()) {
        const int z = iz.a0, r = iz.a1, c = iz.a2;
        const R val = (ncomp % 2 == 0 || c < ncomp) ? (R)__ldg(src + c * nv + vb + (long long)r * nz + z) : R(0);
        C *e = &bufA[z * ldl + (c >> 1) * rows + r];
        if (c & 1) e->y = val; else e->x = val;
    }
    __syncthreads();
    C *res = fft_lines<R>(bufA, bufB, NL, ldl, d.plz, (const C *)d.twz, -1);
    C *spec = (C *)dstp;
    const long long plane = (long long)nx * ny;
    Idx3 ix(threadIdx.x, blockDim.x, rows, nzh);
    for (int idx = threadIdx.x; idx < np * rows * nzh; idx += blockDim.x, ix.next()) {
        const int r = ix.a0, k = ix.a1, p = ix.a2;
        const int l = p * rows + r;
        const C zk = res[k * ldl + l], zm = res[((nz - k) % nz) * ldl + l];
        C A, B;
        A.x = R(0.5) * (zk.x + zm.x);
        A.y = R(0.5) * (zk.y - zm.y);
        B.x = R(0.5) * (zk.y + zm.y);
        B.y = R(-0.5) * (zk.x - zm.x);
        const long long o = (long long)k * plane + (long long)x * ny + y0 + r;
        spec[(long long)(2 * p) * nzh * plane + o] = A;
        if (ncomp % 2 == 0 || 2 * p + 1 < ncomp) spec[(long long)(2 * p + 1) * nzh * plane + o] = B;
    }
}



template <typename R>
__device__ void fft_y_unit(const RveDesc &d, void *specp, int sign, int xt, int unit)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bufA = reinterpret_cast<C *>(smem_raw);
    const int nx = d.nx, ny = d.ny;
    const int NL = xt, ldl = NL | 1;
    C *bufB = bufA + ny * ldl;
    const int xtiles = nx / xt;
    const int line = unit / xtiles;  // c * nzh + kz
    const int x0 = (unit % xtiles) * xt;
    C *spec = (C *)specp;
    const long long base = ((long long)line * nx + x0) * ny;
    // element (y, xl) is spec[base + xl * ny + y]
    if constexpr (sizeof(R) == 4) {
        Idx3 il(threadIdx.x, blockDim.x, ny, kIdxUnbounded);
        for (int i = threadIdx.x; i < xt * ny; i += blockDim.x, il.next())
            cp_async8(&bufA[il.a0 * ldl + il.a1], spec + base + i);
        cp_async_wait_all();
    } else {
        staged_copy3<CopyDepth<R>::v, C>(
            xt * ny, ny, kIdxUnbounded, [&](int y, int xl, int) { return spec[base + xl * ny + y]; },
            [&](int y, int xl, int, C v) { bufA[y * ldl + xl] = v; });
    }
    __syncthreads();
    C *res = fft_lines<R>(bufA, bufB, NL, ldl, d.ply, (const C *)d.twy, sign);
    Idx3 ix(threadIdx.x, blockDim.x, ny, kIdxUnbounded);
    for (int idx = threadIdx.x; idx < xt * ny; idx += blockDim.x, ix.next())
        spec[base + idx] = res[ix.a0 * ldl + ix.a1];
}


// ---------------------------------------------------------------------------
// The y pass as a stream over a block's
// units, for plans whose RVEs all run the register FFT along y.  A unit's
// tile (NL = yxt lines of L = ny contiguous coefficients) is held line by
// line at pos(l, i) = l LP + i + i / N2, LP = L + N1 + 1: pass 1 (tasks
// (t, l), t fastest) and pass 2 (tasks (k1, l), k1 fastest) then read rows
// of consecutive words, and pass 2 writes X[k1 + N1 k2] of line l straight
// to the spectrum, consecutive threads to consecutive coefficients.  The
// next unit's tile is staged by cp.async while this one transforms (two
// tile buffers of S complex numbers, S >= NL LP of every RVE of the plan).
// ---------------------------------------------------------------------------
template <typename C, int N1, int N2, int S>
__device__ __forceinline__ void ystream_tile(C *A, int NL, C *g, const C *__restrict__ tw)
{
    constexpr int L = N1 * N2, LP = L + N1 + 1;
    const int tid = threadIdx.x, nthr = blockDim.x;
    for (int task = tid; task < NL * N2; task += nthr) {
        const int l = task / N2, t = task - l * N2;
        C *p = A + l * LP + t;
        C x[N1];
        sfor<0, N1>([&](auto jc) { x[decltype(jc)::v] = p[(N2 + 1) * decltype(jc)::v]; });
        sdft<N1, S, 0, 1>(x);
        if (t != 0) {
            const C *wm = tw + L + t;   // the pass-1 twiddle matrix
            sfor<1, N1>([&](auto kc) {
                constexpr int k = decltype(kc)::v, r = dft_pos(N1, k);
                C w = __ldg(wm + k * N2);
                if (S > 0) w.y = -w.y;
                x[r] = cmul<typename RealOf<C>::T>(x[r], w);
            });
        }
        sfor<0, N1>([&](auto kc) { p[(N2 + 1) * decltype(kc)::v] = x[dft_pos(N1, decltype(kc)::v)]; });
    }
    __syncthreads();
    for (int task = tid; task < NL * N1; task += nthr) {
        const int l = task / N1, k1 = task - l * N1;
        const C *p = A + l * LP + (N2 + 1) * k1;
        C x[N2];
#pragma unroll
        for (int t = 0; t < N2; ++t) x[t] = p[t];
        sdft<N2, S, 0, 1>(x);
        C *q = g + l * L + k1;
        sfor<0, N2>([&](auto kc) { q[N1 * decltype(kc)::v] = x[dft_pos(N2, decltype(kc)::v)]; });
    }
}

template <typename R>
__device__ void fft_x_green_unit(const RveDesc &d, int kc, int unit)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bufA = reinterpret_cast<C *>(smem_raw);
    const int nx = d.nx, ny = d.ny, nzh = d.nzh;
    const int NL = 6 * kc, ldl = NL | 1;
    C *bufB = bufA + nx * ldl;
    const int ytiles = ny / kc;
    const int kz = unit / ytiles, y0 = (unit % ytiles) * kc;
    C *spec = (C *)d.spec;
    C *aacc = (C *)d.aacc;
    const long long plane = (long long)nx * ny, cstride = (long long)nzh * plane;
    const long long kb = (long long)kz * plane + y0;
    // element (yl, x, c) is spec[c][kz][x][y0 + yl]
    if constexpr (sizeof(R) == 4) {
        Idx3 il(threadIdx.x, blockDim.x, kc, nx);
        for (int i = threadIdx.x; i < 6 * nx * kc; i += blockDim.x, il.next())
            cp_async8(&bufA[il.a0 + il.a1 * ldl + il.a2 * kc],
                      spec + il.a2 * cstride + kb + (long long)il.a1 * ny + il.a0);
        cp_async_wait_all();
    } else {
        staged_copy3<CopyDepth<R>::v, C>(
            6 * nx * kc, kc, nx,
            [&](int yl, int x, int c) { return spec[c * cstride + kb + (long long)x * ny + yl]; },
            [&](int yl, int x, int c, C v) { bufA[x * ldl + c * kc + yl] = v; });
    }
    __syncthreads();
    C *res = fft_lines<R>(bufA, bufB, NL, ldl, d.plx, (const C *)d.twx, -1);
    C *oth = (res == bufA) ? bufB : bufA;
    const int first = d.macro->first_iter;
    // single precision: the accumulator's tile, acc[(c nx + x) kc + yl], is
    // staged in the free line buffer while the Green loop's operands wait
    C *acc = oth;
    if constexpr (sizeof(R) == 4) {
        if (!first) {
            Idx3 il(threadIdx.x, blockDim.x, kc, nx);
            for (int i = threadIdx.x; i < 3 * nx * kc; i += blockDim.x, il.next())
                cp_async8(acc + i, aacc + il.a2 * cstride + kb + (long long)il.a1 * ny + il.a0);
            cp_async_wait_all();
            __syncthreads();
        }
    }
    Idx3 ig(threadIdx.x, blockDim.x, kc, kIdxUnbounded);
    for (int idx = threadIdx.x; idx < nx * kc; idx += blockDim.x, ig.next()) {
        const int yl = ig.a0, x = ig.a1;
        R br[6], bi[6], ar[3], ai[3];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const C e = res[x * ldl + c * kc + yl];
            br[c] = e.x;
            bi[c] = e.y;
        }
        green_apply<R>(d, x, y0 + yl, kz, kb + (long long)x * ny + yl, br, bi, ar, ai);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            C e;
            e.x = br[c];
            e.y = bi[c];
            res[x * ldl + c * kc + yl] = e;
        }
        const long long o = kb + (long long)x * ny + yl;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            C e;
            if (first) { e.x = ar[c]; e.y = ai[c]; }
            else {
                if constexpr (sizeof(R) == 4) e = acc[(c * nx + x) * kc + yl];
                else e = aacc[c * cstride + o];
                e.x += ar[c];
                e.y += ai[c];
            }
            aacc[c * cstride + o] = e;
        }
    }
    __syncthreads();
    C *res2 = fft_lines<R>(res, oth, NL, ldl, d.plx, (const C *)d.twx, +1);
    Idx3 is(threadIdx.x, blockDim.x, kc, nx);
    for (int idx = threadIdx.x; idx < 6 * nx * kc; idx += blockDim.x, is.next()) {
        const int yl = is.a0, x = is.a1, c = is.a2;
        spec[c * cstride + kb + (long long)x * ny + yl] = res2[x * ldl + c * kc + yl];
    }
}


// ---------------------------------------------------------------------------
// The x pass with the Green operator for an RVE on the register FFT along x.
// The tile's NL = 6 kc lines (line l = c kc + yl:
// component c, column y0 + yl) are held line by line at pos(l, i) = l LP +
// i + i / N2, LP = L + N1 + 1 (odd): the forward transform runs in place on
// A and leaves X[k] at pos(l, k) of B, the Green operator works on B, the
// inverse transform runs in place on B and its second pass writes straight
// to the spectrum.  Every shared-memory index inside the transforms is a
// compile-time offset from one base per task.
// ---------------------------------------------------------------------------
template <typename C, int N1, int N2, int S>
__device__ __forceinline__ void xg_pass1(C *A, int NL, const C *__restrict__ tw)
{
    constexpr int L = N1 * N2, LP = L + N1 + 1;
    for (int task = threadIdx.x; task < NL * N2; task += blockDim.x) {
        const int l = task / N2, t = task - l * N2;
        C *p = A + l * LP + t;
        C x[N1];
        sfor<0, N1>([&](auto jc) { x[decltype(jc)::v] = p[(N2 + 1) * decltype(jc)::v]; });
        sdft<N1, S, 0, 1>(x);
        if (t != 0) {
            const C *wm = tw + L + t;   // the pass-1 twiddle matrix
            sfor<1, N1>([&](auto kc) {
                constexpr int k = decltype(kc)::v, r = dft_pos(N1, k);
                C w = __ldg(wm + k * N2);
                if (S > 0) w.y = -w.y;
                x[r] = cmul<typename RealOf<C>::T>(x[r], w);
            });
        }
        sfor<0, N1>([&](auto kc) { p[(N2 + 1) * decltype(kc)::v] = x[dft_pos(N1, decltype(kc)::v)]; });
    }
}

template <typename C, int N1, int N2>
__device__ void xg_unit(const RveDesc &d, int kc, int unit)
{
    typedef typename RealOf<C>::T R;
    constexpr int L = N1 * N2, LP = L + N1 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *A = reinterpret_cast<C *>(smem_raw);
    const int NL = 6 * kc;
    C *B = A + NL * LP;
    const int ny = d.ny, nzh = d.nzh;
    const int ytiles = ny / kc;
    const int kz = unit / ytiles, y0 = (unit % ytiles) * kc;
    C *spec = (C *)d.spec, *aacc = (C *)d.aacc;
    const long long plane = (long long)L * ny, cstride = (long long)nzh * plane;
    const long long kb = (long long)kz * plane + y0;
    const C *tw = (const C *)d.twx;
    const int tid = threadIdx.x, nthr = blockDim.x;
    {   // element (yl, x, c), yl fastest
        Idx3 il(tid, nthr, kc, L);
        for (int i = tid; i < NL * L; i += nthr, il.next()) {
            const int yl = il.a0, x = il.a1, c = il.a2;
            cp_asyncc(A + (c * kc + yl) * LP + x + x / N2, spec + c * cstride + kb + (long long)x * ny + yl);
        }
        cp_async_wait_all();
    }
    __syncthreads();
    xg_pass1<C, N1, N2, -1>(A, NL, tw);
    __syncthreads();
    for (int task = tid; task < NL * N1; task += nthr) {
        const int l = task / N1, k1 = task - l * N1;
        const C *p = A + l * LP + (N2 + 1) * k1;
        C x[N2];
#pragma unroll
        for (int t = 0; t < N2; ++t) x[t] = p[t];
        sdft<N2, -1, 0, 1>(x);
        C *q = B + l * LP;
        sfor<0, N2>([&](auto mc) {
            const int k = k1 + N1 * decltype(mc)::v;
            q[k + k / N2] = x[dft_pos(N2, decltype(mc)::v)];
        });
    }
    __syncthreads();
    // the accumulator's tile, acc[(c L + x) kc + yl], staged in the free A
    const int first = d.macro->first_iter;
    if (!first) {
        Idx3 il(tid, nthr, kc, L);
        for (int i = tid; i < 3 * L * kc; i += nthr, il.next())
            cp_asyncc(A + i, aacc + il.a2 * cstride + kb + (long long)il.a1 * ny + il.a0);
        cp_async_wait_all();
        __syncthreads();
    }
    // the Green operator at frequency (x, y0 + yl, kz), yl fastest
    Idx3 ig(tid, nthr, kc, kIdxUnbounded);
    for (int idx = tid; idx < L * kc; idx += nthr, ig.next()) {
        const int yl = ig.a0, x = ig.a1, px = x + x / N2;
        R br[6], bi[6], ar[3], ai[3];
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            const C e = B[(c * kc + yl) * LP + px];
            br[c] = e.x;
            bi[c] = e.y;
        }
        const long long o = kb + (long long)x * ny + yl;
        green_apply<R>(d, x, y0 + yl, kz, o, br, bi, ar, ai);
#pragma unroll
        for (int c = 0; c < 6; ++c) B[(c * kc + yl) * LP + px] = mkc<C>(br[c], bi[c]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            C e = mkc<C>(ar[c], ai[c]);
            if (!first) {
                const C a = A[(c * L + x) * kc + yl];
                e.x += a.x;
                e.y += a.y;
            }
            aacc[c * cstride + o] = e;
        }
    }
    __syncthreads();
    xg_pass1<C, N1, N2, 1>(B, NL, tw);
    __syncthreads();
    // inverse pass 2: tasks (l, k1), l fastest, written to spectrum line l
    {
        const long long sN = (long long)N1 * ny;
        const int dl = nthr % NL, dk = nthr / NL;
        int l = tid % NL, k1 = tid / NL;
        for (int task = tid; task < NL * N1; task += nthr) {
            const C *p = B + l * LP + (N2 + 1) * k1;
            C x[N2];
#pragma unroll
            for (int t = 0; t < N2; ++t) x[t] = p[t];
            sdft<N2, 1, 0, 1>(x);
            const int c = l / kc, yl = l - c * kc;
            C *g = spec + c * cstride + kb + yl + (long long)k1 * ny;
            sfor<0, N2>([&](auto mc) { g[decltype(mc)::v * sN] = x[dft_pos(N2, decltype(mc)::v)]; });
            l += dl;
            k1 += dk;
            if (l >= NL) { l -= NL; ++k1; }
        }
    }
}

// smem of xg_unit, bytes
template <typename C>
__host__ __device__ inline size_t xg_smem(int nx, int n1, int kc)
{
    return 2 * sizeof(C) * (size_t)(6 * kc) * (size_t)(nx + n1 + 1);
}
// whether the RVE's x pass runs xg_unit: an axis on the register FFT whose
// tile fits in a block in xg_unit's padded layout.  A larger tile, which fits
// in the two line buffers of fft_lines alone, goes through those
// (fft_x_green_unit), with the same results.
template <typename C>
__host__ __device__ inline bool xg_fits(const RveDesc &d)
{
    return d.plx.n1 > 0 && xg_smem<C>(d.nx, d.plx.n1, d.xkc) <= kBlockSmem;
}

template <typename R>
__device__ void fft_x_unit(const RveDesc &d, void *specp, int ncomp, int sign, int kc, int unit)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bufA = reinterpret_cast<C *>(smem_raw);
    const int nx = d.nx, ny = d.ny, nzh = d.nzh;
    const int NL = ncomp * kc, ldl = NL | 1;
    C *bufB = bufA + nx * ldl;
    const int ytiles = ny / kc;
    const int kz = unit / ytiles, y0 = (unit % ytiles) * kc;
    C *spec = (C *)specp;
    const long long plane = (long long)nx * ny, cstride = (long long)nzh * plane;
    const long long kb = (long long)kz * plane + y0;
    if constexpr (sizeof(R) == 4) {
        Idx3 il(threadIdx.x, blockDim.x, kc, nx);
        for (int i = threadIdx.x; i < ncomp * nx * kc; i += blockDim.x, il.next())
            cp_async8(&bufA[il.a0 + il.a1 * ldl + il.a2 * kc],
                      spec + il.a2 * cstride + kb + (long long)il.a1 * ny + il.a0);
        cp_async_wait_all();
    } else {
        staged_copy3<CopyDepth<R>::v, C>(
            ncomp * nx * kc, kc, nx,
            [&](int yl, int x, int c) { return spec[c * cstride + kb + (long long)x * ny + yl]; },
            [&](int yl, int x, int c, C v) { bufA[x * ldl + c * kc + yl] = v; });
    }
    __syncthreads();
    C *res = fft_lines<R>(bufA, bufB, NL, ldl, d.plx, (const C *)d.twx, sign);
    Idx3 is(threadIdx.x, blockDim.x, kc, nx);
    for (int idx = threadIdx.x; idx < ncomp * nx * kc; idx += blockDim.x, is.next()) {
        const int yl = is.a0, x = is.a1, c = is.a2;
        spec[c * cstride + kb + (long long)x * ny + yl] = res[x * ldl + c * kc + yl];
    }
}


// Shared memory of the single-precision z passes, in complex floats.  The
// forward pass stages the six stress runs (rows x nz doubles each) behind
// its first line buffer; the inverse one (mode 0) stages the raw half-spectrum
// columns there and the old displacement-gradient runs after both buffers.
__host__ __device__ inline long long zf32_lines(int nz, int rows) { return (long long)nz * ((3 * rows) | 1); }
__host__ __device__ inline long long zf32_fwd_size(int nz, int rows)
{
    const long long a = zf32_lines(nz, rows), st = 6LL * rows * nz;   // 6 runs of doubles
    return a + (a > st ? a : st);
}
__host__ __device__ inline long long zi32_bregion(int nz, int nzh, int rows)
{
    const long long a = zf32_lines(nz, rows), st = 6LL * nzh * rows;
    return a > st ? a : st;
}
__host__ __device__ inline long long zi32_size(int nz, int nzh, int rows)
{
    return zf32_lines(nz, rows) + zi32_bregion(nz, nzh, rows) + 6LL * rows * nz;   // + 6 runs of doubles
}

// Single-precision inverse z transform of the six stress-update components
// into the symmetric displacement gradient (mode 0 of fft_z_inv_unit, with
// the same arithmetic).  The raw columns S[(c nzh + ks) rows + r] and the
// old gradient runs D[c rows nz + r nz + z] are staged by asynchronous
// copies, the columns first: the block waits for them, and the gradient
// runs arrive while the lines transform.
static __device__ void fft_z_inv_dgs_f32(const RveDesc &d, int rows, int unit)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *bufA = reinterpret_cast<float2 *>(smem_raw);
    const int nx = d.nx, ny = d.ny, nz = d.nz, nzh = d.nzh, half = nz / 2;
    const long long nv = d.nv;
    const int NL = 3 * rows, ldl = NL | 1;
    float2 *bufB = bufA + nz * ldl;
    float2 *S = bufB;
    double *D = reinterpret_cast<double *>(bufA + zf32_lines(nz, rows) + zi32_bregion(nz, nzh, rows));
    const int ytiles = ny / rows;
    const int x = unit / ytiles, y0 = (unit % ytiles) * rows;
    const float2 *spec = (const float2 *)d.spec;
    const long long plane = (long long)nx * ny, cstride = (long long)nzh * plane;
    const long long xy = (long long)x * ny + y0, vb = xy * nz;
    const int run = rows * nz, half_run = run / 2;
    {
        Idx3 is(threadIdx.x, blockDim.x, rows, nzh);   // (r, ks, c)
        for (int i = threadIdx.x; i < 6 * nzh * rows; i += blockDim.x, is.next())
            cp_async8(S + i, spec + is.a2 * cstride + (long long)is.a1 * plane + xy + is.a0);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    {
        Idx3 ic(threadIdx.x, blockDim.x, half_run, kIdxUnbounded);
        for (int i = threadIdx.x; i < 6 * half_run; i += blockDim.x, ic.next())
            cp_async16(D + 2 * i, d.dgs + ic.a1 * nv + vb + 2 * ic.a0);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    // element (r, k, p): line p's coefficient k of row r (components 2p, 2p + 1)
    Idx3 ik(threadIdx.x, blockDim.x, rows, nz);
    for (int i = threadIdx.x; i < 3 * nz * rows; i += blockDim.x, ik.next()) {
        const int r = ik.a0, k = ik.a1, p = ik.a2;
        const int ks = k <= half ? k : nz - k;
        float2 A = S[(2 * p * nzh + ks) * rows + r], B = S[((2 * p + 1) * nzh + ks) * rows + r];
        if (k == 0 || k == half) { A.y = 0.f; B.y = 0.f; }
        if (k > half) { A.y = -A.y; B.y = -B.y; }
        bufA[k * ldl + p * rows + r] = make_float2(A.x - B.y, A.y + B.x);
    }
    __syncthreads();
    const float2 *res = fft_lines<float>(bufA, bufB, NL, ldl, d.plz, (const float2 *)d.twz, +1);
    cp_async_wait_all();
    __syncthreads();
    const MacroDev *m = d.macro;
    // the update val/N as a float product (exact for a power-of-two N):
    // one FP64-pipe operation fewer per value than a product in FP64
    const float inv = (float)d.inv_nv;
    // no mean correction (a load given by its velocity gradient alone): one
    // FP64 addition per value instead of two
    bool mean = false;
#pragma unroll
    for (int c = 0; c < 6; ++c) mean = mean || m->ddg6[c] != 0.0;
    // element (z, r, c) is dgs[c][vb + r * nz + z] = D[i]
    Idx3 iz(threadIdx.x, blockDim.x, nz, rows);
    for (int i = threadIdx.x; i < 6 * run; i += blockDim.x, iz.next()) {
        const int z = iz.a0, r = iz.a1, c = iz.a2;
        const float2 e = res[z * ldl + (c >> 1) * rows + r];
        const float vf = ((c & 1) ? e.y : e.x) * inv;
        double val = finite_f(vf) ? f2d(vf) : (double)vf;
        if (mean) val += m->ddg6[c];
        d.dgs[(long long)c * nv + vb + (long long)r * nz + z] = D[i] + val;
    }
}

// ---------------------------------------------------------------------------
// The z passes of an RVE on the register FFT along z.  A tile is rows lines of
// y at one x; its 3 rows complex lines (two components each, line l = p rows +
// r) are transformed in the layout of the y stream, element (l, i) at l LP +
// i + i / N2.  Pass 1 takes its inputs straight from the staged data -- the
// stress runs, converted on the way, or the half-spectrum columns, unpacked on
// the way -- and the inverse pass 2 adds its outputs straight to the
// displacement gradient, so that a line crosses shared memory once less in
// each direction than through fft_lines and a tile needs two block barriers
// fewer.  Everything is staged by asynchronous copies.
// us per launch, forward / inverse, against the passes through fft_lines:
// single precision 256^3 461 / 950 -> 376 / 667, 96^3 34 / 64 -> 32 / 44; FP64
// 128^3 359 / 408 -> 321 / 329.  Those passes stay for the Stockham stages
// and for tiles that do not fit in a block in this layout (zf_fits, zi_fits).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float from_double(double x, float) { return d2f_rn(x); }
__device__ __forceinline__ double from_double(double x, double) { return x; }

template <typename C, int N1, int N2>
__device__ void zf_unit(const RveDesc &d, int rows, int unit)
{
    typedef typename RealOf<C>::T R;
    constexpr int L = N1 * N2, LP = L + N1 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NL = 3 * rows, run = rows * L, half_run = run / 2;
    C *W = reinterpret_cast<C *>(smem_raw);
    double *stage = reinterpret_cast<double *>(W + ((NL * LP + 1) & ~1));   // the six runs (z fastest)
    C *res = reinterpret_cast<C *>(stage);                                  // then the transformed lines, at l (L + 1) + k
    const int ny = d.ny, nzh = d.nzh, ytiles = ny / rows;
    const int x = unit / ytiles, y0 = (unit - x * ytiles) * rows;
    const long long nv = d.nv, vb = ((long long)x * ny + y0) * L;
    const C *tw = (const C *)d.twz;
    const int tid = threadIdx.x, nthr = blockDim.x;
    {
        Idx3 ic(tid, nthr, half_run, kIdxUnbounded);
        for (int i = tid; i < 6 * half_run; i += nthr, ic.next())
            cp_async16(stage + 2 * i, d.sig + ic.a1 * nv + vb + 2 * ic.a0);
        cp_async_wait_all();
    }
    __syncthreads();
    for (int task = tid; task < NL * N2; task += nthr) {
        const int l = task / N2, t = task - l * N2, p = l / rows, r = l - p * rows;
        const double *a = stage + 2 * p * run + r * L + t;
        C v[N1];
        sfor<0, N1>([&](auto jc) {
            constexpr int j = decltype(jc)::v;
            v[j] = mkc<C>(from_double(a[j * N2], R(0)), from_double(a[run + j * N2], R(0)));
        });
        sdft<N1, -1, 0, 1>(v);
        if (t != 0) {
            const C *wm = tw + L + t;   // the pass-1 twiddle matrix
            sfor<1, N1>([&](auto kc) {
                constexpr int k = decltype(kc)::v, q = dft_pos(N1, k);
                v[q] = cmul<R>(v[q], __ldg(wm + k * N2));
            });
        }
        C *w = W + l * LP + t;
        sfor<0, N1>([&](auto kc) { w[(N2 + 1) * decltype(kc)::v] = v[dft_pos(N1, decltype(kc)::v)]; });
    }
    __syncthreads();
    for (int task = tid; task < NL * N1; task += nthr) {
        const int l = task / N1, k1 = task - l * N1;
        const C *w = W + l * LP + (N2 + 1) * k1;
        C v[N2];
#pragma unroll
        for (int t = 0; t < N2; ++t) v[t] = w[t];
        sdft<N2, -1, 0, 1>(v);
        C *q = res + l * (L + 1) + k1;
        sfor<0, N2>([&](auto mc) { q[N1 * decltype(mc)::v] = v[dft_pos(N2, decltype(mc)::v)]; });
    }
    __syncthreads();
    C *spec = (C *)d.spec;
    const long long plane = (long long)d.nx * ny;
    Idx3 ix(tid, nthr, rows, nzh);
    for (int i = tid; i < 3 * rows * nzh; i += nthr, ix.next()) {
        const int r = ix.a0, k = ix.a1, p = ix.a2;
        const C *q = res + (p * rows + r) * (L + 1);
        const C zk = q[k], zm = q[k ? L - k : 0];
        const long long o = (long long)k * plane + (long long)x * ny + y0 + r;
        spec[(long long)(2 * p) * nzh * plane + o] = mkc<C>(R(0.5) * (zk.x + zm.x), R(0.5) * (zk.y - zm.y));
        spec[(long long)(2 * p + 1) * nzh * plane + o] = mkc<C>(R(0.5) * (zk.y + zm.y), R(-0.5) * (zk.x - zm.x));
    }
}

template <typename C>
__host__ __device__ inline size_t zf_smem(int nz, int n1, int rows)
{
    const size_t w = (((size_t)(3 * rows) * (nz + n1 + 1) + 1) & ~(size_t)1) * sizeof(C);
    const size_t st = sizeof(double) * 6 * (size_t)rows * nz, res = sizeof(C) * (size_t)(3 * rows) * (nz + 1);
    return w + (st > res ? st : res);
}

// the inverse pass into the symmetric displacement gradient (evolution.c:383-394)
template <bool MEAN, bool FINITE>
__device__ __forceinline__ double add_update(double old, float v, float inv, double m)
{
    const float f = v * inv;   // (exact for a power-of-two number of voxels)
    const double x = FINITE ? f2d(f) : (double)f;
    return MEAN ? old + (x + m) : old + x;
}
template <bool MEAN, bool FINITE>
__device__ __forceinline__ double add_update(double old, double v, double inv, double m)
{
    return MEAN ? old + fma(v, inv, m) : fma(v, inv, old);
}

// pass 2 of zi_unit; MEAN: the update has a mean part (MacroDev::ddg6)
template <typename C, int N1, int N2, bool MEAN>
__device__ __forceinline__ void zi_pass2(const RveDesc &d, const C *W, const double *D, int rows, long long vb)
{
    typedef typename RealOf<C>::T R;
    constexpr int L = N1 * N2, LP = L + N1 + 1;
    const int run = rows * L;
    const long long nv = d.nv;
    const MacroDev *m = d.macro;
    const R inv = (R)d.inv_nv;
    for (int task = threadIdx.x; task < 3 * rows * N1; task += blockDim.x) {
        const int l = task / N1, k1 = task - l * N1, p = l / rows, r = l - p * rows;
        const C *w = W + l * LP + (N2 + 1) * k1;
        C v[N2];
#pragma unroll
        for (int t = 0; t < N2; ++t) v[t] = w[t];
        sdft<N2, 1, 0, 1>(v);
        const double *o = D + 2 * p * run + r * L + k1;
        double *g = d.dgs + 2 * p * nv + vb + r * L + k1;
        const double m0 = MEAN ? m->ddg6[2 * p] : 0.0, m1 = MEAN ? m->ddg6[2 * p + 1] : 0.0;
        auto put = [&](auto finite) {
            sfor<0, N2>([&](auto mc) {
                constexpr int q = N1 * decltype(mc)::v, e = dft_pos(N2, decltype(mc)::v);
                g[q] = add_update<MEAN, decltype(finite)::v>(o[q], v[e].x, inv, m0);
                g[nv + q] = add_update<MEAN, decltype(finite)::v>(o[run + q], v[e].y, inv, m1);
            });
        };
        // X[0] is the sum of the inputs: it is finite only if all of them are
        // (single precision converts finite values alone by their bits)
        if (sizeof(R) == 8 || finite_f((float)v[0].x + (float)v[0].y)) put(IC<1>());
        else put(IC<0>());
    }
}

template <typename C, int N1, int N2>
__device__ void zi_unit(const RveDesc &d, int rows, int unit)
{
    typedef typename RealOf<C>::T R;
    constexpr int L = N1 * N2, LP = L + N1 + 1, nzh = L / 2 + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NL = 3 * rows, run = rows * L, half_run = run / 2;
    C *W = reinterpret_cast<C *>(smem_raw);
    double *D = reinterpret_cast<double *>(W + ((NL * LP + 1) & ~1));   // the old gradient: six runs (z fastest)
    C *S = reinterpret_cast<C *>(D + 6 * run);                          // columns: S[(c nzh + k) rows + r]
    const int ny = d.ny, ytiles = ny / rows;
    const int x = unit / ytiles, y0 = (unit - x * ytiles) * rows;
    const long long nv = d.nv, xy = (long long)x * ny + y0, vb = xy * L;
    const long long plane = (long long)d.nx * ny, cstride = (long long)nzh * plane;
    const C *spec = (const C *)d.spec, *tw = (const C *)d.twz;
    const int tid = threadIdx.x, nthr = blockDim.x;
    {
        Idx3 is(tid, nthr, rows, nzh);   // (r, k, c)
        for (int i = tid; i < 6 * nzh * rows; i += nthr, is.next())
            cp_asyncc(S + i, spec + is.a2 * cstride + (long long)is.a1 * plane + xy + is.a0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        Idx3 ic(tid, nthr, half_run, kIdxUnbounded);
        for (int i = tid; i < 6 * half_run; i += nthr, ic.next())
            cp_async16(D + 2 * i, d.dgs + ic.a1 * nv + vb + 2 * ic.a0);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
    }
    __syncthreads();
    {
        const int dl = nthr % NL, dt = nthr / NL;
        int l = tid % NL, t = tid / NL;
        for (int task = tid; task < NL * N2; task += nthr) {
            const int p = l / rows, r = l - p * rows;
            const C *a = S + (long long)2 * p * nzh * rows + r, *b = a + nzh * rows;
            C v[N1];
            sfor<0, N1>([&](auto jc) {
                constexpr int j = decltype(jc)::v;
                constexpr bool hi = j >= N1 / 2;   // coefficient k = t + N2 j: k >= L / 2
                const int k = hi ? L - t - N2 * j : t + N2 * j;
                C A = a[k * rows], B = b[k * rows];
                if (hi) { A.y = -A.y; B.y = -B.y; }
                if ((j == 0 || j == N1 / 2) && t == 0) { A.y = R(0); B.y = R(0); }
                v[j] = mkc<C>(A.x - B.y, A.y + B.x);
            });
            sdft<N1, 1, 0, 1>(v);
            if (t != 0) {
                const C *wm = tw + L + t;
                sfor<1, N1>([&](auto kc) {
                    constexpr int k = decltype(kc)::v, q = dft_pos(N1, k);
                    C w = __ldg(wm + k * N2);
                    w.y = -w.y;
                    v[q] = cmul<R>(v[q], w);
                });
            }
            C *w = W + l * LP + t;
            sfor<0, N1>([&](auto kc) { w[(N2 + 1) * decltype(kc)::v] = v[dft_pos(N1, decltype(kc)::v)]; });
            l += dl;
            t += dt;
            if (l >= NL) { l -= NL; ++t; }
        }
    }
    cp_async_wait_all();
    __syncthreads();
    // no mean correction (a load given by its velocity gradient alone): one
    // FP64 operation per value fewer
    const double *g6 = d.macro->ddg6;
    long long any = 0;
#pragma unroll
    for (int c = 0; c < 6; ++c) any |= __double_as_longlong(g6[c]) << 1;   // (but for the sign)
    if (any) zi_pass2<C, N1, N2, true>(d, W, D, rows, vb);
    else zi_pass2<C, N1, N2, false>(d, W, D, rows, vb);
}

template <typename C>
__host__ __device__ inline size_t zi_smem(int nz, int n1, int rows)
{
    return (((size_t)(3 * rows) * (nz + n1 + 1) + 1) & ~(size_t)1) * sizeof(C) + sizeof(double) * 6 * (size_t)rows * nz +
           sizeof(C) * 6 * (size_t)(nz / 2 + 1) * rows;
}

// whether the RVE's z passes run zf_unit, zi_unit (as xg_fits): larger tiles
// go through fft_lines
template <typename C>
__host__ __device__ inline bool zf_fits(const RveDesc &d)
{
    return d.plz.n1 > 0 && zf_smem<C>(d.nz, d.plz.n1, d.zrows) <= kBlockSmem;
}
template <typename C>
__host__ __device__ inline bool zi_fits(const RveDesc &d)
{
    return d.plz.n1 > 0 && zi_smem<C>(d.nz, d.plz.n1, d.zirows) <= kBlockSmem;
}

// inverse z transform (Hermitian half spectrum -> real); mode 0 adds the
// result to the symmetric displacement gradient (evolution.c:383-394),
// mode 1 writes it (scaled by 1/N) to rotl, mode 2 (scaled by 1/N) to
// out[ncomp * v + c], voxel by voxel
template <typename R>
__device__ void fft_z_inv_unit(const RveDesc &d, void *specp, int ncomp, int rows, int mode, int unit,
                               double *out = nullptr)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *bufA = reinterpret_cast<C *>(smem_raw);
    const int nx = d.nx, ny = d.ny, nz = d.nz, nzh = d.nzh;
    const long long nv = d.nv;
    const int np = (ncomp + 1) / 2;
    const int NL = np * rows, ldl = NL | 1;
    C *bufB = bufA + nz * ldl;
    const int ytiles = ny / rows;
    const int x = unit / ytiles, y0 = (unit % ytiles) * rows;
    const C *spec = (const C *)specp;
    const long long plane = (long long)nx * ny, cstride = (long long)nzh * plane;
    const long long xy = (long long)x * ny + y0;
    const int half = nz / 2;
    struct AB { C a, b; };
    // element (r, k, p): line p's coefficient k of row r
    staged_copy3<kZCopyDepth, AB>(
        np * nz * rows, rows, nz,
        [&](int r, int k, int p) {
            const int ca = 2 * p, cb = 2 * p + 1;
            const int ks = k <= half ? k : nz - k;
            const long long o = (long long)ks * plane + xy + r;
            AB v;
            v.a = spec[ca * cstride + o];
            if (cb < ncomp) v.b = spec[cb * cstride + o];
            else { v.b.x = R(0); v.b.y = R(0); }
            return v;
        },
        [&](int r, int k, int p, AB v) {
            const bool lo = k <= half;
            C A = v.a, B = v.b;
            if (k == 0 || k == half) { A.y = R(0); B.y = R(0); }
            if (!lo) { A.y = -A.y; B.y = -B.y; }
            C Z;
            Z.x = A.x - B.y;
            Z.y = A.y + B.x;
            bufA[k * ldl + p * rows + r] = Z;
        });
    __syncthreads();
    const C *res = fft_lines<R>(bufA, bufB, NL, ldl, d.plz, (const C *)d.twz, +1);
    const long long vb = xy * nz;
    const double inv = d.inv_nv;
    if (mode == 0) {
        const MacroDev *m = d.macro;
        // on the register FFT, the arithmetic of zi_unit's add_update
        bool direct = d.plz.n1 > 0;
#pragma unroll
        for (int c = 0; c < 6; ++c) direct = direct && m->ddg6[c] == 0.0;
        // element (z, r, c) is dgs[c][vb + r * nz + z]
        staged_copy3<kZCopyDepth, double>(
            ncomp * rows * nz, nz, rows,
            [&](int z, int r, int c) { return d.dgs[(long long)c * nv + vb + (long long)r * nz + z]; },
            [&](int z, int r, int c, double old) {
                const C e = res[z * ldl + (c >> 1) * rows + r];
                const double val = (double)((c & 1) ? e.y : e.x);
                d.dgs[(long long)c * nv + vb + (long long)r * nz + z] =
                    direct ? fma(val, inv, old) : old + fma(val, inv, m->ddg6[c]);
            });
    } else if (mode == 1) {
        Idx3 iz(threadIdx.x, blockDim.x, nz, rows);
        for (int idx = threadIdx.x; idx < ncomp * rows * nz; idx += blockDim.x, iz.next()) {
            const int z = iz.a0, r = iz.a1, c = iz.a2;
            const C e = res[z * ldl + (c >> 1) * rows + r];
            const double val = (double)((c & 1) ? e.y : e.x);
            d.rotl[(long long)c * nv + vb + (long long)r * nz + z] = val * inv;
        }
    } else {
        for (int idx = threadIdx.x; idx < ncomp * rows * nz; idx += blockDim.x) {
            const int c = idx % ncomp, t = idx / ncomp, z = t % nz, r = t / nz;
            const C e = res[z * ldl + (c >> 1) * rows + r];
            const double val = (double)((c & 1) ? e.y : e.x);
            out[ncomp * (vb + (long long)r * nz + z) + c] = val * inv;
        }
    }
}


// ===========================================================================
// batched entry points: one launch per phase covers many RVEs.  Work item w
// of a phase is map[w] = (rve, unit); the unit functions are the ones the
// single-RVE kernels call, so an RVE computes the same numbers alone and in
// a batch.  RVEs are skipped per phase by their macro flags.
// ===========================================================================
enum { MASK_ACTIVE = 0, MASK_CONVERGED = 1, MASK_PRELUDE = 2 };

__device__ __forceinline__ bool unit_on(const RveDesc &d, int mask)
{
    const MacroDev *m = d.macro;
    if (!m->active) return false;
    if (mask == MASK_CONVERGED) return m->converged != 0;
    if (mask == MASK_PRELUDE) return m->pending_prelude != 0;
    return true;
}

// resident blocks per SM the single-precision z passes are compiled for
// (256^3, mixed forms, us per launch: z forward / inverse 461 / 946 at 2,
// 524 / 1239 at 3, 586 / 1319 at 4, 461 / 1098 at 1)
// The FP64 passes run blocks of 128 threads, six per SM (five for the Green
// pass): they are bound by the FP64 pipe, and a block that loads or stores
// leaves it to the others.  64^3, us per launch of z forward / y / x + Green /
// z inverse, with the register FFT: 256 threads, 2 blocks 56 / 41 / 149 / 67,
// 3 blocks 52 / 41 / 146 / 60; 128 threads, 4 blocks 53 / 40 / 137 / 63, 5
// blocks 47 / 38 / 131 / 57; 64 threads, 8 blocks 52 / 40 / 141 / 64.  The
// Stockham stages, 256 threads: 53 / 51 / 157 / 66.
template <typename R> struct FftThreads { static constexpr int v = 256; };
template <> struct FftThreads<double> { static constexpr int v = 128; };
constexpr int kFft64Blocks = 6, kFftXg64Blocks = 5;
// most blocks of a pass's grid, per SM
template <typename R> struct FftGrid { static constexpr int v = 4; };
template <> struct FftGrid<double> { static constexpr int v = 2 * kFft64Blocks; };
#ifndef VOCE_FFTZ32_BLOCKS
#define VOCE_FFTZ32_BLOCKS 2
#endif
template <typename R>
__global__ void __launch_bounds__(FftThreads<R>::v, sizeof(R) == 4 ? VOCE_FFTZ32_BLOCKS : kFft64Blocks)
kb_fft_z_fwd(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_ACTIVE)) continue;
        typedef typename Cx<R>::T C;
        if (zf_fits<C>(d)) {
#define VOCE_CALL(N1, N2) if constexpr (N1 * N2 % 2 == 0) zf_unit<C, N1, N2>(d, d.zrows, e.y)   /* nz is even */
            VOCE_REG_SPLITS(d.nz, VOCE_CALL)
#undef VOCE_CALL
        } else {
            fft_z_fwd_unit<R>(d, d.zrows, e.y);
        }
        __syncthreads();
    }
}

// which: 0 spectrum forward, 1 spectrum inverse, 2 antisymmetric accumulator inverse
// cp.async of a y tile (NL lines of L contiguous coefficients at g) into the
// stream layout; where L divides the number of threads a thread keeps its
// coefficient index and steps by whole lines
template <typename C, int N1, int N2, int NT>
__device__ __forceinline__ void ystream_issue(C *A, const C *g, int NL)
{
    constexpr int L = N1 * N2, LP = L + N1 + 1;
    if constexpr (NT % L == 0) {   // (NT threads)
        constexpr int dl = NT / L;
        const int i = threadIdx.x % L;
        C *s = A + (threadIdx.x / L) * LP + i + i / N2;
        const C *src = g + threadIdx.x;
        for (int l = threadIdx.x / L; l < NL; l += dl, s += dl * LP, src += NT) cp_asyncc(s, src);
    } else {
        for (int e = threadIdx.x; e < NL * L; e += blockDim.x) {
            const int l = e / L, i = e - l * L;
            cp_asyncc(A + l * LP + i + i / N2, g + e);
        }
    }
}

template <typename R>
__device__ void fft_y_stream(const RveDesc *descs, const int2 *map, int total, int which, int S)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *cur = reinterpret_cast<C *>(smem_raw), *nxt = cur + S;
    const int mask = which == 2 ? MASK_CONVERGED : MASK_ACTIVE;
    const int sign = which == 0 ? -1 : +1;
    auto next_on = [&](int w) {
        while (w < total && !unit_on(descs[map[w].x], mask)) w += gridDim.x;
        return w;
    };
    // the unit's RVE, its spectrum (y lines: contiguous) and tile base
    auto tile = [&](int w, const RveDesc *&dp, C *&g) {
        const int2 e = map[w];
        dp = &descs[e.x];
        const RveDesc &d = *dp;
        const int xtiles = d.nx / d.yxt;
        const int line = e.y / xtiles, x0 = (e.y % xtiles) * d.yxt;
        g = (C *)(which == 2 ? d.aacc : d.spec) + ((long long)line * d.nx + x0) * d.ny;
    };
    auto issue = [&](int w, C *A) {
        const RveDesc *dp;
        C *g;
        tile(w, dp, g);
#define VOCE_CALL(N1, N2) ystream_issue<C, N1, N2, FftThreads<R>::v>(A, g, dp->yxt)
        VOCE_REG_SPLITS(dp->ny, VOCE_CALL)
#undef VOCE_CALL
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int w = next_on(blockIdx.x);
    if (w < total) issue(w, cur);
    while (w < total) {
        const int nw = next_on(w + gridDim.x);
        if (nw < total) {
            issue(nw, nxt);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            cp_async_wait_all();
        }
        __syncthreads();
        const RveDesc *dp;
        C *g;
        tile(w, dp, g);
        const C *tw = (const C *)dp->twy;
        const int NL = dp->yxt;
        if (sign < 0) {
#define VOCE_CALL(N1, N2) ystream_tile<C, N1, N2, -1>(cur, NL, g, tw)
            VOCE_REG_SPLITS(dp->ny, VOCE_CALL)
#undef VOCE_CALL
        } else {
#define VOCE_CALL(N1, N2) ystream_tile<C, N1, N2, 1>(cur, NL, g, tw)
            VOCE_REG_SPLITS(dp->ny, VOCE_CALL)
#undef VOCE_CALL
        }
        __syncthreads();
        C *t = cur; cur = nxt; nxt = t;
        w = nw;
    }
}

// resident blocks per SM the single-precision y and Green passes are
// compiled for (their register budget)
#ifndef VOCE_FFTY32_BLOCKS
#define VOCE_FFTY32_BLOCKS 2
#endif
#ifndef VOCE_FFTXG32_BLOCKS
#define VOCE_FFTXG32_BLOCKS 2
#endif
template <typename R>
__global__ void __launch_bounds__(FftThreads<R>::v, sizeof(R) == 4 ? VOCE_FFTY32_BLOCKS : kFft64Blocks)
kb_fft_y(const RveDesc *descs, const int2 *map, int total, int which, int stream)
{
    if (stream > 0) {
        fft_y_stream<R>(descs, map, total, which, stream);
        return;
    }
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, which == 2 ? MASK_CONVERGED : MASK_ACTIVE)) continue;
        fft_y_unit<R>(d, which == 2 ? d.aacc : d.spec, which == 0 ? -1 : +1, d.yxt, e.y);
        __syncthreads();
    }
}

// resident blocks per SM the Green pass is compiled for (registers) with the
// FP32 spectrum (256^3, us per launch: 641 at 2, 1095 at 3, 1227 at 4: the register
// FFT spills below 128 registers)
template <typename R>
__global__ void __launch_bounds__(FftThreads<R>::v, sizeof(R) == 8 ? kFftXg64Blocks : VOCE_FFTXG32_BLOCKS)
kb_fft_x_green(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_ACTIVE)) continue;
        typedef typename Cx<R>::T C;
        if (xg_fits<C>(d)) {
#define VOCE_CALL(N1, N2) xg_unit<C, N1, N2>(d, d.xkc, e.y)
            VOCE_REG_SPLITS(d.nx, VOCE_CALL)
#undef VOCE_CALL
        } else {
            fft_x_green_unit<R>(d, d.xkc, e.y);
        }
        __syncthreads();
    }
}

template <typename R>
__global__ void __launch_bounds__(FftThreads<R>::v) kb_fft_x_aacc(const RveDesc *descs, const int2 *map, int total)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, MASK_CONVERGED)) continue;
        fft_x_unit<R>(d, d.aacc, 3, +1, d.xkc3, e.y);
        __syncthreads();
    }
}

// mode 0: spectrum -> displacement gradient; 1: accumulator -> rotl
template <typename R>
__global__ void __launch_bounds__(FftThreads<R>::v, sizeof(R) == 4 ? VOCE_FFTZ32_BLOCKS : kFft64Blocks)
kb_fft_z_inv(const RveDesc *descs, const int2 *map, int total, int mode)
{
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int2 e = map[w];
        const RveDesc &d = descs[e.x];
        if (!unit_on(d, mode == 0 ? MASK_ACTIVE : MASK_CONVERGED)) continue;
        typedef typename Cx<R>::T C;
        if (mode == 0 && zi_fits<C>(d)) {
#define VOCE_CALL(N1, N2) if constexpr (N1 * N2 % 2 == 0) zi_unit<C, N1, N2>(d, d.zirows, e.y)
            VOCE_REG_SPLITS(d.nz, VOCE_CALL)
#undef VOCE_CALL
        } else if (mode == 0) {
            if constexpr (sizeof(R) == 4) fft_z_inv_dgs_f32(d, d.zirows, e.y);
            else fft_z_inv_unit<R>(d, d.spec, 6, d.zirows, 0, e.y);
        } else {
            fft_z_inv_unit<R>(d, d.aacc, 3, d.zirows3, 1, e.y);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename R>
static size_t smem_lines(int L, int NL)
{
    return (size_t)2 * L * (size_t)(NL | 1) * sizeof(typename Cx<R>::T);
}


static inline int grid_for(int total, int cap)
{
    return total < cap ? (total > 0 ? total : 1) : cap;
}


template <typename R>
static void launch_fft_t(const BatchPlan &bp, FftPass pass, cudaStream_t s)
{
    static const int phase[] = {BP_ZF, BP_Y6, BP_XG, BP_Y6, BP_ZI, BP_X3, BP_Y3, BP_Z3};
    const int ph = phase[pass], n = bp.total[ph], g = grid_for(n, 152 * FftGrid<R>::v);
    const size_t sm = bp.smem[ph];
    const RveDesc *D = bp.descs;
    const int2 *map = bp.map[ph];
    constexpr int T = FftThreads<R>::v;
    switch (pass) {
    case FFT_ZF: kb_fft_z_fwd<R><<<g, T, sm, s>>>(D, map, n); break;
    case FFT_YF: kb_fft_y<R><<<g, T, sm, s>>>(D, map, n, 0, bp.ystream); break;
    case FFT_XG: kb_fft_x_green<R><<<g, T, sm, s>>>(D, map, n); break;
    case FFT_YI: kb_fft_y<R><<<g, T, sm, s>>>(D, map, n, 1, bp.ystream); break;
    case FFT_ZI: kb_fft_z_inv<R><<<g, T, sm, s>>>(D, map, n, 0); break;
    case FFT_X3: kb_fft_x_aacc<R><<<g, T, sm, s>>>(D, map, n); break;
    case FFT_Y3: kb_fft_y<R><<<g, T, sm, s>>>(D, map, n, 2, bp.ystream); break;
    case FFT_Z3: kb_fft_z_inv<R><<<g, T, sm, s>>>(D, map, n, 1); break;
    }
}

template <typename R>
static cudaError_t set_fft_smem_t(const BatchPlan &bp)
{
    auto set = [](const void *fn, size_t b) {
        if (b) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b);
    };
    set((const void *)kb_fft_z_fwd<R>, bp.smem[BP_ZF]);
    set((const void *)kb_fft_y<R>, std::max(bp.smem[BP_Y6], bp.smem[BP_Y3]));
    set((const void *)kb_fft_x_green<R>, bp.smem[BP_XG]);
    set((const void *)kb_fft_x_aacc<R>, bp.smem[BP_X3]);
    set((const void *)kb_fft_z_inv<R>, std::max(bp.smem[BP_ZI], bp.smem[BP_Z3]));
    return cudaGetLastError();
}

#define VOCE_FFT_INSTANCE(R) \
    template <> void launch_fft<R>(const BatchPlan &bp, FftPass pass, cudaStream_t s) { launch_fft_t<R>(bp, pass, s); } \
    template <> cudaError_t set_fft_smem<R>(const BatchPlan &bp) { return set_fft_smem_t<R>(bp); }

}  // namespace voce
