// The displacement fluctuation, and the probe of the line FFT.
#include "voce_fft.cuh"

namespace voce {

// ---------------------------------------------------------------------------
// Displacement fluctuation: the periodic field u~ whose gradient is the
// fluctuating part of DisGrad, in voxel units of length.  The reference means
// to compute it at evolution.c:532-560 from
//   u^_i(k) = -i sum_j F^_ij(k) g_j(k),   u~ = Re(IFFT(u^)) / N
// but sums tmp_re/tmp_im into one scalar per component over all voxels, then
// stores it at a stale voxel index, and its g = xi/|xi| (init.c:660-676)
// lacks the 1/|xi| an inverse gradient needs.  Here F is DisGrad (its
// fluctuating part is the reference's `fluctuation`, evolution.c:392, up to
// the uniform terms that only reach k = 0), g_j = xi_j/|xi|^2 with the
// reference's frequencies xi, g(0) = 0, and the real part is taken the way
// the Green operator takes it: the spectrum is replaced by its Hermitian part
// (X(k) + conj X(-k))/2, which turns g into (g(k) - g(-k))/2 and cancels the
// terms along a Nyquist coordinate.  The work array holds [9][nzh][nx][ny]
// complex values of the spectrum type: DisGrad's six B-basis symmetric
// components, then its three antisymmetric ones.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void freq_over_sq(const RveDesc &d, int ix, int iy, int iz, double (&q)[3])
{
    const double g0 = kfreq(ix, d.inv_n[0]), g1 = kfreq(iy, d.inv_n[1]), g2 = kfreq(iz, d.inv_n[2]);
    const double s = 1.0 / (g0 * g0 + g1 * g1 + g2 * g2);
    q[0] = g0 * s; q[1] = g1 * s; q[2] = g2 * s;
}

// which 0: the symmetric part into components 0-5; 1: the antisymmetric
// part into 6-8
template <typename R>
__global__ void __launch_bounds__(256) k_disp_z_fwd(RveDesc d, void *work, int which, int total)
{
    typedef typename Cx<R>::T C;
    C *anti = (C *)work + 6 * d.nspec;
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        if (which == 0) fft_z_fwd_src<R, 6>(d, d.dgs, work, d.zrows, u);
        else fft_z_fwd_src<R, 3>(d, d.dga, anti, d.zirows3, u);
        __syncthreads();
    }
}

template <typename R>
__global__ void __launch_bounds__(256) k_disp_fft_y(RveDesc d, void *work, int sign, int total)
{
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        fft_y_unit<R>(d, work, sign, d.yxt, u);
        __syncthreads();
    }
}

template <typename R>
__global__ void __launch_bounds__(256) k_disp_fft_x(RveDesc d, void *work, int ncomp, int sign, int kc, int total)
{
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        fft_x_unit<R>(d, work, ncomp, sign, kc, u);
        __syncthreads();
    }
}

// per frequency: the nine transformed components -> u^ in components 0-2
template <typename R>
__global__ void __launch_bounds__(256) k_disp_spec(RveDesc d, void *work)
{
    typedef typename Cx<R>::T C;
    C *w = (C *)work;
    const long long ns = d.nspec, plane = (long long)d.nx * d.ny;
    for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < ns;
         o += (long long)gridDim.x * blockDim.x) {
        const int iz = (int)(o / plane), ix = (int)((o % plane) / d.ny), iy = (int)(o % d.ny);
        double q[3] = {0.0, 0.0, 0.0};
        if ((ix | iy | iz) != 0) {
            double a[3], b[3];
            freq_over_sq(d, ix, iy, iz, a);
            freq_over_sq(d, (d.nx - ix) % d.nx, (d.ny - iy) % d.ny, (d.nz - iz) % d.nz, b);
            for (int m = 0; m < 3; ++m) q[m] = 0.5 * (a[m] - b[m]);
        }
        double br[6], bi[6], Fr[9], Fi[9];
        for (int c = 0; c < 6; ++c) {
            const C e = w[c * ns + o];
            br[c] = (double)e.x;
            bi[c] = (double)e.y;
        }
        sym9_from_b(br, Fr);
        sym9_from_b(bi, Fi);
        // antisymmetric parts (D12-D21)/2, (D02-D20)/2, (D01-D10)/2
        const int ij[3] = {5, 2, 1}, ji[3] = {7, 6, 3};
        for (int c = 0; c < 3; ++c) {
            const C e = w[(6 + c) * ns + o];
            Fr[ij[c]] += (double)e.x; Fr[ji[c]] -= (double)e.x;
            Fi[ij[c]] += (double)e.y; Fi[ji[c]] -= (double)e.y;
        }
        for (int i = 0; i < 3; ++i) {
            double ur = 0.0, ui = 0.0;   // -i (Fr + i Fi) q = Fi q - i Fr q
            for (int j = 0; j < 3; ++j) {
                ur = fma(Fi[3 * i + j], q[j], ur);
                ui = fma(-Fr[3 * i + j], q[j], ui);
            }
            C e;
            e.x = (R)ur;
            e.y = (R)ui;
            w[i * ns + o] = e;
        }
    }
}

template <typename R>
__global__ void __launch_bounds__(256) k_disp_z_inv(RveDesc d, void *work, double *out, int total)
{
    for (int u = blockIdx.x; u < total; u += gridDim.x) {
        fft_z_inv_unit<R>(d, work, 3, d.zirows3, 2, u, out);
        __syncthreads();
    }
}

template <typename R>
static cudaError_t disp_fluct_t(const RveDesc &d, void *work, double *out, cudaStream_t s)
{
    const int FG = 152 * FftGrid<R>::v;
    const int budget = (sizeof(R) == 8) ? 2048 : 4096;
    const int kc9 = pick_div(d.ny, (budget * 3 / 2) / (9 * d.nx));
    const int xt = d.nx / d.yxt, nzh = d.nzh;
    const size_t sz = std::max(smem_lines<R>(d.nz, 3 * d.zrows), smem_lines<R>(d.nz, 2 * d.zirows3));
    const size_t sy = smem_lines<R>(d.ny, d.yxt);
    const size_t sx = std::max(smem_lines<R>(d.nx, 9 * kc9), smem_lines<R>(d.nx, 3 * d.xkc3));
    const size_t si = smem_lines<R>(d.nz, 2 * d.zirows3);
    cudaFuncSetAttribute(k_disp_z_fwd<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sz);
    cudaFuncSetAttribute(k_disp_fft_y<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sy);
    cudaFuncSetAttribute(k_disp_fft_x<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sx);
    cudaFuncSetAttribute(k_disp_z_inv<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)si);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int uz6 = d.nx * (d.ny / d.zrows), uz3 = d.nx * (d.ny / d.zirows3);
    k_disp_z_fwd<R><<<grid_for(uz6, FG), 256, smem_lines<R>(d.nz, 3 * d.zrows), s>>>(d, work, 0, uz6);
    k_disp_z_fwd<R><<<grid_for(uz3, FG), 256, smem_lines<R>(d.nz, 2 * d.zirows3), s>>>(d, work, 1, uz3);
    const int uy9 = 9 * nzh * xt, uy3 = 3 * nzh * xt;
    k_disp_fft_y<R><<<grid_for(uy9, FG), 256, sy, s>>>(d, work, -1, uy9);
    const int ux9 = nzh * (d.ny / kc9), ux3 = nzh * (d.ny / d.xkc3);
    k_disp_fft_x<R><<<grid_for(ux9, FG), 256, smem_lines<R>(d.nx, 9 * kc9), s>>>(d, work, 9, -1, kc9, ux9);
    int blocks = (int)((d.nspec + 255) / 256);
    if (blocks > 152 * 8) blocks = 152 * 8;
    k_disp_spec<R><<<blocks, 256, 0, s>>>(d, work);
    k_disp_fft_x<R><<<grid_for(ux3, FG), 256, smem_lines<R>(d.nx, 3 * d.xkc3), s>>>(d, work, 3, +1, d.xkc3, ux3);
    k_disp_fft_y<R><<<grid_for(uy3, FG), 256, sy, s>>>(d, work, +1, uy3);
    k_disp_z_inv<R><<<grid_for(uz3, FG), 256, si, s>>>(d, work, out, uz3);
    return cudaGetLastError();
}

size_t disp_work_bytes(const RveDesc &d)
{
    return (size_t)9 * (size_t)d.nspec * (d.mixed ? sizeof(float2) : sizeof(double2));
}

cudaError_t launch_disp_fluct(const RveDesc &d, void *work, double *out, cudaStream_t s)
{
    return d.mixed ? disp_fluct_t<float>(d, work, out, s) : disp_fluct_t<double>(d, work, out, s);
}

// One block transforms nl lines of length pl.L with the line FFT of the
// spectrum passes: in and out are [nl][L] complex doubles, rounded to R on
// the way in.
template <typename R>
__global__ void __launch_bounds__(256) k_fft_probe(FftPlan1 pl, const typename Cx<R>::T *__restrict__ tw,
                                                   const double2 *__restrict__ in, double2 *__restrict__ out,
                                                   int nl, int sign)
{
    typedef typename Cx<R>::T C;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *a = reinterpret_cast<C *>(smem_raw);
    const int L = pl.L, ldl = nl | 1;
    C *b = a + L * ldl;
    for (int e = threadIdx.x; e < nl * L; e += blockDim.x) {
        const int l = e / L, i = e - l * L;
        a[i * ldl + l] = mkc<C>((R)in[e].x, (R)in[e].y);
    }
    __syncthreads();
    const C *res = fft_lines<R>(a, b, nl, ldl, pl, tw, sign);
    for (int e = threadIdx.x; e < nl * L; e += blockDim.x) {
        const int l = e / L, i = e - l * L;
        const C v = res[i * ldl + l];
        out[e] = make_double2(v.x, v.y);
    }
}

template <typename R>
static cudaError_t fft_probe_t(const FftPlan1 &pl, const void *tw, const double *in, double *out, int nl, int sign,
                               cudaStream_t s)
{
    const size_t smem = smem_lines<R>(pl.L, nl);
    cudaError_t e = cudaFuncSetAttribute((const void *)k_fft_probe<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    k_fft_probe<R><<<1, 256, smem, s>>>(pl, (const typename Cx<R>::T *)tw, (const double2 *)in, (double2 *)out, nl, sign);
    return cudaGetLastError();
}

cudaError_t launch_fft_probe(const FftPlan1 &pl, bool f32, const void *tw, const double *in, double *out, int nl,
                             int sign, cudaStream_t s)
{
    return f32 ? fft_probe_t<float>(pl, tw, in, out, nl, sign, s) : fft_probe_t<double>(pl, tw, in, out, nl, sign, s);
}

}  // namespace voce
