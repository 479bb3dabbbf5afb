// One box's mesh transforms for precision R: included by one source file per
// precision, which instantiates launch_fft_fixed.
#pragma once
#include "fft.cuh"

namespace pinyb200 {

// Device time, B200, warm L2, against one complex line per real row with
// radix 8 and 4 passes (powers of two) or a direct DFT (other lengths):
//   64^3, 32 beads, FP32: forward planes 31.8 -> 27.0 us, convolution 51.9 ->
//   33.8, inverse planes 34.2 -> 24.3 (205 MB of grid and spectrum);
//   36^3, 8 beads, FP32: 92.0 -> 4.7, 38.1 -> 6.4, 89.8 -> 4.8 us;
//   80^3, 4 beads, FP32: the three together 3121 -> about 50 us.
template <typename R, int N>
static cudaError_t launch_fft_n(pinyb200_ctx *c, int P, const FftArgs &f)
{
    typedef FftGeom<N> G;
    constexpr size_t sp = fft_plane_smem<R, N>(), ss = fft_slab_smem<R, N>();
    cudaError_t err = cudaSuccess;
    if (sp > 48 * 1024) {
        err = smem_optin((const void *)fft_plane_fwd_kernel<R, N>, (int)sp);
        if (err == cudaSuccess) err = smem_optin((const void *)fft_plane_inv_kernel<R, N>, (int)sp);
        if (err != cudaSuccess) return err;
    }
    if (ss > 47 * 1024) {
        err = smem_optin((const void *)fft_conv_kernel<R, N>, (int)ss);
        if (err != cudaSuccess) return err;
    }
    fft_plane_fwd_kernel<R, N><<<P * N, G::PLANE_T, sp, c->stream>>>(f);
    if ((err = kt_mark(c, "pme_plane_fwd")) != cudaSuccess) return err;
    fft_conv_kernel<R, N><<<P * N, G::CONV_T, ss, c->stream>>>(f);
    if ((err = kt_mark(c, "pme_conv_c")) != cudaSuccess) return err;
    fft_plane_inv_kernel<R, N><<<P * N, G::PLANE_T, sp, c->stream>>>(f);
    if ((err = kt_mark(c, "pme_plane_inv")) != cudaSuccess) return err;
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_fft_fixed(pinyb200_ctx *c, int N, int P, const FftArgs &f)
{
    switch (N) {
#define PINYB200_FFT_CASE(n) \
    case n:                                                          \
        if constexpr (sizeof(R) == 4 || n <= PINYB200_FFT_MAX_FP64)  \
            return launch_fft_n<R, n>(c, P, f);                      \
        else                                                         \
            return cudaErrorInvalidValue;
        PINYB200_FFT_EDGES(PINYB200_FFT_CASE)
#undef PINYB200_FFT_CASE
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pinyb200
