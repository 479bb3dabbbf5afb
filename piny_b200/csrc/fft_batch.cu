// Mesh transforms of many MIXED boxes per launch (boxtab.cuh).
#include "fft.cuh"

namespace pinyb200 {

template <int N>
__global__ void __launch_bounds__(FftGeom<N>::PLANE_T, fft_blocks<float, N>(FftGeom<N>::PLANE_T, true))
    fft_plane_fwd_batch_kernel(const __grid_constant__ BoxTab<FftArgs> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (fft_plane_fwd_body<float, N>(t.arg[i], vb)));
}
template <int N>
__global__ void __launch_bounds__(FftGeom<N>::CONV_T, fft_blocks<float, N>(FftGeom<N>::CONV_T, true))
    fft_conv_batch_kernel(const __grid_constant__ BoxTab<FftArgs> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (fft_conv_body<float, N>(t.arg[i], vb)));
}
template <int N>
__global__ void __launch_bounds__(FftGeom<N>::PLANE_T, fft_blocks<float, N>(FftGeom<N>::PLANE_T, true))
    fft_plane_inv_batch_kernel(const __grid_constant__ BoxTab<FftArgs> t)
{
    PINYB200_BOX_LOOP(t, i, vb, (fft_plane_inv_body<float, N>(t.arg[i], vb)));
}

template <int N>
static cudaError_t launch_fft_batch_n(const std::vector<FftArgs> &bx, const std::vector<int> &P, int sm_count,
                                      cudaStream_t st, int stage)
{
    typedef FftGeom<N> G;
    constexpr size_t sp = fft_plane_smem<float, N>(), ss = fft_slab_smem<float, N>();
    BoxTabBuilder<FftArgs> tb;
    for (size_t i = 0; i < bx.size(); i++) tb.add(bx[i], P[i] * N, 1, (double)P[i]);
    if (stage == 0)
        return launch_tables(
            tb, (const void *)fft_plane_fwd_batch_kernel<N>, G::PLANE_T, sp, sm_count,
            [&](const BoxTab<FftArgs> &t, int g) { fft_plane_fwd_batch_kernel<N><<<g, G::PLANE_T, sp, st>>>(t); });
    if (stage == 1)
        return launch_tables(
            tb, (const void *)fft_conv_batch_kernel<N>, G::CONV_T, ss, sm_count,
            [&](const BoxTab<FftArgs> &t, int g) { fft_conv_batch_kernel<N><<<g, G::CONV_T, ss, st>>>(t); });
    return launch_tables(
        tb, (const void *)fft_plane_inv_batch_kernel<N>, G::PLANE_T, sp, sm_count,
        [&](const BoxTab<FftArgs> &t, int g) { fft_plane_inv_batch_kernel<N><<<g, G::PLANE_T, sp, st>>>(t); });
}

cudaError_t launch_fft_fixed_batch(int N, const std::vector<FftArgs> &bx, const std::vector<int> &P, int sm_count,
                                   cudaStream_t st, int stage)
{
    switch (N) {
#define PINYB200_FFT_CASE(n) \
    case n: return launch_fft_batch_n<n>(bx, P, sm_count, st, stage);
        PINYB200_FFT_EDGES(PINYB200_FFT_CASE)
#undef PINYB200_FFT_CASE
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pinyb200
