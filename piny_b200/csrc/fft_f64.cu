// Mesh transforms of one box in FP64.
#include "fft_one.cuh"

namespace pinyb200 {
template cudaError_t launch_fft_fixed<double>(pinyb200_ctx *c, int N, int P, const FftArgs &f);
}
