// pgm_fft_f32.cu -- the FFT passes of pgm_fft.cuh in FP32 (mixed precision).
#include "pgm_fft_impl.cuh"

namespace pgmfft {

size_t plane_smem(int N, size_t real_size) {
  size_t b = 0;
  with_length(N, [&](auto Lc) {
    constexpr int L = decltype(Lc)::value;
    if constexpr (L <= PLANE_MAX) b = real_size == 4 ? plane_bytes<float, L>() : plane_bytes<double, L>();
  });
  return b;
}

template bool supported<float>(int);
template cudaError_t prepare<float>(Pass, int);
template cudaError_t launch<float>(Pass, int, const Args<float> &, const Tiles &, int, int, int, cudaStream_t, bool);

}  // namespace pgmfft
