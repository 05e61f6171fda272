// pgm_fft_f64.cu -- the FFT passes of pgm_fft.cuh in FP64.
#include "pgm_fft_impl.cuh"

namespace pgmfft {

template bool supported<double>(int);
template cudaError_t prepare<double>(Pass, int);
template cudaError_t launch<double>(Pass, int, const Args<double> &, const Tiles &, int, int, int, cudaStream_t, bool);

}  // namespace pgmfft
