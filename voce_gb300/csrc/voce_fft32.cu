// The spectrum passes in single precision (voce_fft.cuh).
#include "voce_fft.cuh"

namespace voce {

VOCE_FFT_INSTANCE(float)

}  // namespace voce
