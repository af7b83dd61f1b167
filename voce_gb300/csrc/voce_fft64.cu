// The spectrum passes in double precision (voce_fft.cuh).
#include "voce_fft.cuh"

namespace voce {

VOCE_FFT_INSTANCE(double)

}  // namespace voce
