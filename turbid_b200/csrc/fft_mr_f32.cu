// The transforms of fft_mr_impl.cuh in single precision.
#include "fft_mr_impl.cuh"

namespace tg {
TG_MR_INSTANTIATE(float)
}
