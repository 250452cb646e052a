// Half-step kernels: FP32 per-cell coefficients.
#define FDTD_HALF_DEFINE
#include "fdtd_half.cuh"

namespace fdtd {
FDTD_HALF(float, ArrayCoef<float>, true)
}  // namespace fdtd
