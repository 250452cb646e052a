// Half-step kernels: FP64 per-cell coefficients.
#define FDTD_HALF_DEFINE
#include "fdtd_half.cuh"

namespace fdtd {
FDTD_HALF(double, ArrayCoef<double>, true)
}  // namespace fdtd
