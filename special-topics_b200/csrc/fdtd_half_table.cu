// Half-step kernels: FP32 material tables.
#define FDTD_HALF_DEFINE
#include "fdtd_half.cuh"

namespace fdtd {
FDTD_HALF(float, TableCoef, false)
}  // namespace fdtd
