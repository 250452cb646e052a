// fdtd_half.cuh -- which half-step kernel serves a prefetch depth and launch
// mode.  The definitions are instantiated once per coefficient layout, in
// fdtd_half_f64.cu, fdtd_half_f32.cu and fdtd_half_table.cu, so that the three
// compile side by side and apart from the host code.
#pragma once
#include "fdtd_batch.cuh"
#include "fdtd_step.cuh"

namespace fdtd {

template <typename T, class C, bool EXACT>
void (*step_kernel(bool electric, int pf))(StepParams<T, C>);
template <typename T, class C, bool EXACT>
void (*batch_kernel(bool electric, int pf, bool persist))(const Instance<T, C>*, const BatchTile*, int, BatchCtl*,
                                                           int);
template <typename T, class C, bool EXACT>
void (*batch_group_kernel(bool electric, int pf))(const BatchGroup<T, C>);

#ifdef FDTD_HALF_DEFINE
// Step kernels for a prefetch depth: 1, 2 = planes prefetched in registers;
// 3, 4 = planes staged through shared memory (material-table problems only).
template <typename T, class C, bool EXACT>
void (*step_kernel(bool electric, int pf))(StepParams<T, C>) {
  if constexpr (C::kTable) {
    if (pf == 3) return electric ? k_step_e<T, C, EXACT, 3> : k_step_h<T, C, EXACT, 3>;
    if (pf == 4) return electric ? k_step_e<T, C, EXACT, 4> : k_step_h<T, C, EXACT, 4>;
    if (pf == 5) return electric ? k_step_e<T, C, EXACT, 5> : k_step_h<T, C, EXACT, 5>;
  }
  if (pf == 2) return electric ? k_step_e<T, C, EXACT, 2> : k_step_h<T, C, EXACT, 2>;
  return electric ? k_step_e<T, C, EXACT, 1> : k_step_h<T, C, EXACT, 1>;
}

// Batched H/E kernel for a prefetch depth (as step_kernel) and grid kind.
template <typename T, class C, bool EXACT>
void (*batch_kernel(bool electric, int pf, bool persist))(const Instance<T, C>*, const BatchTile*, int, BatchCtl*,
                                                           int) {
#define FDTD_BK(PF)                                                                                           \
  (electric ? (persist ? k_batch_half<T, C, EXACT, PF, true, true> : k_batch_half<T, C, EXACT, PF, true, false>) \
            : (persist ? k_batch_half<T, C, EXACT, PF, false, true> : k_batch_half<T, C, EXACT, PF, false, false>))
  if constexpr (C::kTable) {
    if (pf == 3) return FDTD_BK(3);
    if (pf == 4) return FDTD_BK(4);
  }
  if (pf == 2) return FDTD_BK(2);
  return FDTD_BK(1);
#undef FDTD_BK
}

// Grouped H/E kernel for a prefetch depth (as step_kernel).
template <typename T, class C, bool EXACT>
void (*batch_group_kernel(bool electric, int pf))(const BatchGroup<T, C>) {
#define FDTD_GK(PF) (electric ? k_batch_group<T, C, EXACT, PF, true> : k_batch_group<T, C, EXACT, PF, false>)
  if constexpr (C::kTable) {
    if (pf == 3) return FDTD_GK(3);
    if (pf == 4) return FDTD_GK(4);
  }
  if (pf == 2) return FDTD_GK(2);
  return FDTD_GK(1);
#undef FDTD_GK
}

#define FDTD_HALF(T, C, EXACT)                                                                                \
  template void (*step_kernel<T, C, EXACT>(bool, int))(StepParams<T, C>);                                     \
  template void (*batch_kernel<T, C, EXACT>(bool, int, bool))(const Instance<T, C>*, const BatchTile*, int,   \
                                                              BatchCtl*, int);                                \
  template void (*batch_group_kernel<T, C, EXACT>(bool, int))(const BatchGroup<T, C>);
#endif

}  // namespace fdtd
