// fdtd_fused.cu -- launches of the one-pass step (fdtd_fused.cuh), compiled
// apart from the half-step kernels.
#include "fdtd_fused.cuh"

namespace fdtd {

namespace {

// A launch; `early`: its blocks may start before the launch ahead of it has ended.
template <typename... P, typename... A>
cudaError_t launch(bool early, void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st,
                         A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

template <typename T, bool EXACT>
cudaError_t fused_step(const FusedParams<T>& p, bool early, cudaStream_t st) {
  const int smem = fused_smem_bytes<T>(), tiles = p.tk * p.tj * p.tx;
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_fused<T, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  return launch(early, k_fused<T, EXACT>, (unsigned)tiles, FusedShape<T>::kThreads, (size_t)smem, st, p);
}

template <typename T, bool EXACT>
cudaError_t fused_wall(const FusedParams<T>& p, cudaStream_t st) {
  const unsigned n = (unsigned)((p.ny + 1) * (p.nz + 1));
  k_fused_wall<T, EXACT><<<(n + 255) / 256, 256, 0, st>>>(p);
  return cudaGetLastError();
}

template <typename T>
cudaError_t fused_epilogue(const FusedParams<T>& p, const FarField& ff, const Probes& pr, unsigned blocks,
                           bool late, bool early, cudaStream_t st) {
  return launch(early, k_fused_epilogue<T>, blocks, 256, 0, st, p, ff, pr, (int)late);
}

template <typename T, class C>
cudaError_t fused_class_find(const StepParams<T, C>& s, int pitch, unsigned n, const ClassTable& tb, cudaStream_t st) {
  k_class_find<T, C><<<148 * 8, 256, 0, st>>>(s, pitch, n, tb);
  return cudaGetLastError();
}

template <typename T, class C>
cudaError_t fused_class_rows(const StepParams<T, C>& s, int pitch, unsigned n, const ClassTable& tb,
                             const ClassLayout& layout, T* tab, unsigned short* cls, cudaStream_t st) {
  for (int fill = 1; fill >= 0; fill--) k_class_rows<T, C><<<148 * 8, 256, 0, st>>>(s, pitch, n, tb, layout, tab, cls, fill);
  return cudaGetLastError();
}

template <typename T>
cudaError_t fused_repack(T* pad, long long si, long long sj, T* dense, int ni, int nj, int nk, int to_pad,
                         cudaStream_t st) {
  const long long n = (long long)ni * nj * nk;
  if (n <= 0) return cudaSuccess;
  const unsigned blocks = (unsigned)(n / 256 + 1 < 148 * 16 ? n / 256 + 1 : 148 * 16);
  k_repack<T><<<blocks, 256, 0, st>>>(pad, si, sj, dense, ni, nj, nk, to_pad);
  return cudaGetLastError();
}

#define FDTD_FUSED(T, EXACT)                                                                                       \
  template cudaError_t fused_step<T, EXACT>(const FusedParams<T>&, bool, cudaStream_t); \
  template cudaError_t fused_wall<T, EXACT>(const FusedParams<T>&, cudaStream_t);
FDTD_FUSED(double, true)
FDTD_FUSED(float, true)
FDTD_FUSED(float, false)
#define FDTD_FUSED_T(T)                                                                                            \
  template cudaError_t fused_epilogue<T>(const FusedParams<T>&, const FarField&, const Probes&, unsigned, bool,    \
                                         bool, cudaStream_t);                                                            \
  template cudaError_t fused_repack<T>(T*, long long, long long, T*, int, int, int, int, cudaStream_t);
FDTD_FUSED_T(double)
FDTD_FUSED_T(float)
#define FDTD_FUSED_C(T, C)                                                                                         \
  template cudaError_t fused_class_find<T, C>(const StepParams<T, C>&, int, unsigned, const ClassTable&,           \
                                              cudaStream_t);                                                       \
  template cudaError_t fused_class_rows<T, C>(const StepParams<T, C>&, int, unsigned, const ClassTable&,           \
                                              const ClassLayout&, T*, unsigned short*, cudaStream_t);
FDTD_FUSED_C(double, ArrayCoef<double>)
FDTD_FUSED_C(float, ArrayCoef<float>)
FDTD_FUSED_C(float, TableCoef)

}  // namespace fdtd
