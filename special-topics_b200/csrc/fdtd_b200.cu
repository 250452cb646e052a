// fdtd_b200.cu -- host side of the C ABI declared in include/fdtd_b200.h:
// problem handles, uploads with validation, the per-step launch sequence
// (captured into a CUDA graph per batch of steps), readbacks and the legacy
// global-context entry points of js_fdtd/src/backends/cuda/native/fdtd_cuda.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <initializer_list>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/fdtd_b200.h"
#include "fdtd_common.cuh"
#include "fdtd_material.cuh"
#include "fdtd_step.cuh"
#include "fdtd_batch.cuh"
#include "fdtd_ffpost.cuh"
#include "fdtd_fused.cuh"
#include "fdtd_half.cuh"
#include "fdtd_internal.h"
#include "run_plan.h"

#include <map>
#include <utility>

using namespace fdtd;

static thread_local char g_err[512] = "no error";

static int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

namespace {
cudaError_t dev_malloc(int device, void** p, size_t bytes);
}

cudaError_t fdtd_internal_malloc(int device, void** p, size_t bytes) { return dev_malloc(device, p, bytes); }

int fdtd_internal_fail(int code, const char* msg) { return fail(code, "%s", msg); }

#define CK(call)                                                                              \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess) return fail(FDTD_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

namespace {

struct HostFace {
  bool present = false;
  int nc = 0, m_start = 0, e_start = 0;
  void* prof[4] = {};   // b_e a_e b_m a_m (field type)
  float* inv_k[2] = {};  // 1/kappa_e, 1/kappa_m (table problems)
  void* block = nullptr;  // the allocation that holds the face's arrays
  void* psi[4] = {};
  void* cpsi[4] = {};
  long long n[4] = {};
};

struct HostSource {
  SourceBox box;
  int count;
  void* cs;
  void* wave;
};

struct HostVProbe {
  int comp, count;
  int* idx;
  double csvf;
  std::vector<int> cells;   // idx on the host
};

struct HostIProbe {
  int count;
  int* comp;
  int* idx;
  double* w;
  std::vector<int> comps, cells;  // comp and idx on the host
};

}  // namespace

// CUDA graphs of whole runs (run_plan.h).  Every graph a run needs is captured
// before the run's first launch, so no capture falls inside a timed region.
struct RunGraphs {
  GraphCache<cudaGraphExec_t> cache;
  void clear() {
    for (auto& e : cache.g) cudaGraphExecDestroy(e.exec);
    cache.g.clear();
    rev++;
  }
  long long rev = 0;  // times cleared: what else captured the same set-up is stale then
};

// The padded state of the one-pass step (fdtd_fused.cuh): allocated at the
// first run that can use it, dropped when the set-up changes.
struct FusedState {
  bool tried = false, ok = false;  // built (or found unusable) for the present set-up
  int no_room_at = -1;             // unusable for want of memory alone, found at this step
  bool valid = false;              // holds the current fields and Psi, in copy `cur`
  int cur = 0;
  int ts_at = -1;                  // step index in d_ts[cur]
  void* f[2][6] = {};
  void* ph[3][2][2] = {};          // H Psi by axis, copy, slot
  void* pe[3][2] = {};
  void* prof[2][3][2] = {};
  unsigned short* cls = nullptr;
  void* tab = nullptr;             // class table
  ClassLayout layout = {};         // of the table's rows, and the z slabs
  int* d_ts = nullptr;
  int* v_idx[kMaxProbes] = {};
  int* i_idx[kMaxProbes] = {};
  std::vector<void*> owned;
};

struct fdtd_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int prec = FDTD_PREC_F64;
  size_t esz = 8;  // bytes per field value
  int nx = 0, ny = 0, nz = 0, nsteps = 0;
  double dx = 0, dy = 0, dz = 0, dt = 0;
  int ts = 0;  // completed steps
  long long ncomp[6] = {};  // Hx Hy Hz Ex Ey Ez element counts
  void* fields = nullptr;   // contiguous Hx..Ez (+ slack)
  void* coef[18] = {};
  bool coef_set[18] = {};
  bool coef_device = false;     // FP64 coefficients built by fdtd_ctx_build_material
  bool kappa_done[6] = {};      // face whose CPML band of them was divided by kappa on the device
  // material-table problem
  unsigned char* ids[6] = {};
  bool ids_set[6] = {};
  std::vector<float> table[6];
  std::vector<double> rows64[6];  // the same rows in FP64 (rows x 3), for overrides and readback
  float* d_tab = nullptr;      // [6][kTableRows] float4 rows (self, curl1, curl2, 0), field order
  float* d_invk[6] = {};       // 1/kappa per axis position: E x y z, H x y z
  bool table_dirty = true;
  TableCoef tcoef{};
  HostFace face[6];
  std::vector<HostSource> src;
  std::vector<HostVProbe> vprobe;
  std::vector<HostIProbe> iprobe;
  double* V = nullptr;  // traces
  double* I = nullptr;
  int nv_alloc = -1, ni_alloc = -1;
  // far field
  int nFreq = 0;
  int li = 0, lj = 0, lk = 0, ui = 0, uj = 0, uk = 0;
  double* ph = nullptr;
  double* acc = nullptr;
  std::vector<double> ffreq;  // far-field frequencies (Hz)
  int acc_kahan = 0;          // FP32 problems: compensated FP32 accumulator pairs instead of FP64
  int dft_block = 0;          // FP32 problems: steps per time block of the surface DFT (0: every step)
  int x_wall = 0;             // 1: Ey, Ez at i = nx stay zero (see fdtd_ctx_set_x_wall)
  bool half_steps = false;    // see fdtd_ctx_set_step_path
  float* dft_samples = nullptr;
  int* d_dft_done = nullptr;
  long long ffsz[3] = {};
  long long ffoff[24] = {};
  void* ex0b = nullptr;
  int* d_ts = nullptr;
  int* d_status = nullptr;
  // launch shape of the step kernels: x planes per thread, thread rows per block
  int ichunk = 1, block_rows = 8, prefetch = 1;
  int block_w = 32;   // threads of a block along k (32: a warp is one row; 16: a warp spans two rows)
  FusedState fs;
  bool dense_valid = true;  // `fields` and the faces' Psi hold the current state
  // graph cache
  RunGraphs graphs;
  bool dirty = true;
  std::vector<void*> owned;  // every device allocation
  // Running digest of everything the handle was set up with: shape, spacing,
  // dt, step count, precision and the arguments of every upload call in call
  // order.  A saved state carries it and loads only where it matches.
  unsigned long long setup_digest = 0x6a09e667f3bcc908ULL;
  std::recursive_mutex mu;  // held by every call that touches the set-up, the graphs or `fs`, see reclaim_padded
  std::atomic<bool> padded{false};  // `fs` holds memory
  std::atomic<bool> wanted{false};  // another thread waits for that memory
};

namespace {

int to_dense(fdtd_ctx* c);
int fused_drop(fdtd_ctx* c);
using Using = std::lock_guard<std::recursive_mutex>;

// The handles of the process, so that one short of memory can take back what
// others hold for speed alone.
struct Handles {
  std::mutex mu;
  std::vector<fdtd_ctx*> all;
};
Handles& handles() {
  static Handles* h = new Handles;
  return *h;
}

// A handle on the device gives up its padded state (a later run builds it again,
// or takes the half-step path): without it, what fits beside the dense arrays of
// the handles would not.  A handle in another thread's call is asked to, and
// waited for: it does at its next run, or is idle by then.  A handle in a call of
// this thread gives up its own; no call allocates through here between making its
// padded state current and launching on it.  False: none had any.
bool reclaim_padded(int device) {
  constexpr int kWaitMs = 60000;
  for (int waited = 0;; waited++) {
    bool busy = false;
    {
      std::lock_guard<std::mutex> g(handles().mu);
      for (fdtd_ctx* o : handles().all) {
        if (o->device != device || !o->padded) continue;
        std::unique_lock<std::recursive_mutex> use(o->mu, std::try_to_lock);
        if (!use.owns_lock())
          o->wanted = busy = true;
        else if (fused_drop(o) == FDTD_OK)
          return true;
      }
    }
    if (!busy) return waited > 0;  // given up meanwhile
    if (waited >= kWaitMs) return false;
    std::this_thread::sleep_for(std::chrono::milliseconds(1));
  }
}

// cudaMalloc on the current device, `device`, that takes back padded states while
// memory is short.  Every allocation of the library but the padded states' own.
cudaError_t dev_malloc(int device, void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  for (int tries = 0; e == cudaErrorMemoryAllocation && tries < 1000; tries++) {
    cudaGetLastError();
    if (!reclaim_padded(device)) break;
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess) *p = nullptr;
  return e;
}
template <typename V>
cudaError_t dev_malloc(const fdtd_ctx* c, V** p, size_t bytes) {
  return dev_malloc(c->device, (void**)p, bytes);
}

int dalloc(fdtd_ctx* c, void** p, size_t bytes) {
  if (bytes == 0) bytes = 16;
  cudaError_t e = dev_malloc(c, p, bytes);
  if (e != cudaSuccess) return fail(FDTD_ERR_OOM, "cudaMalloc(%zu bytes): %s", bytes, cudaGetErrorString(e));
  c->owned.push_back(*p);
  // Zero on the handle's stream and wait: later uploads may use either stream,
  // and the zeroing must not land after them.
  e = cudaMemsetAsync(*p, 0, bytes, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return fail(FDTD_ERR_CUDA, "zeroing a new buffer: %s", cudaGetErrorString(e));
  return FDTD_OK;
}

// Arrays that live together, in one allocation: what bounds the set-up of a small
// problem is not bytes but the number of allocations, zeroings and releases.  A
// 64^3 FP64 problem with one for each of its some 90 arrays took 7.1 ms to create,
// 5.0 for its CPML faces and 8.6 to free; now 0.9, 4.3 and 3.2 ms.
struct Arena {
  struct Part {
    void** p;
    size_t at;
  };
  std::vector<Part> parts;
  size_t size = 0;
  template <typename V>
  void add(V** p, size_t bytes) {
    parts.push_back({(void**)p, size});
    size += (bytes + 255) / 256 * 256;
  }
  void place(void* base) const {
    for (const Part& q : parts) *q.p = (char*)base + q.at;
  }
};

void dfree(fdtd_ctx* c, void* p) {
  if (!p) return;
  auto it = std::find(c->owned.begin(), c->owned.end(), p);
  if (it != c->owned.end()) c->owned.erase(it);
  cudaFree(p);
}

// Copy on the handle's stream and wait.  Every set-up copy goes through here so
// that it is ordered with the zeroing in dalloc and with the kernels, which all
// run on that (non-blocking) stream.
cudaError_t xfer(fdtd_ctx* c, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, kind, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e;
}

// Host FP64 array -> device array of the problem's field type.
int upload_real(fdtd_ctx* c, void* dst, const double* src, long long n) {
  if (n <= 0) return FDTD_OK;
  if (c->esz == 8) {
    CK(cudaMemcpyAsync(dst, src, n * 8, cudaMemcpyHostToDevice, c->stream));
  } else {
    std::vector<float> tmp(n);
    for (long long q = 0; q < n; q++) tmp[q] = (float)src[q];
    CK(cudaMemcpyAsync(dst, tmp.data(), n * 4, cudaMemcpyHostToDevice, c->stream));
  }
  CK(cudaStreamSynchronize(c->stream));
  return FDTD_OK;
}

int read_real(fdtd_ctx* c, const void* srcdev, double* dst, long long n) {
  if (n <= 0) return FDTD_OK;
  if (c->esz == 8) {
    CK(cudaMemcpyAsync(dst, srcdev, n * 8, cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
  } else {
    std::vector<float> tmp(n);
    CK(cudaMemcpyAsync(tmp.data(), srcdev, n * 4, cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    for (long long q = 0; q < n; q++) dst[q] = tmp[q];
  }
  return FDTD_OK;
}

// Coefficient id -> (component, count) in cudaBackend.js:53-60 order.
long long coef_count(const fdtd_ctx* c, int which) {
  static const int comp_of[18] = {3, 3, 3, 4, 4, 4, 5, 5, 5, 0, 0, 0, 1, 1, 1, 2, 2, 2};
  return c->ncomp[comp_of[which]];
}

void* field_ptr(const fdtd_ctx* c, int which) {
  char* base = (char*)c->fields;
  long long off = 0;
  for (int q = 0; q < which; q++) off += c->ncomp[q];
  return base + off * c->esz;
}

// Expected Psi slot sizes (cpml.js:147-448) for face f with nc cells.
void psi_sizes(const fdtd_ctx* c, int f, int nc, long long out[4]) {
  const long long nx = c->nx, ny = c->ny, nz = c->nz, X = nx + 1, Y = ny + 1, Z = nz + 1;
  if (f / 2 == 0) {
    out[0] = nc * Y * nz; out[1] = nc * ny * Z; out[2] = nc * ny * Z; out[3] = nc * Y * nz;
  } else if (f / 2 == 1) {
    out[0] = X * nc * nz; out[1] = nx * nc * Z; out[2] = X * nc * nz; out[3] = nx * nc * Z;
  } else {
    out[0] = X * ny * nc; out[1] = nx * Y * nc; out[2] = nx * Y * nc; out[3] = X * ny * nc;
  }
}

void invalidate(fdtd_ctx* c) {
  c->dirty = true;
  c->table_dirty = true;
  c->graphs.clear();
}

template <typename T>
Face<T> dev_face(const HostFace& h) {
  Face<T> f{};
  if (!h.present) return f;
  f.nc = h.nc;
  f.m_start = h.m_start;
  f.e_start = h.e_start;
  f.b_e = (const T*)h.prof[0];
  f.a_e = (const T*)h.prof[1];
  f.b_m = (const T*)h.prof[2];
  f.a_m = (const T*)h.prof[3];
  f.inv_ke = h.inv_k[0];
  f.inv_km = h.inv_k[1];
  for (int s = 0; s < 4; s++) {
    f.psi[s] = (T*)h.psi[s];
    f.cpsi[s] = (const T*)h.cpsi[s];
  }
  return f;
}

template <typename T>
Fields<T> dev_fields(const fdtd_ctx* c) {
  Fields<T> f;
  f.Hx = (T*)field_ptr(c, 0);
  f.Hy = (T*)field_ptr(c, 1);
  f.Hz = (T*)field_ptr(c, 2);
  f.Ex = (T*)field_ptr(c, 3);
  f.Ey = (T*)field_ptr(c, 4);
  f.Ez = (T*)field_ptr(c, 5);
  return f;
}

template <typename T>
Sources<T> dev_sources(const fdtd_ctx* c) {
  Sources<T> s{};
  s.n = (int)c->src.size();
  for (int q = 0; q < s.n; q++) {
    s.box[q] = c->src[q].box;
    s.cs[q] = (const T*)c->src[q].cs;
    s.wave[q] = (const T*)c->src[q].wave;
  }
  return s;
}

Probes dev_probes(const fdtd_ctx* c) {
  Probes p{};
  p.n_v = (int)c->vprobe.size();
  p.n_i = (int)c->iprobe.size();
  for (int q = 0; q < p.n_v; q++) {
    p.v_comp[q] = c->vprobe[q].comp;
    p.v_count[q] = c->vprobe[q].count;
    p.v_idx[q] = c->vprobe[q].idx;
    p.v_csvf[q] = c->vprobe[q].csvf;
  }
  for (int q = 0; q < p.n_i; q++) {
    p.i_count[q] = c->iprobe[q].count;
    p.i_comp[q] = c->iprobe[q].comp;
    p.i_idx[q] = c->iprobe[q].idx;
    p.i_w[q] = c->iprobe[q].w;
  }
  p.V = c->V;
  p.I = c->I;
  p.nsteps = c->nsteps;
  p.status = c->d_status;
  return p;
}

FarField dev_ff(const fdtd_ctx* c) {
  FarField ff{};
  ff.nFreq = c->nFreq;
  if (c->nFreq == 0) return ff;
  ff.LI = c->li - 1; ff.LJ = c->lj - 1; ff.LK = c->lk - 1;
  ff.UI = c->ui - 1; ff.UJ = c->uj - 1; ff.UK = c->uk - 1;
  ff.ni = c->ui - c->li; ff.nj = c->uj - c->lj; ff.nk = c->uk - c->lk;
  ff.ph = c->ph;
  ff.acc = c->acc;
  for (int a = 0; a < 24; a++) ff.off[a] = c->ffoff[a];
  for (int a = 0; a < 3; a++) ff.sz[a] = c->ffsz[a];
  ff.kahan = c->acc_kahan;
  ff.block = c->dft_block;
  ff.samples = c->dft_samples;
  ff.done = c->d_dft_done;
  return ff;
}

// Trace buffers follow the probe counts.
int ensure_traces(fdtd_ctx* c) {
  const int nv = (int)c->vprobe.size(), ni = (int)c->iprobe.size();
  if (nv != c->nv_alloc) {
    dfree(c, c->V);
    c->V = nullptr;
    int rc = dalloc(c, (void**)&c->V, sizeof(double) * std::max(nv, 1) * (size_t)c->nsteps);
    if (rc) return rc;
    c->nv_alloc = nv;
  }
  if (ni != c->ni_alloc) {
    dfree(c, c->I);
    c->I = nullptr;
    int rc = dalloc(c, (void**)&c->I, sizeof(double) * std::max(ni, 1) * (size_t)c->nsteps);
    if (rc) return rc;
    c->ni_alloc = ni;
  }
  return FDTD_OK;
}

int check_ready(fdtd_ctx* c) {
  if (c->prec == FDTD_PREC_F32_TABLE) {
    for (int q = 0; q < 6; q++)
      if (!c->ids_set[q]) return fail(FDTD_ERR_STATE, "material ids of component %d not uploaded", q);
  } else {
    for (int q = 0; q < 18; q++)
      if (!c->coef_set[q]) return fail(FDTD_ERR_STATE, "coefficient array %d not uploaded", q);
  }
  return FDTD_OK;
}

// True when, on every axis, the two faces' H bands are disjoint and so are
// their E bands: a position then lies in at most one band per axis.
int bands_disjoint(const fdtd_ctx* c) {
  for (int a = 0; a < 3; a++) {
    const HostFace& n = c->face[2 * a];
    const HostFace& q = c->face[2 * a + 1];
    if (!n.present || !q.present || n.nc == 0 || q.nc == 0) continue;
    const bool h = n.m_start + n.nc <= q.m_start || q.m_start + q.nc <= n.m_start;
    const bool e = n.e_start + n.nc <= q.e_start || q.e_start + q.nc <= n.e_start;
    if (!h || !e) return 0;
  }
  return 1;
}

// Kernel parameters shared by both coefficient layouts.
template <typename T, class C>
StepParams<T, C> step_params(const fdtd_ctx* c, const C& coef) {
  StepParams<T, C> p{};
  p.g = GridDims{c->nx, c->ny, c->nz};
  p.f = dev_fields<T>(c);
  p.coef = coef;
  for (int q = 0; q < 6; q++) p.face[q] = dev_face<T>(c->face[q]);
  p.ex0b = (T*)c->ex0b;
  p.ts = c->d_ts;
  p.src = dev_sources<T>(c);
  p.dcell[0] = (T)c->dx;
  p.dcell[1] = (T)c->dy;
  p.dcell[2] = (T)c->dz;
  p.ichunk = c->ichunk;
  p.bands_disjoint = bands_disjoint(c);
  p.dft_block = c->dft_block;
  p.dft_done = c->d_dft_done;
  p.x_wall = c->x_wall;
  p.fault = c->d_status;
  return p;
}

// Dynamic shared memory of a step launch; raises the kernel's limit when the
// stages need more than the default 48 KB.
template <class K>
int stage_smem(K kernel, int pf, int threads, size_t* bytes) {
  *bytes = pf == 5 ? (size_t)bulk_smem_bytes(threads) : pf >= 3 ? (size_t)stage_smem_bytes(pf, threads) : 0;
  if (*bytes > 48 * 1024)
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*bytes));
  return FDTD_OK;
}

// Per-kernel timing of a profiled run: events around each launch.
struct KernelTimer {
  cudaEvent_t ev[5];
  double ms[4] = {0, 0, 0, 0};
};

// A launch shape is whole warps of at most 256 threads (the step kernels'
// launch bounds).
int check_block(int w, int rows) {
  const int t = w * rows;
  if ((w != 16 && w != 32) || t > 256 || t % 32 != 0)
    return fail(FDTD_ERR_BADARG, "block of %d x %d threads: need width 16 or 32, whole warps, at most 256", w, rows);
  return FDTD_OK;
}

// The launch shape the caller set, whichever path the run takes.
int check_shape(const fdtd_ctx* c) {
  int rc = check_block(c->block_w, c->block_rows);
  if (!rc && c->prefetch == 5 && c->block_w != 32)
    return fail(FDTD_ERR_BADARG, "prefetch mode 5 (bulk-copied stages) needs 32-wide blocks, got %d", c->block_w);
  return rc;
}

// Enqueue `count` steps on stream `st` (default: the handle's stream; with
// `tm`, one step at a time, timing each kernel).
template <typename T, class C, bool EXACT>
int enqueue_steps(fdtd_ctx* c, const C& coef, int count, KernelTimer* tm = nullptr, cudaStream_t st = nullptr) {
  if (!st) st = c->stream;
  StepParams<T, C> p = step_params<T, C>(c, coef);
  Probes pr = dev_probes(c);
  FarField ff = dev_ff(c);
  // a thread per (j, k) column walks `ichunk` x planes
  int rc0 = check_shape(c);
  if (rc0) return rc0;
  const dim3 blk(c->block_w, c->block_rows);
  const dim3 grd((c->nz + c->block_w) / c->block_w, (c->ny + c->block_rows) / c->block_rows,
                 (c->nx + 1 + c->ichunk - 1) / c->ichunk);
  const long long plane = (long long)c->ny * (c->nz + 1);
  const unsigned mid_blocks = (unsigned)((plane + pr.n_i + 255) / 256);
  const long long nff = (c->nFreq > 0) ? c->ffsz[0] + c->ffsz[1] + c->ffsz[2] : 0;
  const unsigned epi_blocks = (unsigned)((nff + pr.n_v + 255) / 256);
  auto kh = step_kernel<T, C, EXACT>(false, c->prefetch);
  auto ke = step_kernel<T, C, EXACT>(true, c->prefetch);
  size_t smem = 0;
  int rc = stage_smem(kh, c->prefetch, c->block_w * c->block_rows, &smem);
  if (!rc) rc = stage_smem(ke, c->prefetch, c->block_w * c->block_rows, &smem);
  if (rc) return rc;
  for (int s = 0; s < count; s++) {
    if (tm) CK(cudaEventRecord(tm->ev[0], st));
    kh<<<grd, blk, smem, st>>>(p);
    if (tm) CK(cudaEventRecord(tm->ev[1], st));
    k_step_mid<T, C, EXACT><<<mid_blocks, 256, 0, st>>>(p, pr);
    if (tm) CK(cudaEventRecord(tm->ev[2], st));
    ke<<<grd, blk, smem, st>>>(p);
    if (tm) CK(cudaEventRecord(tm->ev[3], st));
    if (epi_blocks) k_epilogue<T><<<epi_blocks, 256, 0, st>>>(p.f, p.g, ff, pr, c->d_ts);
    if (c->dft_block > 0) CK(dft_flush(ff, c->d_ts, -1, st));
    if (tm) {
      CK(cudaEventRecord(tm->ev[4], st));
      CK(cudaEventSynchronize(tm->ev[4]));
      for (int q = 0; q < 4; q++) {
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, tm->ev[q], tm->ev[q + 1]));
        tm->ms[q] += ms;
      }
    }
  }
  CK(cudaGetLastError());
  return FDTD_OK;
}

template <typename T>
ArrayCoef<T> array_coef(const fdtd_ctx* c) {
  ArrayCoef<T> a{};
  for (int comp = 0; comp < 6; comp++)
    for (int w = 0; w < 3; w++) {
      const int id = comp < 3 ? 9 + 3 * comp + w : 3 * (comp - 3) + w;
      a.c[comp][w] = (const T*)c->coef[id];
    }
  return a;
}

// Material tables and 1/kappa profiles to the device (once per change; never
// called while the stream is being captured).
int prepare_table(fdtd_ctx* c, TableCoef* out) {
  const int n_axis[3] = {c->nx, c->ny, c->nz};
  if (!c->d_tab) {
    int rc = dalloc(c, (void**)&c->d_tab, 6 * kTableRows * 4 * sizeof(float));
    if (rc) return rc;
    for (int q = 0; q < 6; q++) {
      rc = dalloc(c, (void**)&c->d_invk[q], (n_axis[q % 3] + 1) * sizeof(float));
      if (rc) return rc;
    }
  }
  if (c->table_dirty) {
    std::vector<float> tab(6 * kTableRows * 4, 0.f);
    for (int f = 0; f < 6; f++) {
      const std::vector<float>& t = c->table[(f + 3) % 6];
      for (int r = 0; r < kTableRows; r++)
        for (int w = 0; w < 3; w++) tab[(f * kTableRows + r) * 4 + w] = t[3 * r + w];
    }
    CK(xfer(c, c->d_tab, tab.data(), tab.size() * sizeof(float), cudaMemcpyHostToDevice));
    for (int a = 0; a < 3; a++) {
      std::vector<float> ie(n_axis[a] + 1, 1.f), im(n_axis[a] + 1, 1.f);
      for (int side = 0; side < 2; side++) {
        const HostFace& h = c->face[2 * a + side];
        if (!h.present) continue;
        std::vector<float> ke(h.nc), km(h.nc);
        CK(xfer(c, ke.data(), h.inv_k[0], h.nc * sizeof(float), cudaMemcpyDeviceToHost));
        CK(xfer(c, km.data(), h.inv_k[1], h.nc * sizeof(float), cudaMemcpyDeviceToHost));
        for (int q = 0; q < h.nc; q++) {
          ie[h.e_start + q] = ke[q];
          im[h.m_start + q] = km[q];
        }
      }
      CK(xfer(c, c->d_invk[a], ie.data(), ie.size() * sizeof(float), cudaMemcpyHostToDevice));
      CK(xfer(c, c->d_invk[3 + a], im.data(), im.size() * sizeof(float), cudaMemcpyHostToDevice));
    }
  }
  TableCoef t{};
  for (int f = 0; f < 6; f++) t.ids[f] = c->ids[(f + 3) % 6];
  t.tab = (const float4*)c->d_tab;
  for (int q = 0; q < 6; q++) t.inv[q] = c->d_invk[q];
  *out = t;
  c->table_dirty = false;
  return FDTD_OK;
}

// ---------------------------------------------------------------------------
// One-pass step: state, set-up and launches (fdtd_fused.cuh).
// ---------------------------------------------------------------------------
int fused_pitch(const fdtd_ctx* c) {
  // whole 32-byte sectors per row; eight values, so that a row of 16-bit classes
  // is whole 16-byte units
  const int a = 8;
  return (c->nz + 1 + a - 1) / a * a;
}
long long fused_plane(const fdtd_ctx* c) { return (long long)(c->ny + 1) * fused_pitch(c); }

// Memory for the padded state: no other handle's is taken for it.
int fused_malloc(fdtd_ctx* c, void** p, size_t bytes) {
  if (cudaMalloc(p, bytes) == cudaSuccess) return FDTD_OK;
  cudaGetLastError();  // no room: the caller takes the half-step path
  *p = nullptr;
  c->fs.no_room_at = c->ts;
  return FDTD_ERR_OOM;
}

// One zeroed allocation of the padded state.
int fused_alloc(fdtd_ctx* c, void** p, size_t bytes) {
  if (int rc = fused_malloc(c, p, bytes)) return rc;
  c->fs.owned.push_back(*p);
  c->padded = true;
  CK(cudaMemsetAsync(*p, 0, bytes, c->stream));
  return FDTD_OK;
}

// Field q between its dense array and copy `cur`.
template <typename T>
int fused_copy_field(fdtd_ctx* c, int q, int to_pad) {
  const int nx = c->nx, ny = c->ny, nz = c->nz;
  const int ni = (q == 1 || q == 2 || q == 3) ? nx : nx + 1, nj = (q == 0 || q == 2 || q == 4) ? ny : ny + 1,
            nk = (q == 0 || q == 1 || q == 5) ? nz : nz + 1;
  CK(fused_repack<T>((T*)c->fs.f[c->fs.cur][q], fused_plane(c), fused_pitch(c), (T*)field_ptr(c, q), ni, nj, nk, to_pad,
                     c->stream));
  return FDTD_OK;
}

// Psi slot s of face f.
template <typename T>
int fused_copy_psi(fdtd_ctx* c, int f, int s, int to_pad) {
  FusedState& fs = c->fs;
  const HostFace& h = c->face[f];
  const int nx = c->nx, ny = c->ny, nz = c->nz, P = fused_pitch(c);
  const long long S = fused_plane(c);
  const int ax = f / 2, el = s >= 2, nb = fs.layout.row.n[ax];
  const int c0 = ax == 2 ? (f % 2 ? fs.layout.zw[el][0] : 0) + (el ? h.e_start : h.m_start) - fs.layout.z0[el][f % 2]
                         : (f % 2 ? c->face[2 * ax].nc : 0);
  T* pad = (T*)(s < 2 ? fs.ph[ax][fs.cur][s] : fs.pe[ax][s - 2]);
  // extents of the slot's component, the band along the face axis (cpml.js:147-448)
  const bool first = s == 0 || s == 3;
  int n[3] = {nx, ny, nz};
  if (f / 2 == 0) n[first ? 1 : 2]++;
  if (f / 2 == 1) n[s % 2 == 0 ? 0 : 2]++;
  if (f / 2 == 2) n[first ? 0 : 1]++;
  n[f / 2] = h.nc;
  long long si, sj;
  if (ax == 0) {
    si = S;
    sj = P;
    pad += c0 * S;
  } else if (ax == 1) {
    si = (long long)nb * P;
    sj = P;
    pad += (long long)c0 * P;
  } else {
    si = (long long)(ny + 1) * nb;
    sj = nb;
    pad += c0;
  }
  CK(fused_repack<T>(pad, si, sj, (T*)h.psi[s], n[0], n[1], n[2], to_pad, c->stream));
  return FDTD_OK;
}

// Every field and present Psi slot.
template <typename T>
int fused_copy(fdtd_ctx* c, int to_pad) {
  for (int q = 0; q < 6; q++)
    if (int rc = fused_copy_field<T>(c, q, to_pad)) return rc;
  for (int f = 0; f < 6; f++)
    for (int s = 0; s < 4 && c->face[f].present; s++)
      if (int rc = fused_copy_psi<T>(c, f, s, to_pad)) return rc;
  return FDTD_OK;
}

int fused_copy_any(fdtd_ctx* c, int to_pad) {
  return c->esz == 8 ? fused_copy<double>(c, to_pad) : fused_copy<float>(c, to_pad);
}

// Brings the dense arrays and the half-step path's counter up to date.
int to_dense(fdtd_ctx* c) {
  if (c->dense_valid) return FDTD_OK;
  CK(cudaSetDevice(c->device));
  int rc = fused_copy_any(c, 0);
  if (rc) return rc;
  const int dts = c->ts - 1;
  CK(xfer(c, c->d_ts, &dts, sizeof(int), cudaMemcpyHostToDevice));
  c->dense_valid = true;
  return FDTD_OK;
}

// The half-step path, or a load, is about to change the dense arrays.
int claim_dense(fdtd_ctx* c) {
  int rc = to_dense(c);
  if (!rc) c->fs.valid = false;
  return rc;
}

void fused_free(fdtd_ctx* c) {
  for (void* p : c->fs.owned) cudaFree(p);
  c->fs = FusedState();
  c->padded = c->wanted = false;
}

// Frees the padded state (after saving what it holds): the set-up changes.
int fused_drop(fdtd_ctx* c) {
  Using use(c->mu);
  int rc = to_dense(c);
  if (rc) return rc;
  c->graphs.clear();
  if (c->stream) cudaStreamSynchronize(c->stream);
  fused_free(c);
  return FDTD_OK;
}

// Layout of a class row for the problem's bands, and the z bands widened to
// whole groups.  *ok = false: the slabs of the two z faces meet.
ClassLayout class_layout(const fdtd_ctx* c, bool* ok) {
  ClassLayout L{};
  const int V = 8 / (int)c->esz;
  int nbz = 0;
  *ok = true;
  for (int el = 0; el < 2; el++) {
    for (int side = 0; side < 2; side++) {
      const HostFace& h = c->face[4 + side];
      const int st = el ? h.e_start : h.m_start;
      L.z0[el][side] = st / V * V;
      L.zw[el][side] = h.nc ? (st + h.nc + V - 1) / V * V - st / V * V : 0;
    }
    nbz = std::max(nbz, L.zw[el][0] + L.zw[el][1]);
    if (L.zw[el][0] && L.zw[el][1] && L.z0[el][0] + L.zw[el][0] > L.z0[el][1] &&
        L.z0[el][1] + L.zw[el][1] > L.z0[el][0])
      *ok = false;
  }
  int o = kRowBands;
  for (int a = 0; a < 3; a++) {
    L.row.o[a] = o;
    L.row.n[a] = a == 2 ? nbz : c->face[2 * a].nc + c->face[2 * a + 1].nc;
    o += 4 * L.row.n[a];  // stays a multiple of 4
  }
  L.row.stride = o;
  return L;
}

constexpr size_t kMaxClassTable = (size_t)256 << 20;  // bytes

template <typename T, class C>
int fused_classes(fdtd_ctx* c, const C& coef, bool* ok) {
  FusedState& fs = c->fs;
  const StepParams<T, C> sp = step_params<T, C>(c, coef);
  const unsigned n = (unsigned)((c->nx + 1) * fused_plane(c));
  ClassTable tb{};
  void* scratch = nullptr;
  const size_t kb = kClassSlots * sizeof(unsigned long long), ib = kClassSlots * sizeof(unsigned);
  if (fused_malloc(c, &scratch, kb + ib + 16)) return FDTD_OK;  // not usable
  tb.key = (unsigned long long*)scratch;
  tb.id = (unsigned*)((char*)scratch + kb);
  tb.count = (int*)(tb.id + kClassSlots);
  int cnt[2] = {0, 0};
  int rc = FDTD_OK;
  const ClassLayout& L = fs.layout;
  cudaError_t e = cudaMemsetAsync(scratch, 0, kb + ib + 16, c->stream);
  if (e == cudaSuccess) e = fused_class_find<T, C>(sp, fused_pitch(c), n, tb, c->stream);
  if (e == cudaSuccess) e = xfer(c, cnt, tb.count, sizeof(cnt), cudaMemcpyDeviceToHost);
  const size_t bytes = (size_t)cnt[0] * L.row.stride * sizeof(T);
  if (e == cudaSuccess && !cnt[1] && bytes <= kMaxClassTable) {
    rc = fused_alloc(c, &fs.tab, bytes);
    if (!rc) {
      e = fused_class_rows<T, C>(sp, fused_pitch(c), n, tb, L, (T*)fs.tab, fs.cls, c->stream);
      if (e == cudaSuccess) e = xfer(c, cnt, tb.count, sizeof(cnt), cudaMemcpyDeviceToHost);
      *ok = e == cudaSuccess && !cnt[1];
    }
  }
  cudaFree(scratch);
  if (e != cudaSuccess) return fail(FDTD_ERR_CUDA, "cell classes: %s", cudaGetErrorString(e));
  return rc == FDTD_ERR_OOM ? FDTD_OK : rc;
}

// Profiles b, a over a whole axis, zero outside the bands; along z in FP32, where
// a slab holds other columns too, b is -0 there (in_band).
int fused_axis_values(const fdtd_ctx* c, int a) { return (a == 0 ? c->nx + 1 : a == 1 ? c->ny + 1 : fused_pitch(c)) + 8; }

int fused_profiles(fdtd_ctx* c) {
  for (int el = 0; el < 2; el++) {
    if (c->esz == 4)  // the sign bytes
      CK(cudaMemset2DAsync((char*)c->fs.prof[el][2][0] + 3, 4, 0x80, 1, fused_axis_values(c, 2), c->stream));
    for (int f = 0; f < 6; f++) {
      const HostFace& h = c->face[f];
      for (int w = 0; w < 2 && h.present; w++)
        CK(cudaMemcpyAsync((char*)c->fs.prof[el][f / 2][w] + (el ? h.e_start : h.m_start) * c->esz,
                           h.prof[(el ? 0 : 2) + w], h.nc * c->esz, cudaMemcpyDeviceToDevice, c->stream));
    }
  }
  return FDTD_OK;
}

// Probe cells in the padded layout, probe after probe.
std::vector<int> fused_probe_cells(const fdtd_ctx* c) {
  const int P = fused_pitch(c);
  const long long S = fused_plane(c);
  std::vector<int> v;
  auto put = [&](int comp, int idx) {
    const int nj = (comp == 0 || comp == 2 || comp == 4) ? c->ny : c->ny + 1,
              nk = (comp == 0 || comp == 1 || comp == 5) ? c->nz : c->nz + 1;
    v.push_back((int)((idx / (nj * nk)) * S + (long long)((idx / nk) % nj) * P + idx % nk));
  };
  for (const auto& pr : c->vprobe)
    for (int x : pr.cells) put(3 + pr.comp, x);
  for (const auto& pr : c->iprobe)
    for (size_t m = 0; m < pr.cells.size(); m++) put(pr.comps[m], pr.cells[m]);
  return v;
}

// Builds the padded state.  It serves problems whose CPML bands are disjoint
// per axis (along z as whole groups), whose padded arrays have 32-bit indices,
// with at most 65,536 cell classes, and whose padded state takes at most half
// of the device memory that is free; others keep the half-step path.
int fused_build(fdtd_ctx* c) {
  FusedState& fs = c->fs;
  const int P = fused_pitch(c);
  const long long S = fused_plane(c);
  const long long elems = (long long)(c->nx + 1) * S;
  if (!bands_disjoint(c) || elems + 2 * S > (1LL << 31) - 1) return FDTD_OK;
  bool slabs = false;
  fs.layout = class_layout(c, &slabs);
  if (!slabs) return FDTD_OK;
  const size_t comp = (size_t)elems * c->esz;
  long long psi[3] = {};
  size_t need = 12 * comp + (size_t)elems * 2;
  for (int a = 0; a < 3; a++) {
    const int nb = fs.layout.row.n[a];
    psi[a] = nb * (a == 0 ? S : (long long)(c->nx + 1) * (a == 1 ? P : c->ny + 1));
    if (psi[a] > (1LL << 31) - 1) return FDTD_OK;
    need += 6 * (size_t)psi[a] * c->esz;
  }
  size_t free_b = 0, total_b = 0;
  CK(cudaMemGetInfo(&free_b, &total_b));
  if (need > free_b / 2) {
    fs.no_room_at = c->ts;
    return FDTD_OK;
  }
  Arena ar;
  for (int w = 0; w < 2; w++)
    for (int q = 0; q < 6; q++) ar.add(&fs.f[w][q], comp);
  for (int a = 0; a < 3; a++)
    for (int s = 0; s < 2 && psi[a]; s++) {
      for (int w = 0; w < 2; w++) ar.add(&fs.ph[a][w][s], (size_t)psi[a] * c->esz);
      ar.add(&fs.pe[a][s], (size_t)psi[a] * c->esz);
    }
  ar.add(&fs.cls, (size_t)elems * 2);
  ar.add(&fs.d_ts, 2 * sizeof(int));
  for (int el = 0; el < 2; el++)
    for (int a = 0; a < 3; a++)
      for (int w = 0; w < 2; w++) ar.add(&fs.prof[el][a][w], fused_axis_values(c, a) * c->esz);
  const std::vector<int> cells = fused_probe_cells(c);
  int* d_cells = nullptr;
  ar.add(&d_cells, cells.size() * sizeof(int));
  void* base = nullptr;
  int rc = fused_alloc(c, &base, ar.size);
  if (!rc) {
    ar.place(base);
    rc = fused_profiles(c);
  }
  if (!rc && !cells.empty()) {
    CK(cudaMemcpyAsync(d_cells, cells.data(), cells.size() * sizeof(int), cudaMemcpyHostToDevice, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    for (size_t q = 0; q < c->vprobe.size(); d_cells += c->vprobe[q++].cells.size()) fs.v_idx[q] = d_cells;
    for (size_t q = 0; q < c->iprobe.size(); d_cells += c->iprobe[q++].cells.size()) fs.i_idx[q] = d_cells;
  }
  bool ok = false;
  if (!rc) {
    if (c->prec == FDTD_PREC_F64)
      rc = fused_classes<double, ArrayCoef<double>>(c, array_coef<double>(c), &ok);
    else if (c->prec == FDTD_PREC_F32)
      rc = fused_classes<float, ArrayCoef<float>>(c, array_coef<float>(c), &ok);
    else
      rc = fused_classes<float, TableCoef>(c, c->tcoef, &ok);
  }
  if (rc == FDTD_ERR_OOM) rc = FDTD_OK;  // no room after all
  fs.ok = !rc && ok;
  return rc;
}

// A padded state that was refused for want of memory is tried again after so many
// steps: memory may be free by then, and a question costs little over them.
constexpr int kRetrySteps = 512;
bool fused_retry(const fdtd_ctx* c) {
  return c->fs.tried && !c->fs.ok && c->fs.no_room_at >= 0 && std::abs(c->ts - c->fs.no_room_at) >= kRetrySteps;
}

// Builds the padded state where there is none; *use = false: half-step path.
int fused_usable(fdtd_ctx* c, bool* use) {
  FusedState& fs = c->fs;
  *use = false;
  if (c->half_steps) return FDTD_OK;
  if (fused_retry(c)) fs = FusedState();
  if (c->wanted) return fused_drop(c);  // this run takes the half-step path, a later one builds again
  if (!fs.tried) {
    int rc = fused_build(c);
    if (rc || !fs.ok) {
      const int no_room_at = fs.no_room_at;
      fused_free(c);
      fs.no_room_at = no_room_at;
      fs.tried = rc == FDTD_OK;
      if (rc) return rc;
    } else {
      fs.tried = true;
    }
  }
  *use = fs.ok;
  return FDTD_OK;
}

// And makes it hold the current fields and step, where the one-pass step is used.
int fused_ready(fdtd_ctx* c, bool* use) {
  FusedState& fs = c->fs;
  int rc = fused_usable(c, use);
  if (rc || !*use) return rc;
  if (!fs.valid) {
    rc = fused_copy_any(c, 1);
    if (rc) return rc;
    fs.valid = true;
    fs.ts_at = -1;
  }
  if (fs.ts_at != c->ts) {
    CK(xfer(c, fs.d_ts + fs.cur, &c->ts, sizeof(int), cudaMemcpyHostToDevice));
    fs.ts_at = c->ts;
  }
  return FDTD_OK;
}

// cuTensorMapEncodeTiled, through the runtime (the library does not link the driver).
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
    return (EncodeTiled)p;
  }();
  return fn;
}

// Tensor map of one padded array: (w, rows, 1) tiles of (k, j, i).
template <typename T>
bool fused_map(const fdtd_ctx* c, CUtensorMap* m, const T* base, int w, int rows) {
  const cuuint64_t dim[3] = {(cuuint64_t)fused_pitch(c), (cuuint64_t)c->ny + 1, (cuuint64_t)c->nx + 1};
  const cuuint64_t stride[2] = {dim[0] * sizeof(T), (cuuint64_t)fused_plane(c) * sizeof(T)};
  const CUtensorMapDataType type = sizeof(T) == 8   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64
                                   : sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                                    : CU_TENSOR_MAP_DATA_TYPE_UINT16;
  const cuuint32_t box[3] = {(cuuint32_t)w, (cuuint32_t)rows, 1}, one[3] = {1, 1, 1};
  const EncodeTiled enc = encode_tiled();
  return enc && enc(m, type, 3,
                    (void*)base, dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tiles: a row as few k tiles of equal width as hold it, then the number of x
// chunks (one tile of each per block): a chunk recomputes one H plane, sets up
// and fills its pipeline, about kFusedFill planes' time, and a plane with Psi
// takes about 1 + kFusedBand times that of one without (512 x 512 x 640,
// material table, 8-cell CPML: 2.3 ms of 2.97 without the z bands' Psi, 2.6
// without the y bands', 1.7 without any).
constexpr double kFusedFill = 5, kFusedBand = 0.6;
template <typename T>
void fused_shape(const fdtd_ctx* c, FusedParams<T>& p, double share) {
  const int cols = c->nz + 1;
  // owned columns: all of them, or a multiple of four (a tile starts on 16
  // bytes) with room for the halo group
  constexpr int V = FusedShape<T>::V;
  p.halo_k = cols > kTileCols;
  p.tk = p.halo_k ? (cols + kTileCols - 5) / (kTileCols - 4) : 1;
  p.rk = (p.halo_k ? ((cols + p.tk - 1) / p.tk + 3) / 4 * 4 : (cols + V - 1) / V * V) / V + p.halo_k;
  p.tj = (c->ny + kTileRows - 1) / (kTileRows - 1);
  // tiles that meet a band, from the low and from the high end
  auto slow = [](const FusedAxis<T>& x, int width, int n, int* out) {
    int lo = 0, hi = n;
    for (int e = 0; e < 2; e++) {
      if (x.nc[e][0] > 0) lo = std::max(lo, (x.start[e][0] + x.nc[e][0] - 1) / width + 1);
      if (x.nc[e][1] > 0) hi = std::min(hi, x.start[e][1] / width);
    }
    out[0] = std::min(lo, n);
    out[1] = n - std::max(std::min(hi, n), out[0]);
  };
  slow(p.axis[1], kTileRows - 1, p.tj, p.slow_j);
  slow(p.axis[2], (p.rk - p.halo_k) * V, p.tk, p.slow_k);
  const int nxp = c->nx + 1;
  // Blocks of the three kinds that fused_place orders, per x chunk, and their
  // time per plane: the device takes them in that order, a free slot the next.
  const int nj = p.slow_j[0] + p.slow_j[1], nk = p.slow_k[0] + p.slow_k[1];
  const int kind[3] = {nj * p.tk, (p.tj - nj) * nk, (p.tj - nj) * (p.tk - nk)};
  int xb[2] = {0, 0};  // planes in the x bands
  for (int f = 0; f < 2; f++) xb[f] = std::max(p.axis[0].nc[0][f], p.axis[0].nc[1][f]);
  double t_best = -1;
  const int slots = std::max(1, (int)(148 * FusedShape<T>::kBlocks * share));
  const int n_max = std::min(nxp, 64 + 4 * slots / (p.tk * p.tj));
  for (int n = 1; n <= n_max; n++) {
    std::map<double, int> free_at;  // time -> slots
    free_at[0] = slots;
    double end = 0;
    const double planes = (nxp + n - 1) / n;
    for (int q = 0; q < 3; q++)
      for (int z = 0; z < 2; z++) {  // the chunks at the ends, the others
        long long blocks = (long long)kind[q] * (z ? std::max(0, n - 2) : std::min(n, 2));
        const double band = z ? 0 : std::min(planes, (double)std::max(xb[0], xb[1]) * (n == 1 ? 2 : 1));
        const double t = (planes + kFusedFill + kFusedBand * band) * (q < 2 ? 1 + kFusedBand : 1.0);
        while (blocks > 0) {
          const auto it = free_at.begin();
          const double at = it->first + t;
          const int m = (int)std::min<long long>(blocks, it->second);
          if (m == it->second) free_at.erase(it); else it->second -= m;
          free_at[at] += m;
          end = std::max(end, at);
          blocks -= m;
        }
      }
    if (t_best < 0 || end < t_best) {
      t_best = end;
      p.tx = n;
    }
  }
}

template <typename T>
FusedParams<T> fused_params(const fdtd_ctx* c, int flip, double share) {
  const FusedState& fs = c->fs;
  FusedParams<T> p{};
  p.nx = c->nx; p.ny = c->ny; p.nz = c->nz;
  p.pitch = fused_pitch(c);
  p.plane = (unsigned)fused_plane(c);
  for (int q = 0; q < 6; q++) {
    p.fi[q] = (const T*)fs.f[flip][q];
    p.fo[q] = (T*)fs.f[flip ^ 1][q];
  }
  p.cls = fs.cls;
  p.tab = (const T*)fs.tab;
  p.row = fs.layout.row;
  for (int a = 0; a < 3; a++) {
    FusedAxis<T>& x = p.axis[a];
    for (int el = 0; el < 2; el++)
      for (int f = 0; f < 2; f++) {
        const HostFace& h = c->face[2 * a + f];
        x.nc[el][f] = a == 2 ? fs.layout.zw[el][f] : h.nc;
        x.start[el][f] = a == 2 ? fs.layout.z0[el][f] : el ? h.e_start : h.m_start;
      }
    x.nb = fs.layout.row.n[a];
    for (int s = 0; s < 2; s++) {
      x.phi[s] = (const T*)fs.ph[a][flip][s];
      x.pho[s] = (T*)fs.ph[a][flip ^ 1][s];
      x.pe[s] = (T*)fs.pe[a][s];
      for (int w = 0; w < 2; w++) x.prof[s][w] = (const T*)fs.prof[s][a][w];
    }
  }
  p.ts = fs.d_ts + flip;
  p.ts_next = fs.d_ts + (flip ^ 1);
  p.src = dev_sources<T>(c);
  p.x_wall = c->x_wall;
  p.fault = c->d_status;
  fused_shape(c, p, share);
  for (int q = 0; q < 6; q++) {
    if (!fused_map(c, &p.map[q], p.fi[q], kTileW, q < 3 ? kTileRows : kTileRows + 1)) p.tx = 0;  // no maps: no launch
  }
  if (!fused_map(c, &p.map[6], p.cls, kTileC, kTileRows)) p.tx = 0;
  return p;
}

Probes fused_dev_probes(const fdtd_ctx* c) {
  Probes p = dev_probes(c);
  for (int q = 0; q < p.n_v; q++) p.v_idx[q] = c->fs.v_idx[q];
  for (int q = 0; q < p.n_i; q++) p.i_idx[q] = c->fs.i_idx[q];
  return p;
}

long long surface_points(const fdtd_ctx* c) { return c->nFreq > 0 ? c->ffsz[0] + c->ffsz[1] + c->ffsz[2] : 0; }

// `count` steps from copy `flip` and step `ts` on stream `st`.  Alone on the
// device (share 1), a step's epilogue is queued after the next step's launch and
// runs beside it, the last one's after its own; with other problems' launches
// around it (share < 1, its part of the device) a launch waits for the one ahead
// instead of holding slots that they could use.
template <typename T, bool EXACT>
int fused_enqueue_steps(fdtd_ctx* c, int count, int flip, int ts, KernelTimer* tm, cudaStream_t st, double share) {
  const bool alone = share == 1;
  const FusedParams<T> pf[2] = {fused_params<T>(c, 0, share), fused_params<T>(c, 1, share)};  // by the copy read
  if (pf[0].tx == 0 || pf[1].tx == 0) return fail(FDTD_ERR_CUDA, "cannot encode the step's tensor maps");
  const Probes pr = fused_dev_probes(c);
  const FarField ff = dev_ff(c);
  const int probes = pr.n_v + pr.n_i;
  const long long pts = surface_points(c);
  const unsigned epi = pts + probes ? (unsigned)((epilogue_threads(pts, probes) + 255) / 256) : 0;
  // the epilogue of step `step`, under the parameters of the step after it or its own
  auto epilogue = [&](const FusedParams<T>& p, int step, bool late) -> cudaError_t {
    if (!epi) return cudaSuccess;
    cudaError_t e = fused_epilogue<T>(p, ff, pr, epi, late, alone, st);
    if (e == cudaSuccess && c->dft_block > 0 && (step + 1) % c->dft_block == 0)
      e = dft_flush(ff, late ? p.ts : p.ts_next, -2, st);
    return e;
  };
  for (int s = 0; s < count; s++, flip ^= 1) {
    const FusedParams<T>& p = pf[flip];
    if (tm) CK(cudaEventRecord(tm->ev[0], st));
    CK((fused_step<T, EXACT>(p, alone, st)));
    if (tm) CK(cudaEventRecord(tm->ev[1], st));
    if (!p.x_wall) CK((fused_wall<T, EXACT>(p, st)));
    if (tm) {
      CK(cudaEventRecord(tm->ev[2], st));
      CK(cudaEventRecord(tm->ev[3], st));
    }
    const bool late = alone && !tm;
    if (late && s > 0) CK(epilogue(p, ts + s - 1, true));
    if (!late || s + 1 == count) CK(epilogue(p, ts + s, false));
    if (tm) {
      CK(cudaEventRecord(tm->ev[4], st));
      CK(cudaEventSynchronize(tm->ev[4]));
      for (int q = 0; q < 4; q++) {
        if (q == 2 || (q == 1 && p.x_wall)) continue;  // no launch
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, tm->ev[q], tm->ev[q + 1]));
        tm->ms[q] += ms;
      }
    }
  }
  CK(cudaGetLastError());
  return FDTD_OK;
}

// `count` steps, `at` steps on from the handle's present state.
int fused_enqueue(fdtd_ctx* c, int at, int count, KernelTimer* tm = nullptr, cudaStream_t st = nullptr,
                  double share = 1) {
  if (!st) st = c->stream;
  const int flip = c->fs.cur ^ (at & 1), ts = c->ts + at;
  if (c->prec == FDTD_PREC_F64) return fused_enqueue_steps<double, true>(c, count, flip, ts, tm, st, share);
  if (c->prec == FDTD_PREC_F32) return fused_enqueue_steps<float, true>(c, count, flip, ts, tm, st, share);
  return fused_enqueue_steps<float, false>(c, count, flip, ts, tm, st, share);
}

int enqueue(fdtd_ctx* c, int count, KernelTimer* tm = nullptr, cudaStream_t st = nullptr) {
  if (c->prec == FDTD_PREC_F64)
    return enqueue_steps<double, ArrayCoef<double>, true>(c, array_coef<double>(c), count, tm, st);
  if (c->prec == FDTD_PREC_F32)
    return enqueue_steps<float, ArrayCoef<float>, true>(c, array_coef<float>(c), count, tm, st);
  return enqueue_steps<float, TableCoef, false>(c, c->tcoef, count, tm, st);
}

// End of a run that reached step `upto` with the time-blocked DFT: accumulate
// what the run left buffered (the open block) and mark it done.
int close_dft_block(fdtd_ctx* c, int upto, cudaStream_t st) {
  if (c->dft_block <= 0) return FDTD_OK;
  if (upto % c->dft_block != 0) CK(dft_flush(dev_ff(c), c->d_ts, upto, st));
  CK(cudaMemcpyAsync(c->d_dft_done, &upto, sizeof(int), cudaMemcpyHostToDevice, st));
  CK(cudaStreamSynchronize(st));  // `upto` is read from this frame
  return FDTD_OK;
}

// The graph of a piece of a run that starts as `s` says, from the cache, captured
// on `st` through `enq` (which enqueues those steps) when missing.
template <class Enq>
int graph_for(RunGraphs& rg, cudaStream_t st, const RunPiece& piece, const RunStart& s, int launches_per_step, Enq enq,
              cudaGraphExec_t* out) {
  const long long key = s.after(piece.at).key(piece.steps);
  if (cudaGraphExec_t* have = rg.cache.find(key)) {
    *out = *have;
    return FDTD_OK;
  }
  cudaGraph_t g;
  CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  int erc = enq(piece.at, piece.steps);
  cudaError_t ce = cudaStreamEndCapture(st, &g);
  if (erc) return erc;
  if (ce != cudaSuccess) return fail(FDTD_ERR_CUDA, "graph capture: %s", cudaGetErrorString(ce));
  cudaGraphExec_t ge = nullptr;
  ce = cudaGraphInstantiate(&ge, g, 0);
  cudaGraphDestroy(g);
  if (ce != cudaSuccess) return fail(FDTD_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(ce));
  rg.cache.add(key, (long long)piece.steps * launches_per_step, ge, [](cudaGraphExec_t old) { cudaGraphExecDestroy(old); });
  *out = ge;
  return FDTD_OK;
}

// The graph launches of a run of `count` steps that starts as `s` says, in pieces
// of at most `cap` steps (0: as many as a graph may hold), each captured (if
// missing) now: enq(at, steps) enqueues `steps` steps, `at` steps into the run.
template <class Enq>
int run_plan(RunGraphs& rg, cudaStream_t st, int count, int launches_per_step, const RunStart& s, Enq enq,
             std::vector<cudaGraphExec_t>* plan, int cap = 0) {
  plan->clear();
  for (const RunPiece& piece : run_pieces(count, s, launches_per_step, cap)) {
    cudaGraphExec_t ge = nullptr;
    if (int rc = graph_for(rg, st, piece, s, launches_per_step, enq, &ge)) return rc;
    plan->push_back(ge);
  }
  return FDTD_OK;
}

// Where the one-pass step's next run starts.
RunStart fused_start(const fdtd_ctx* c) {
  RunStart s;
  s.one_pass = true;
  s.copy = c->fs.cur;
  s.block = c->dft_block;
  s.phase = s.block > 0 ? c->ts % s.block : 0;
  return s;
}

constexpr int kMaxBatchStreams = 32;

// What the handle's two status words say about the run that just ended, read on
// stream `st`; `who` names the handle in the message ("" or "batch member 3: ").
int check_status(const fdtd_ctx* c, cudaStream_t st, const std::string& who = "") {
  int w[2];
  CK(cudaMemcpyAsync(w, c->d_status, sizeof(w), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (w[0] == FDTD_ERR_CUDA) return fail(FDTD_ERR_CUDA, "%sa bounded device wait of the step ran out", who.c_str());
  if (w[0] != 0) return fail(FDTD_ERR_NONFINITE, "%snon-finite port sample at step %d", who.c_str(), w[1]);
  return FDTD_OK;
}

int run_steps(fdtd_ctx* c, int count, float* elapsed_ms = nullptr, KernelTimer* tm = nullptr) {
  if (count < 0) return fail(FDTD_ERR_BADARG, "negative step count %d", count);
  Using use(c->mu);
  if (c->ts + count > c->nsteps)
    return fail(FDTD_ERR_BADARG, "running %d steps from step %d exceeds numberOfTimeSteps=%d", count, c->ts,
                c->nsteps);
  int rc = check_ready(c);
  if (rc) return rc;
  rc = ensure_traces(c);
  if (rc) return rc;
  CK(cudaSetDevice(c->device));
  if (c->prec == FDTD_PREC_F32_TABLE && c->table_dirty) {
    rc = prepare_table(c, &c->tcoef);
    if (rc) return rc;
  }
  if (count > 0) {
    rc = check_shape(c);
    if (rc) return rc;
  }
  bool fused = false;
  if (count > 0) {
    rc = fused_ready(c, &fused);
    if (!rc && !fused) rc = claim_dense(c);
    if (rc) return rc;
  }
  // the whole run as cached graphs, captured before the first launch
  if (c->dirty) {
    c->graphs.clear();
    c->dirty = false;
  }
  std::vector<cudaGraphExec_t> plan;
  if (!tm && fused) {
    rc = run_plan(c->graphs, c->stream, count, 3, fused_start(c), [c](int at, int n) { return fused_enqueue(c, at, n); },
                  &plan);
    if (rc) return rc;
  } else if (!tm) {
    rc = run_plan(c->graphs, c->stream, count, c->dft_block > 0 ? 5 : 4, RunStart(),
                  [c](int, int n) { return enqueue(c, n); }, &plan);
    if (rc) return rc;
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  if (elapsed_ms) {
    CK(cudaEventCreate(&ev0));
    CK(cudaEventCreate(&ev1));
    CK(cudaEventRecord(ev0, c->stream));
  }
  if (fused) {
    // from here the padded state runs ahead of the dense one
    c->dense_valid = false;
    c->fs.valid = true;
  }
  if (tm) {
    rc = fused ? fused_enqueue(c, 0, count, tm) : enqueue(c, count, tm);
    if (rc) return rc;
  }
  for (cudaGraphExec_t ge : plan) CK(cudaGraphLaunch(ge, c->stream));
  if (fused) {
    c->fs.cur ^= count & 1;
    c->fs.ts_at = c->ts + count;
  }
  if (elapsed_ms) {
    CK(cudaEventRecord(ev1, c->stream));
    CK(cudaEventSynchronize(ev1));
    CK(cudaEventElapsedTime(elapsed_ms, ev0, ev1));
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
  }
  if (count > 0) {
    rc = close_dft_block(c, c->ts + count, c->stream);
    if (rc) return rc;
  }
  CK(cudaStreamSynchronize(c->stream));
  c->ts += count;
  return check_status(c, c->stream);
}

unsigned long long mix64(unsigned long long h, unsigned long long w) {
  h ^= w;
  h *= 0xff51afd7ed558ccdULL;
  return h ^ (h >> 33);
}

// Folds `n` bytes at `p`, with the call's tag and the byte count, into the
// handle's set-up digest: eight independent lanes of eight bytes (so the
// multiplies overlap; a 168 MB material grid takes about 12 ms), then the
// remaining words and bytes.
void digest(fdtd_ctx* c, int tag, const void* p, size_t n) {
  unsigned long long h = mix64(c->setup_digest, ((unsigned long long)tag << 48) ^ (unsigned long long)n);
  const unsigned char* b = (const unsigned char*)p;
  size_t i = 0;
  if (n >= 64) {
    unsigned long long lane[8];
    for (int l = 0; l < 8; l++) lane[l] = h + 0x9e3779b97f4a7c15ULL * (unsigned long long)(l + 1);
    for (; i + 64 <= n; i += 64)
      for (int l = 0; l < 8; l++) {
        unsigned long long w;
        memcpy(&w, b + i + 8 * l, 8);
        lane[l] = mix64(lane[l], w);
      }
    for (int l = 0; l < 8; l++) h = mix64(h, lane[l]);
  }
  for (; i + 8 <= n; i += 8) {
    unsigned long long w;
    memcpy(&w, b + i, 8);
    h = mix64(h, w);
  }
  unsigned long long t = 0;
  for (; i < n; i++) t = (t << 8) | b[i];
  c->setup_digest = mix64(h, t);
}

void digest_vals(fdtd_ctx* c, int tag, std::initializer_list<double> v) {
  std::vector<double> a(v);
  digest(c, tag, a.data(), a.size() * sizeof(double));
}

}  // namespace

int fdtd_internal_traces(const fdtd_ctx* c, const double** V, const double** I, int* nsteps, int* steps,
                         int* device) {
  if (c->vprobe.empty() || c->iprobe.empty())
    return fail(FDTD_ERR_STATE, "handle has no voltage probe or no current probe");
  *V = c->V;
  *I = c->I;
  *nsteps = c->nsteps;
  *steps = c->ts;
  *device = c->device;
  return FDTD_OK;
}

// ===========================================================================
// Handle API
// ===========================================================================
extern "C" {

static int set_rows(fdtd_ctx* c, int comp, const std::vector<double>& rows);

const char* fdtd_last_error(void) { return g_err; }

int fdtd_device_count(int* count) {
  if (!count) return fail(FDTD_ERR_BADARG, "count is NULL");
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) n = 0;
  *count = n;
  return FDTD_OK;
}

int fdtd_create(const FdtdConfig* cfg, fdtd_ctx** out) {
  if (!cfg || !out) return fail(FDTD_ERR_BADARG, "NULL argument");
  *out = nullptr;
  if (cfg->nx < 2 || cfg->ny < 2 || cfg->nz < 2) return fail(FDTD_ERR_BADARG, "grid %dx%dx%d too small", cfg->nx, cfg->ny, cfg->nz);
  if ((long long)(cfg->nx + 1) * (cfg->ny + 1) * (cfg->nz + 1) > (1LL << 31) - 1)
    return fail(FDTD_ERR_BADARG, "grid too large for 32-bit component indices");
  if (cfg->numberOfTimeSteps < 1) return fail(FDTD_ERR_BADARG, "numberOfTimeSteps must be >= 1");
  if (cfg->precision < FDTD_PREC_F64 || cfg->precision > FDTD_PREC_F32_TABLE)
    return fail(FDTD_ERR_BADARG, "unknown precision %d", cfg->precision);
  if (!(cfg->dx > 0 && cfg->dy > 0 && cfg->dz > 0 && cfg->dt > 0)) return fail(FDTD_ERR_BADARG, "non-positive spacing");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || cfg->device < 0 || cfg->device >= ndev)
    return fail(FDTD_ERR_CUDA, "CUDA device %d not available", cfg->device);
  fdtd_ctx* c = new fdtd_ctx();
  c->device = cfg->device;
  c->prec = cfg->precision;
  c->esz = (c->prec == FDTD_PREC_F64) ? 8 : 4;
  c->nx = cfg->nx; c->ny = cfg->ny; c->nz = cfg->nz;
  c->dx = cfg->dx; c->dy = cfg->dy; c->dz = cfg->dz; c->dt = cfg->dt;
  c->nsteps = cfg->numberOfTimeSteps;
  c->x_wall = c->prec == FDTD_PREC_F64 ? 0 : 1;
  digest_vals(c, 1, {(double)c->nx, (double)c->ny, (double)c->nz, c->dx, c->dy, c->dz, c->dt, (double)c->nsteps,
                     (double)c->prec});
  const long long nx = c->nx, ny = c->ny, nz = c->nz;
  c->ncomp[0] = (nx + 1) * ny * nz;
  c->ncomp[1] = nx * (ny + 1) * nz;
  c->ncomp[2] = nx * ny * (nz + 1);
  c->ncomp[3] = nx * (ny + 1) * (nz + 1);
  c->ncomp[4] = (nx + 1) * ny * (nz + 1);
  c->ncomp[5] = (nx + 1) * (ny + 1) * nz;
  int rc = FDTD_OK;
  if (cudaSetDevice(c->device) != cudaSuccess || cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete c;
    return fail(FDTD_ERR_CUDA, "cannot create a stream on device %d", cfg->device);
  }
  long long tot = 0;
  for (int q = 0; q < 6; q++) tot += c->ncomp[q];
  tot += (ny + 1) * (nz + 1) + 64;  // slack plane past Ez
  Arena ar;
  ar.add(&c->fields, tot * c->esz);
  ar.add(&c->ex0b, (size_t)(ny + 1) * (nz + 1) * c->esz);
  ar.add(&c->d_ts, sizeof(int));
  ar.add(&c->d_status, 2 * sizeof(int));
  // ids: 64 bytes of padding, as the staged kernels copy whole aligned words of
  // ids, and the bulk-copied rows (32 ids widened to 16-byte boundaries) may
  // reach up to 47 bytes past the last id
  for (int q = 0; q < 18 && c->prec != FDTD_PREC_F32_TABLE; q++) ar.add(&c->coef[q], coef_count(c, q) * c->esz);
  for (int q = 0; q < 6 && c->prec == FDTD_PREC_F32_TABLE; q++) ar.add(&c->ids[q], c->ncomp[(q + 3) % 6] + 64);
  void* base = nullptr;
  rc = dalloc(c, &base, ar.size);
  if (!rc) ar.place(base);
  if (!rc) {
    int init_ts = -1;
    int st[2] = {0, 1 << 30};
    if (xfer(c, c->d_ts, &init_ts, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess ||
        xfer(c, c->d_status, st, sizeof(st), cudaMemcpyHostToDevice) != cudaSuccess)
      rc = fail(FDTD_ERR_CUDA, "cannot initialise step counter");
  }
  if (!rc) rc = ensure_traces(c);
  if (!rc) {
    // default launch shape: enough x chunks for about four waves of 2048-thread SMs
    const long long cols = (long long)(ny + 1) * (nz + 1);
    const long long want = 4LL * 148 * 2048;
    long long ch = cols * (nx + 1) / want;
    c->ichunk = (int)std::max<long long>(1, std::min<long long>(64, ch));
  }
  if (!rc && cudaStreamSynchronize(c->stream) != cudaSuccess) rc = fail(FDTD_ERR_CUDA, "stream sync failed");
  if (rc) {
    std::string msg = g_err;
    fdtd_free(c);
    return fail(rc, "%s", msg.c_str());
  }
  {
    std::lock_guard<std::mutex> g(handles().mu);
    handles().all.push_back(c);
  }
  *out = c;
  return FDTD_OK;
}

void fdtd_free(fdtd_ctx* c) {
  if (!c) return;
  {
    // after this no other thread's reclaim_padded finds the handle
    std::lock_guard<std::mutex> g(handles().mu);
    auto& all = handles().all;
    all.erase(std::remove(all.begin(), all.end(), c), all.end());
  }
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  c->graphs.clear();
  fused_free(c);
  for (void* p : c->owned) cudaFree(p);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

int fdtd_ctx_upload_coeff(fdtd_ctx* c, int which, const double* host, long n) {
  if (!c || !host) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (c->prec == FDTD_PREC_F32_TABLE) return fail(FDTD_ERR_STATE, "material-table problem takes fdtd_ctx_upload_material");
  if (which < 0 || which >= 18) return fail(FDTD_ERR_BADARG, "coefficient id %d out of range 0..17", which);
  if (n != coef_count(c, which)) return fail(FDTD_ERR_BADARG, "coefficient %d: got %ld values, expected %lld", which, n, coef_count(c, which));
  digest_vals(c, 2, {(double)which});
  digest(c, 2, host, (size_t)n * sizeof(double));
  CK(cudaSetDevice(c->device));
  int rc = fused_drop(c);
  if (!rc) rc = upload_real(c, c->coef[which], host, n);
  if (!rc) c->coef_set[which] = true;
  c->coef_device = false;  // host arrays carry their own kappa division and come with CPsi
  return rc;
}

// The CPML bands of face f on the four per-cell FP64 coefficient arrays its
// Psi slots correct (cpml.js:212-243): per slot, CPsi = coefficient x cell size
// over the band (into the face's CPsi array), then the coefficient is divided
// by kappa of its band cell.  Slots: x face Chyez Chzey Ceyhz Cezhy, y face
// Chxez Chzex Cezhx Cexhz, z face Chxey Chyex Cexhy Ceyhx (ids as in
// fdtd_ctx_upload_coeff); the H slots use the H band and kappa_m, the E slots
// the E band and kappa_e.
static int cpml_band_on_device(fdtd_ctx* c, int f, const double* kappa_e, const double* kappa_m) {
  static const int coef_id[3][4] = {{13, 17, 5, 7}, {11, 16, 8, 1}, {10, 14, 2, 4}};
  const int axis = f / 2;
  HostFace& h = c->face[f];
  const double cell = axis == 0 ? c->dx : (axis == 1 ? c->dy : c->dz);
  double* d_kap = nullptr;
  if (dev_malloc(c, &d_kap, 2 * h.nc * sizeof(double)) != cudaSuccess) return fail(FDTD_ERR_OOM, "kappa profiles");
  int rc = FDTD_OK;
  if (xfer(c, d_kap, kappa_e, h.nc * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
      xfer(c, d_kap + h.nc, kappa_m, h.nc * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
    rc = fail(FDTD_ERR_CUDA, "kappa upload");
  for (int s = 0; s < 4 && !rc; s++) {
    const int id = coef_id[axis][s], comp = id / 3;   // API order Ex Ey Ez Hx Hy Hz
    const int ni = (comp == 0 || comp == 4 || comp == 5) ? c->nx : c->nx + 1;
    const int nj = (comp == 1 || comp == 3 || comp == 5) ? c->ny : c->ny + 1;
    const int nk = (comp == 2 || comp == 3 || comp == 4) ? c->nz : c->nz + 1;
    const int st = s < 2 ? h.m_start : h.e_start;
    const long long n = (long long)(axis == 0 ? h.nc : ni) * (axis == 1 ? h.nc : nj) * (axis == 2 ? h.nc : nk);
    if (n != h.n[s]) { rc = fail(FDTD_ERR_STATE, "face %d slot %d: band of %lld cells, Psi of %lld", f, s, n, h.n[s]); break; }
    k_cpml_band<<<148 * 8, 256, 0, c->stream>>>((double*)c->coef[id], ni, nj, nk, axis, st, h.nc, cell,
                                                s < 2 ? d_kap + h.nc : d_kap, (double*)h.cpsi[s]);
  }
  if (!rc && cudaStreamSynchronize(c->stream) != cudaSuccess)
    rc = fail(FDTD_ERR_CUDA, "CPML band: %s", cudaGetErrorString(cudaGetLastError()));
  cudaFree(d_kap);
  if (!rc) c->kappa_done[f] = true;
  return rc;
}

int fdtd_ctx_upload_cpml(fdtd_ctx* c, int f, int nc, const double* b_e, const double* a_e, const double* b_m,
                         const double* a_m, const double* kappa_e, const double* kappa_m, const double* CPsi0,
                         long n0, const double* CPsi1, long n1, const double* CPsi2, long n2, const double* CPsi3,
                         long n3, int m_start, int e_start) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (f < 0 || f >= 6) return fail(FDTD_ERR_BADARG, "face id %d out of range 0..5", f);
  if (nc < 0) return fail(FDTD_ERR_BADARG, "negative cell count");
  const int axis_n = f / 2 == 0 ? c->nx : (f / 2 == 1 ? c->ny : c->nz);
  if (nc > axis_n / 2) return fail(FDTD_ERR_BADARG, "face %d: %d CPML cells do not fit in %d cells", f, nc, axis_n);
  if (m_start < 0 || m_start + nc > axis_n) return fail(FDTD_ERR_BADARG, "face %d: H band [%d,%d) outside [0,%d)", f, m_start, m_start + nc, axis_n);
  if (e_start < 1 || e_start + nc > axis_n) return fail(FDTD_ERR_BADARG, "face %d: E band [%d,%d) outside [1,%d)", f, e_start, e_start + nc, axis_n);
  if (nc > 0 && (!b_e || !a_e || !b_m || !a_m)) return fail(FDTD_ERR_BADARG, "face %d: missing b/a profile", f);
  const bool table = c->prec == FDTD_PREC_F32_TABLE;
  if (table && nc > 0 && (!kappa_e || !kappa_m)) return fail(FDTD_ERR_BADARG, "face %d: material-table problems need kappa profiles", f);
  long long want[4];
  psi_sizes(c, f, nc, want);
  const double* cp[4] = {CPsi0, CPsi1, CPsi2, CPsi3};
  const long got[4] = {n0, n1, n2, n3};
  digest_vals(c, 3, {(double)f, (double)nc, (double)m_start, (double)e_start, (double)n0, (double)n1, (double)n2,
                     (double)n3});
  for (const double* prof : {b_e, a_e, b_m, a_m, kappa_e, kappa_m})
    if (prof && nc > 0) digest(c, 3, prof, (size_t)nc * sizeof(double));
  for (int s = 0; s < 4; s++)
    if (cp[s] && got[s] > 0) digest(c, 3, cp[s], (size_t)got[s] * sizeof(double));
  // FP64 coefficients built on the device and no CPsi given: CPsi and the
  // kappa division of the band are done here, on the device
  const bool dev = !table && c->coef_device && !CPsi0 && !CPsi1 && !CPsi2 && !CPsi3 && !n0 && !n1 && !n2 && !n3;
  if (dev && nc > 0) {
    if (!kappa_e || !kappa_m) return fail(FDTD_ERR_BADARG, "face %d: device-built coefficients need kappa profiles", f);
    if (c->kappa_done[f]) return fail(FDTD_ERR_STATE, "face %d: its band was already divided by kappa; rebuild the coefficients first", f);
    for (int q = 0; q < nc; q++)
      if (!(kappa_e[q] > 0) || !(kappa_m[q] > 0)) return fail(FDTD_ERR_BADARG, "face %d: kappa must be positive", f);
  }
  for (int s = 0; s < 4; s++) {
    if (table || dev) continue;  // CPsi comes from the coefficient tables, or is made on the device
    if (got[s] != want[s] || (want[s] > 0 && !cp[s]))
      return fail(FDTD_ERR_BADARG, "face %d slot %d: got %ld CPsi values, expected %lld", f, s, got[s], want[s]);
  }
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  HostFace& h = c->face[f];
  dfree(c, h.block);
  h = HostFace();
  h.present = nc > 0;
  h.nc = nc; h.m_start = m_start; h.e_start = e_start;
  invalidate(c);
  if (nc == 0) return FDTD_OK;
  const double* pr[4] = {b_e, a_e, b_m, a_m};
  Arena ar;
  for (int s = 0; s < 4; s++) {
    h.n[s] = want[s];
    ar.add(&h.prof[s], nc * c->esz);
    ar.add(&h.psi[s], want[s] * c->esz);
    if (!table) ar.add(&h.cpsi[s], want[s] * c->esz);
  }
  for (int s = 0; s < 2 && table; s++) ar.add(&h.inv_k[s], nc * sizeof(float));
  int rc = dalloc(c, &h.block, ar.size);
  if (!rc) ar.place(h.block);
  for (int s = 0; s < 4 && !rc; s++) rc = upload_real(c, h.prof[s], pr[s], nc);
  for (int s = 0; s < 4 && !rc && !table && !dev; s++) rc = upload_real(c, h.cpsi[s], cp[s], want[s]);
  if (!rc && dev) rc = cpml_band_on_device(c, f, kappa_e, kappa_m);
  if (!rc && table) {
    std::vector<float> ik(nc);
    const double* kp[2] = {kappa_e, kappa_m};
    for (int s = 0; s < 2 && !rc; s++) {
      for (int q = 0; q < nc; q++) {
        if (!(kp[s][q] > 0)) return fail(FDTD_ERR_BADARG, "face %d: kappa must be positive", f);
        ik[q] = (float)(1.0 / kp[s][q]);
      }
      if (xfer(c, h.inv_k[s], ik.data(), nc * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess)
        rc = fail(FDTD_ERR_CUDA, "kappa upload failed");
    }
  }
  if (rc) h.present = false;
  return rc;
}

int fdtd_ctx_add_vsource(fdtd_ctx* c, int dir, const int* idx, const double* coef, int count, const double* wave,
                         int nSteps) {
  if (!c || !idx || !coef || !wave) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (dir < 0 || dir > 2) return fail(FDTD_ERR_BADARG, "source direction %d not in 0..2", dir);
  if (count <= 0) return fail(FDTD_ERR_BADARG, "source has no cells");
  if (nSteps < c->nsteps) return fail(FDTD_ERR_BADARG, "waveform has %d values, need %d", nSteps, c->nsteps);
  if ((int)c->src.size() >= kMaxSources) return fail(FDTD_ERR_BADARG, "at most %d sources", kMaxSources);
  digest_vals(c, 4, {(double)dir, (double)count});
  digest(c, 4, idx, (size_t)count * sizeof(int));
  digest(c, 4, coef, (size_t)count * sizeof(double));
  digest(c, 4, wave, (size_t)c->nsteps * sizeof(double));
  // component extents of E_dir
  const int ni = dir == 0 ? c->nx : c->nx + 1, nj = dir == 1 ? c->ny : c->ny + 1, nk = dir == 2 ? c->nz : c->nz + 1;
  const long long n = (long long)ni * nj * nk;
  int bi0 = 1 << 30, bi1 = -1, bj0 = 1 << 30, bj1 = -1, bk0 = 1 << 30, bk1 = -1;
  for (int q = 0; q < count; q++) {
    if (idx[q] < 0 || idx[q] >= n) return fail(FDTD_ERR_BADARG, "source index %d out of range", idx[q]);
    const int i = idx[q] / (nj * nk), j = (idx[q] / nk) % nj, k = idx[q] % nk;
    bi0 = std::min(bi0, i); bi1 = std::max(bi1, i);
    bj0 = std::min(bj0, j); bj1 = std::max(bj1, j);
    bk0 = std::min(bk0, k); bk1 = std::max(bk1, k);
  }
  // the list must be the box in createLinearIndexList order (grid.js:228-243)
  const long long bn = (long long)(bi1 - bi0 + 1) * (bj1 - bj0 + 1) * (bk1 - bk0 + 1);
  if (bn != count) return fail(FDTD_ERR_BADARG, "source cells do not form a box");
  int q = 0;
  for (int k = bk0; k <= bk1; k++)
    for (int j = bj0; j <= bj1; j++)
      for (int i = bi0; i <= bi1; i++, q++)
        if (idx[q] != (i * nj + j) * nk + k) return fail(FDTD_ERR_BADARG, "source cells not in k-j-i box order");
  for (int q2 = 0; q2 < count; q2++)
    if (!std::isfinite(coef[q2])) return fail(FDTD_ERR_BADARG, "non-finite source coefficient");
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  HostSource s;
  s.box = SourceBox{dir, bi0, bi1, bj0, bj1, bk0, bk1};
  s.count = count;
  int rc = dalloc(c, &s.cs, count * c->esz);
  if (!rc) rc = upload_real(c, s.cs, coef, count);
  if (!rc) rc = dalloc(c, &s.wave, (size_t)c->nsteps * c->esz);
  if (!rc) rc = upload_real(c, s.wave, wave, c->nsteps);
  if (rc) return rc;
  c->src.push_back(s);
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_add_svoltage(fdtd_ctx* c, int dir, const int* idx, int count, double Csvf) {
  if (!c || !idx) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (dir < 0 || dir > 2) return fail(FDTD_ERR_BADARG, "probe direction %d not in 0..2", dir);
  if (count <= 0) return fail(FDTD_ERR_BADARG, "probe has no cells");
  if ((int)c->vprobe.size() >= kMaxProbes) return fail(FDTD_ERR_BADARG, "at most %d voltage probes", kMaxProbes);
  const long long n = c->ncomp[3 + dir];
  for (int q = 0; q < count; q++)
    if (idx[q] < 0 || idx[q] >= n) return fail(FDTD_ERR_BADARG, "probe index %d out of range", idx[q]);
  digest_vals(c, 5, {(double)dir, (double)count, Csvf});
  digest(c, 5, idx, (size_t)count * sizeof(int));
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  HostVProbe p{dir, count, nullptr, Csvf, std::vector<int>(idx, idx + count)};
  int rc = dalloc(c, (void**)&p.idx, count * sizeof(int));
  if (rc) return rc;
  CK(xfer(c, p.idx, idx, count * sizeof(int), cudaMemcpyHostToDevice));
  c->vprobe.push_back(p);
  invalidate(c);
  return ensure_traces(c);
}

int fdtd_ctx_add_scurrent(fdtd_ctx* c, const int* comp, const int* idx, const double* w, int count) {
  if (!c || !comp || !idx || !w) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (count <= 0) return fail(FDTD_ERR_BADARG, "probe has no samples");
  if ((int)c->iprobe.size() >= kMaxProbes) return fail(FDTD_ERR_BADARG, "at most %d current probes", kMaxProbes);
  for (int q = 0; q < count; q++) {
    if (comp[q] < 0 || comp[q] > 2) return fail(FDTD_ERR_BADARG, "current probe component %d not in 0..2", comp[q]);
    if (idx[q] < 0 || idx[q] >= c->ncomp[comp[q]]) return fail(FDTD_ERR_BADARG, "current probe index %d out of range", idx[q]);
  }
  digest_vals(c, 6, {(double)count});
  digest(c, 6, comp, (size_t)count * sizeof(int));
  digest(c, 6, idx, (size_t)count * sizeof(int));
  digest(c, 6, w, (size_t)count * sizeof(double));
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  HostIProbe p{count, nullptr, nullptr, nullptr, std::vector<int>(comp, comp + count),
               std::vector<int>(idx, idx + count)};
  int rc = dalloc(c, (void**)&p.comp, count * sizeof(int));
  if (!rc) rc = dalloc(c, (void**)&p.idx, count * sizeof(int));
  if (!rc) rc = dalloc(c, (void**)&p.w, count * sizeof(double));
  if (rc) return rc;
  CK(xfer(c, p.comp, comp, count * sizeof(int), cudaMemcpyHostToDevice));
  CK(xfer(c, p.idx, idx, count * sizeof(int), cudaMemcpyHostToDevice));
  CK(xfer(c, p.w, w, count * sizeof(double), cudaMemcpyHostToDevice));
  c->iprobe.push_back(p);
  invalidate(c);
  return ensure_traces(c);
}

int fdtd_ctx_setup_farfield(fdtd_ctx* c, int nFreq, const double* freqs, int li, int lj, int lk, int ui, int uj,
                            int uk) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (nFreq < 0 || (nFreq > 0 && !freqs)) return fail(FDTD_ERR_BADARG, "bad frequency list");
  if (c->nFreq > 0) return fail(FDTD_ERR_STATE, "far field already set up");
  if (nFreq == 0) return FDTD_OK;
  // the 4-point averages reach one cell outside the box on each side
  if (li < 2 || lj < 2 || lk < 2 || ui > c->nx || uj > c->ny || uk > c->nz || ui <= li || uj <= lj || uk <= lk)
    return fail(FDTD_ERR_BADARG, "Huygens box [%d,%d]x[%d,%d]x[%d,%d] does not fit the grid", li, ui, lj, uj, lk, uk);
  digest_vals(c, 7, {(double)nFreq, (double)li, (double)lj, (double)lk, (double)ui, (double)uj, (double)uk});
  digest(c, 7, freqs, (size_t)nFreq * sizeof(double));
  CK(cudaSetDevice(c->device));
  c->nFreq = nFreq;
  c->ffreq.assign(freqs, freqs + nFreq);
  c->li = li; c->lj = lj; c->lk = lk; c->ui = ui; c->uj = uj; c->uk = uk;
  const long long ni = ui - li, nj = uj - lj, nk = uk - lk;
  c->ffsz[0] = nj * nk;
  c->ffsz[1] = ni * nk;
  c->ffsz[2] = ni * nj;
  long long off = 0;
  for (int a = 0; a < 24; a++) {
    c->ffoff[a] = off;
    off += 2 * nFreq * c->ffsz[(a % 12) / 4];
  }
  int rc = dalloc(c, (void**)&c->acc, off * sizeof(double));
  if (rc) return rc;
  // phasors, evaluated as farfield.js:101-110 does
  std::vector<double> ph((size_t)c->nsteps * nFreq * 4);
  for (int ts = 0; ts < c->nsteps; ts++)
    for (int m = 0; m < nFreq; m++) {
      const double w = 2 * M_PI * freqs[m];
      const double wdt = w * c->dt;
      const double phh = wdt * (ts + 0.5), phe = wdt * (ts + 1);
      double* q = &ph[((size_t)ts * nFreq + m) * 4];
      q[0] = std::cos(phh);
      q[1] = -std::sin(phh);
      q[2] = std::cos(phe);
      q[3] = -std::sin(phe);
    }
  rc = dalloc(c, (void**)&c->ph, ph.size() * sizeof(double));
  if (rc) return rc;
  CK(xfer(c, c->ph, ph.data(), ph.size() * sizeof(double), cudaMemcpyHostToDevice));
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_upload_material(fdtd_ctx* c, int comp, const unsigned char* ids, long n, const double* table, int rows) {
  if (!c || !ids || !table) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (c->prec != FDTD_PREC_F32_TABLE) return fail(FDTD_ERR_STATE, "not a material-table problem");
  if (comp < 0 || comp > 5) return fail(FDTD_ERR_BADARG, "component %d not in 0..5", comp);
  const long long want = c->ncomp[(comp + 3) % 6];
  if (n != want) return fail(FDTD_ERR_BADARG, "component %d: got %ld ids, expected %lld", comp, n, want);
  if (rows < 1 || rows > kTableRows) return fail(FDTD_ERR_BADARG, "table rows %d not in 1..%d", rows, kTableRows);
  for (long q = 0; q < n; q++)
    if (ids[q] >= rows) return fail(FDTD_ERR_BADARG, "material id %d >= table rows %d", ids[q], rows);
  digest_vals(c, 8, {(double)comp, (double)rows});
  digest(c, 8, ids, (size_t)n);
  digest(c, 8, table, (size_t)rows * 3 * sizeof(double));
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  CK(xfer(c, c->ids[comp], ids, n, cudaMemcpyHostToDevice));
  int rc = set_rows(c, comp, std::vector<double>(table, table + 3 * rows));
  if (rc) return rc;
  c->ids_set[comp] = true;
  invalidate(c);
  return FDTD_OK;
}

// Coefficient triple (self, curl1, curl2) of a component for an averaged
// material pair, as coefficients.js:22-116 evaluates it (no kappa).
static void coef_row(const fdtd_ctx* c, int comp, double e, double s, double out[3]) {
  const double dt = c->dt;
  const double tdx = 2 * dt / c->dx, tdy = 2 * dt / c->dy, tdz = 2 * dt / c->dz;
  const double scale = comp < 3 ? 8.854187817e-12 : 4 * M_PI * 1e-7;
  const double a = 2 * e * scale;
  const double b = dt * s;
  const double denom = a + b;
  // curl numerators (coefficients.js:32-106): Ex tdy,-tdz | Ey tdz,-tdx | Ez tdx,-tdy |
  // Hx tdz,-tdy | Hy tdx,-tdz | Hz tdy,-tdx
  static const int sel1[6] = {1, 2, 0, 2, 0, 1}, sel2[6] = {2, 0, 1, 1, 2, 0};
  const double t[3] = {tdx, tdy, tdz};
  const double n1 = t[sel1[comp]];
  const double n2 = -t[sel2[comp]];
  out[0] = (a - b) / denom;
  out[1] = n1 / denom;
  out[2] = n2 / denom;
}

static int set_rows(fdtd_ctx* c, int comp, const std::vector<double>& rows) {
  const int nrows = (int)rows.size() / 3;
  if (nrows > kTableRows) return fail(FDTD_ERR_BADARG, "component %d needs %d coefficient rows (limit %d)", comp, nrows, kTableRows);
  c->rows64[comp] = rows;
  c->table[comp].assign(3 * kTableRows, 0.f);
  for (size_t r = 0; r < rows.size(); r++) c->table[comp][r] = (float)rows[r];
  return FDTD_OK;
}

int fdtd_ctx_build_material(fdtd_ctx* c, const unsigned char* mat, long ncells, int ntypes, const double* props,
                            int nplates, const int* plates, const double* plate_sigma) {
  if (!c || !mat || !props || (nplates > 0 && (!plates || !plate_sigma))) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (c->prec == FDTD_PREC_F32)
    return fail(FDTD_ERR_STATE, "per-cell FP32 problems take fdtd_ctx_upload_coeff (FP64 and material-table problems build here)");
  const bool f64 = c->prec == FDTD_PREC_F64;
  if (ncells != (long)c->nx * c->ny * c->nz) return fail(FDTD_ERR_BADARG, "material grid of %ld cells, need %lld", ncells, (long long)c->nx * c->ny * c->nz);
  if (ntypes < 1 || ntypes > 48) return fail(FDTD_ERR_BADARG, "%d material slots (1..48 supported)", ntypes);
  if (nplates < 0 || nplates > kMaxPlates) return fail(FDTD_ERR_BADARG, "%d plates (at most %d)", nplates, kMaxPlates);
  unsigned char mmax = 0;
  for (long q = 0; q < ncells; q++) mmax = std::max(mmax, mat[q]);
  if (mmax >= ntypes) return fail(FDTD_ERR_BADARG, "material id %d has no properties", mmax);
  digest_vals(c, 9, {(double)ncells, (double)ntypes, (double)nplates});
  digest(c, 9, mat, (size_t)ncells);
  digest(c, 9, props, (size_t)ntypes * 4 * sizeof(double));
  if (nplates > 0) {
    digest(c, 9, plates, (size_t)nplates * 7 * sizeof(int));
    digest(c, 9, plate_sigma, (size_t)nplates * sizeof(double));
  }
  MatBuild b{};
  b.nx = c->nx; b.ny = c->ny; b.nz = c->nz; b.M = ntypes; b.nplates = nplates;
  std::vector<double> psig;  // distinct plate conductivities
  const int ext[3][3] = {{c->nx, c->ny + 1, c->nz + 1}, {c->nx + 1, c->ny, c->nz + 1}, {c->nx + 1, c->ny + 1, c->nz}};
  for (int q = 0; q < nplates; q++) {
    const int* P = plates + 7 * q;
    if (P[0] < 0 || P[0] > 2) return fail(FDTD_ERR_BADARG, "plate %d: component %d not in 0..2", q, P[0]);
    const int* e = ext[P[0]];
    if (P[1] < 0 || P[2] >= e[0] || P[3] < 0 || P[4] >= e[1] || P[5] < 0 || P[6] >= e[2] || P[1] > P[2] || P[3] > P[4] || P[5] > P[6])
      return fail(FDTD_ERR_BADARG, "plate %d: box outside its component array", q);
    int sid = -1;
    for (size_t u = 0; u < psig.size(); u++)
      if (psig[u] == plate_sigma[q]) sid = (int)u;
    if (sid < 0) { sid = (int)psig.size(); psig.push_back(plate_sigma[q]); }
    b.plate[q] = PlateBox{P[0], P[1], P[2], P[3], P[4], P[5], P[6], sid};
  }
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  unsigned char* d_mat = nullptr;
  uint8_t *d_present = nullptr, *d_map = nullptr;
  int* d_map64 = nullptr;     // FP64: code -> row
  double* d_rows = nullptr;   // FP64: row triples
  const long long M = ntypes;
  const long long ncode_e = (M * M * M * M + 1) * (long long)(psig.size() + 1);
  const long long ncode_h = M * M + 1;
  int rc = FDTD_OK;
  if (dev_malloc(c, &d_mat, ncells) != cudaSuccess ||
      dev_malloc(c, &d_present, std::max(ncode_e, ncode_h)) != cudaSuccess ||
      dev_malloc(c, &d_map, std::max(ncode_e, ncode_h)) != cudaSuccess ||
      (f64 && dev_malloc(c, &d_map64, std::max(ncode_e, ncode_h) * sizeof(int)) != cudaSuccess)) {
    rc = fail(FDTD_ERR_OOM, "material build buffers");
  }
  if (!rc && xfer(c, d_mat, mat, ncells, cudaMemcpyHostToDevice) != cudaSuccess) rc = fail(FDTD_ERR_CUDA, "material grid upload");
  b.mat = d_mat;
  const double* t_eps = props;  // props rows: eps_r, mu_r, sigma_e, sigma_m per type id
  std::vector<uint8_t> present, map;
  for (int comp = 0; comp < 6 && !rc; comp++) {
    const long long ncode = comp < 3 ? ncode_e : ncode_h;
    present.assign(ncode, 0);
    if (cudaMemsetAsync(d_present, 0, ncode, c->stream) != cudaSuccess) { rc = fail(FDTD_ERR_CUDA, "memset"); break; }
    k_material_mark<<<148 * 8, 256, 0, c->stream>>>(b, comp, d_present);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess ||
        xfer(c, present.data(), d_present, ncode, cudaMemcpyDeviceToHost) != cudaSuccess) {
      rc = fail(FDTD_ERR_CUDA, "material mark: %s", cudaGetErrorString(cudaGetLastError()));
      break;
    }
    std::map<std::pair<double, double>, int> rowof;
    std::vector<double> rows;
    std::vector<int> row_of_code(f64 ? ncode : 0, 0);
    map.assign(ncode, 0);
    const long long fill = comp < 3 ? M * M * M * M : M * M;
    for (long long code = 0; code < ncode; code++) {
      if (!present[code]) continue;
      double e, s;
      if (comp < 3) {
        const long long base = code % (fill + 1), sid = code / (fill + 1) - 1;
        if (base == fill) {
          e = 1.0; s = 0.0;
        } else {
          const long long m1 = base % M, m2 = (base / M) % M, m3 = (base / (M * M)) % M, m4 = base / (M * M * M);
          e = 0.25 * (t_eps[4 * m1] + t_eps[4 * m2] + t_eps[4 * m3] + t_eps[4 * m4]);
          s = 0.25 * (props[4 * m1 + 2] + props[4 * m2 + 2] + props[4 * m3 + 2] + props[4 * m4 + 2]);
        }
        if (sid >= 0) s = psig[sid];
      } else if (code == fill) {
        e = 1.0; s = 0.0;
      } else {
        const long long m1 = code % M, m2 = code / M;
        const double mu1 = props[4 * m1 + 1], mu2 = props[4 * m2 + 1];
        e = 2 * mu1 * mu2 / (mu1 + mu2);
        const double sm1 = props[4 * m1 + 3], sm2 = props[4 * m2 + 3];
        s = 2 * sm1 * sm2 / (sm1 + sm2);
      }
      auto key = std::make_pair(e, s);
      auto it = rowof.find(key);
      int r;
      if (it == rowof.end()) {
        r = (int)rows.size() / 3;
        rowof[key] = r;
        double tr[3];
        coef_row(c, comp, e, s, tr);
        rows.insert(rows.end(), tr, tr + 3);
      } else {
        r = it->second;
      }
      map[code] = (uint8_t)std::min(r, 255);
      if (f64) row_of_code[code] = r;
    }
    if (f64) {
      // every cell takes its row's FP64 triple: coefficient arrays 3 comp .. 3 comp + 2
      const std::vector<int>& map64 = row_of_code;
      cudaFree(d_rows);
      d_rows = nullptr;
      if (dev_malloc(c, &d_rows, std::max<size_t>(rows.size(), 1) * sizeof(double)) != cudaSuccess) {
        rc = fail(FDTD_ERR_OOM, "coefficient rows");
        break;
      }
      if (xfer(c, d_rows, rows.data(), rows.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
          xfer(c, d_map64, map64.data(), ncode * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) {
        rc = fail(FDTD_ERR_CUDA, "coefficient row upload");
        break;
      }
      k_material_coef<<<148 * 8, 256, 0, c->stream>>>(b, comp, d_map64, d_rows, (double*)c->coef[3 * comp],
                                                      (double*)c->coef[3 * comp + 1], (double*)c->coef[3 * comp + 2]);
      if (cudaStreamSynchronize(c->stream) != cudaSuccess) { rc = fail(FDTD_ERR_CUDA, "coefficients: %s", cudaGetErrorString(cudaGetLastError())); break; }
      for (int w = 0; w < 3; w++) c->coef_set[3 * comp + w] = true;
      continue;
    }
    rc = set_rows(c, comp, rows);
    if (rc) break;
    if (xfer(c, d_map, map.data(), ncode, cudaMemcpyHostToDevice) != cudaSuccess) { rc = fail(FDTD_ERR_CUDA, "code map upload"); break; }
    k_material_ids<<<148 * 8, 256, 0, c->stream>>>(b, comp, d_map, c->ids[comp]);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess) { rc = fail(FDTD_ERR_CUDA, "material ids: %s", cudaGetErrorString(cudaGetLastError())); break; }
    c->ids_set[comp] = true;
  }
  cudaFree(d_mat);
  cudaFree(d_present);
  cudaFree(d_map);
  cudaFree(d_map64);
  cudaFree(d_rows);
  if (f64) {
    c->coef_device = rc == FDTD_OK;
    for (int f = 0; f < 6; f++) c->kappa_done[f] = false;
  }
  invalidate(c);
  return rc;
}

// FP64 problems: the triples overwrite coefficient arrays 3 comp .. 3 comp + 2 at the cells.
static int override_coef64(fdtd_ctx* c, int comp, const int* idx, const double* triples, int count) {
  if (comp < 0 || comp > 5) return fail(FDTD_ERR_BADARG, "component %d not in 0..5", comp);
  for (int w = 0; w < 3; w++)
    if (!c->coef_set[3 * comp + w]) return fail(FDTD_ERR_STATE, "component %d has no coefficients yet", comp);
  if (count <= 0) return FDTD_OK;
  const long long n = coef_count(c, 3 * comp);
  for (int q = 0; q < count; q++) {
    if (idx[q] < 0 || idx[q] >= n) return fail(FDTD_ERR_BADARG, "cell index %d out of range", idx[q]);
    for (int w = 0; w < 3; w++)
      if (!std::isfinite(triples[3 * q + w])) return fail(FDTD_ERR_BADARG, "non-finite coefficient");
  }
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  int* d_idx = nullptr;
  double* d_trip = nullptr;
  int rc = FDTD_OK;
  if (dev_malloc(c, &d_idx, count * sizeof(int)) != cudaSuccess ||
      dev_malloc(c, &d_trip, 3 * count * sizeof(double)) != cudaSuccess)
    rc = fail(FDTD_ERR_OOM, "override buffers");
  if (!rc && (xfer(c, d_idx, idx, count * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess ||
              xfer(c, d_trip, triples, 3 * count * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess))
    rc = fail(FDTD_ERR_CUDA, "override upload");
  if (!rc) {
    k_coef_override<<<1, 1, 0, c->stream>>>((double*)c->coef[3 * comp], (double*)c->coef[3 * comp + 1],
                                            (double*)c->coef[3 * comp + 2], d_idx, d_trip, count);
    if (cudaStreamSynchronize(c->stream) != cudaSuccess)
      rc = fail(FDTD_ERR_CUDA, "override: %s", cudaGetErrorString(cudaGetLastError()));
  }
  cudaFree(d_idx);
  cudaFree(d_trip);
  invalidate(c);
  return rc;
}

int fdtd_ctx_override_material(fdtd_ctx* c, int comp, const int* idx, const double* triples, int count) {
  if (!c || !idx || !triples) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  if (count > 0) {
    digest_vals(c, 10, {(double)comp, (double)count});
    digest(c, 10, idx, (size_t)count * sizeof(int));
    digest(c, 10, triples, (size_t)count * 3 * sizeof(double));
  }
  if (c->prec == FDTD_PREC_F64) return override_coef64(c, comp, idx, triples, count);
  if (c->prec != FDTD_PREC_F32_TABLE) return fail(FDTD_ERR_STATE, "not a material-table or FP64 problem");
  if (comp < 0 || comp > 5 || !c->ids_set[comp]) return fail(FDTD_ERR_STATE, "component %d has no material ids yet", comp);
  const long long n = c->ncomp[(comp + 3) % 6];
  std::vector<double> rows = c->rows64[comp];
  CK(cudaSetDevice(c->device));
  if (int rc0 = fused_drop(c)) return rc0;
  for (int q = 0; q < count; q++) {
    if (idx[q] < 0 || idx[q] >= n) return fail(FDTD_ERR_BADARG, "cell index %d out of range", idx[q]);
    int r = -1;
    for (size_t u = 0; u + 2 < rows.size(); u += 3)
      if (rows[u] == triples[3 * q] && rows[u + 1] == triples[3 * q + 1] && rows[u + 2] == triples[3 * q + 2]) r = (int)u / 3;
    if (r < 0) {
      r = (int)rows.size() / 3;
      rows.insert(rows.end(), triples + 3 * q, triples + 3 * q + 3);
    }
    if (r >= kTableRows) return fail(FDTD_ERR_BADARG, "component %d: coefficient rows exceed %d", comp, kTableRows);
    const uint8_t id = (uint8_t)r;
    CK(xfer(c, c->ids[comp] + idx[q], &id, 1, cudaMemcpyHostToDevice));
  }
  int rc = set_rows(c, comp, rows);
  invalidate(c);
  return rc;
}

int fdtd_ctx_read_material(fdtd_ctx* c, int comp, unsigned char* ids, long n, double* table, int* rows) {
  if (!c || !ids || !table || !rows) return fail(FDTD_ERR_BADARG, "NULL argument");
  if (c->prec != FDTD_PREC_F32_TABLE || comp < 0 || comp > 5 || !c->ids_set[comp]) return fail(FDTD_ERR_STATE, "no material ids for component %d", comp);
  if (n != c->ncomp[(comp + 3) % 6]) return fail(FDTD_ERR_BADARG, "id buffer of %ld, need %lld", n, c->ncomp[(comp + 3) % 6]);
  CK(cudaSetDevice(c->device));
  CK(xfer(c, ids, c->ids[comp], n, cudaMemcpyDeviceToHost));
  *rows = (int)c->rows64[comp].size() / 3;
  std::copy(c->rows64[comp].begin(), c->rows64[comp].end(), table);
  return FDTD_OK;
}

int fdtd_ctx_run(fdtd_ctx* c, int count) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  return run_steps(c, count);
}

int fdtd_ctx_set_prefetch(fdtd_ctx* c, int planes) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (planes < 1 || planes > 5) return fail(FDTD_ERR_BADARG, "prefetch depth %d not in 1..5", planes);
  if (planes > 2 && c->prec != FDTD_PREC_F32_TABLE)
    return fail(FDTD_ERR_BADARG, "prefetch modes 3..5 (shared-memory stages) need a material-table problem");
  c->prefetch = planes;
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_set_tiling(fdtd_ctx* c, int x_planes_per_thread, int block_rows) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (x_planes_per_thread < 1 || x_planes_per_thread > c->nx + 1)
    return fail(FDTD_ERR_BADARG, "x planes per thread %d not in 1..%d", x_planes_per_thread, c->nx + 1);
  if (block_rows != 1 && block_rows != 2 && block_rows != 4 && block_rows != 8 && block_rows != 16)
    return fail(FDTD_ERR_BADARG, "block rows %d not in {1,2,4,8,16}", block_rows);
  c->ichunk = x_planes_per_thread;
  c->block_rows = block_rows;
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_set_block_width(fdtd_ctx* c, int threads_along_k) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (threads_along_k != 16 && threads_along_k != 32)
    return fail(FDTD_ERR_BADARG, "block width %d not 16 or 32", threads_along_k);
  c->block_w = threads_along_k;
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_get_block_width(const fdtd_ctx* c, int* threads_along_k) {
  if (!c || !threads_along_k) return fail(FDTD_ERR_BADARG, "NULL argument");
  *threads_along_k = c->block_w;
  return FDTD_OK;
}

int fdtd_ctx_get_tiling(const fdtd_ctx* c, int* x_planes_per_thread, int* block_rows) {
  if (!c || !x_planes_per_thread || !block_rows) return fail(FDTD_ERR_BADARG, "NULL argument");
  *x_planes_per_thread = c->ichunk;
  *block_rows = c->block_rows;
  return FDTD_OK;
}

int fdtd_ctx_run_timed(fdtd_ctx* c, int count, float* ms) {
  if (!c || !ms) return fail(FDTD_ERR_BADARG, "NULL argument");
  return run_steps(c, count, ms);
}

int fdtd_ctx_profile_kernels(fdtd_ctx* c, int count, double* avg_ms) {
  if (!c || !avg_ms || count < 1) return fail(FDTD_ERR_BADARG, "bad arguments");
  KernelTimer tm;
  CK(cudaSetDevice(c->device));
  for (int q = 0; q < 5; q++) CK(cudaEventCreate(&tm.ev[q]));
  int rc = run_steps(c, count, nullptr, &tm);
  for (int q = 0; q < 5; q++) cudaEventDestroy(tm.ev[q]);
  if (rc) return rc;
  for (int q = 0; q < 4; q++) avg_ms[q] = tm.ms[q] / count;
  return FDTD_OK;
}

int fdtd_ctx_step(const fdtd_ctx* c) { return c ? c->ts : -1; }

int fdtd_status(fdtd_ctx* c, int* code, int* step) {
  if (!c || !code || !step) return fail(FDTD_ERR_BADARG, "NULL argument");
  int st[2];
  CK(cudaSetDevice(c->device));
  CK(xfer(c, st, c->d_status, sizeof(st), cudaMemcpyDeviceToHost));
  *code = st[0];
  *step = st[0] ? st[1] : -1;
  return FDTD_OK;
}

int fdtd_ctx_read_trace(fdtd_ctx* c, int kind, int probe, double* out, int n) {
  if (!c || !out) return fail(FDTD_ERR_BADARG, "NULL argument");
  const int np = kind == 0 ? (int)c->vprobe.size() : (int)c->iprobe.size();
  if (kind < 0 || kind > 1 || probe < 0 || probe >= np) return fail(FDTD_ERR_BADARG, "no probe %d of kind %d", probe, kind);
  if (n < 0 || n > c->nsteps) return fail(FDTD_ERR_BADARG, "bad length %d", n);
  CK(cudaSetDevice(c->device));
  const double* src = (kind == 0 ? c->V : c->I) + (size_t)probe * c->nsteps;
  CK(xfer(c, out, src, n * sizeof(double), cudaMemcpyDeviceToHost));
  return FDTD_OK;
}

int fdtd_ctx_read_field(fdtd_ctx* c, int which, double* host, long n) {
  if (!c || !host) return fail(FDTD_ERR_BADARG, "NULL argument");
  if (which < 0 || which > 5) return fail(FDTD_ERR_BADARG, "field id %d not in 0..5", which);
  if (n != c->ncomp[which]) return fail(FDTD_ERR_BADARG, "field %d: buffer of %ld, need %lld", which, n, c->ncomp[which]);
  CK(cudaSetDevice(c->device));
  Using use(c->mu);
  if (!c->dense_valid)  // this array alone
    if (int rc = c->esz == 8 ? fused_copy_field<double>(c, which, 0) : fused_copy_field<float>(c, which, 0)) return rc;
  return read_real(c, field_ptr(c, which), host, n);
}

int fdtd_ctx_read_psi(fdtd_ctx* c, int f, int slot, double* host, long n) {
  if (!c || !host) return fail(FDTD_ERR_BADARG, "NULL argument");
  if (f < 0 || f > 5 || slot < 0 || slot > 3 || !c->face[f].present) return fail(FDTD_ERR_BADARG, "no Psi slot %d on face %d", slot, f);
  if (n != c->face[f].n[slot]) return fail(FDTD_ERR_BADARG, "Psi buffer of %ld, need %lld", n, c->face[f].n[slot]);
  CK(cudaSetDevice(c->device));
  Using use(c->mu);
  if (!c->dense_valid)
    if (int rc = c->esz == 8 ? fused_copy_psi<double>(c, f, slot, 0) : fused_copy_psi<float>(c, f, slot, 0)) return rc;
  return read_real(c, c->face[f].psi[slot], host, n);
}

int fdtd_ctx_read_farfield(fdtd_ctx* c, int array, double* re, double* im, long n) {
  if (!c || !re || !im) return fail(FDTD_ERR_BADARG, "NULL argument");
  if (c->nFreq == 0) return fail(FDTD_ERR_STATE, "no far field set up");
  if (array < 0 || array > 23) return fail(FDTD_ERR_BADARG, "array %d not in 0..23", array);
  const long long m = c->nFreq * c->ffsz[(array % 12) / 4];
  if (n != m) return fail(FDTD_ERR_BADARG, "far-field buffer of %ld, need %lld", n, m);
  CK(cudaSetDevice(c->device));
  CK(xfer(c, re, c->acc + c->ffoff[array], m * sizeof(double), cudaMemcpyDeviceToHost));
  CK(xfer(c, im, c->acc + c->ffoff[array] + m, m * sizeof(double), cudaMemcpyDeviceToHost));
  if (c->acc_kahan) {
    // each 8-byte slot holds (sum, compensation) as two floats; the sum is sum - compensation
    for (double* a : {re, im})
      for (long long q = 0; q < m; q++) {
        float v[2];
        memcpy(v, &a[q], sizeof(v));
        a[q] = (double)v[0] - (double)v[1];
      }
  }
  return FDTD_OK;
}

// ---------------------------------------------------------------------------
// Checkpoint / restore of the evolving state: fields, Psi, port traces,
// far-field accumulators, watchdog and step.  The problem definition
// (coefficients, tables, sources, probes, boxes) is not part of it: a state
// loads into a handle set up with the same problem.
// ---------------------------------------------------------------------------
namespace {

struct StateHeader {
  char magic[8];  // "FDTDST2\0"
  int nx, ny, nz, prec, nsteps, ts, nv, ni, nfreq, kahan;
  long long psi[6][4];
  long long ff_values;
  unsigned long long setup;  // the handle's set-up digest
  long long bytes;  // whole state, header included
};

// The device ranges of a handle's state, in state order.
std::vector<std::pair<void*, size_t>> state_ranges(fdtd_ctx* c) {
  std::vector<std::pair<void*, size_t>> r;
  long long tot = 0;
  for (int q = 0; q < 6; q++) tot += c->ncomp[q];
  r.push_back({c->fields, (size_t)tot * c->esz});
  for (int f = 0; f < 6; f++)
    for (int s = 0; s < 4; s++)
      if (c->face[f].present && c->face[f].psi[s]) r.push_back({c->face[f].psi[s], (size_t)c->face[f].n[s] * c->esz});
  r.push_back({c->V, sizeof(double) * std::max((int)c->vprobe.size(), 1) * (size_t)c->nsteps});
  r.push_back({c->I, sizeof(double) * std::max((int)c->iprobe.size(), 1) * (size_t)c->nsteps});
  if (c->nFreq > 0) r.push_back({c->acc, sizeof(double) * (size_t)(c->ffoff[23] + 2LL * c->nFreq * c->ffsz[2])});
  r.push_back({c->d_status, 2 * sizeof(int)});
  return r;
}

StateHeader state_header(fdtd_ctx* c) {
  StateHeader h{};
  memcpy(h.magic, "FDTDST2", 8);
  h.nx = c->nx; h.ny = c->ny; h.nz = c->nz; h.prec = c->prec; h.nsteps = c->nsteps; h.ts = c->ts;
  h.nv = (int)c->vprobe.size(); h.ni = (int)c->iprobe.size(); h.nfreq = c->nFreq; h.kahan = c->acc_kahan;
  for (int f = 0; f < 6; f++)
    for (int s = 0; s < 4; s++) h.psi[f][s] = (c->face[f].present && c->face[f].psi[s]) ? c->face[f].n[s] : 0;
  h.ff_values = c->nFreq > 0 ? c->ffoff[23] + 2LL * c->nFreq * c->ffsz[2] : 0;
  h.setup = c->setup_digest;
  long long bytes = sizeof(StateHeader);
  for (auto& q : state_ranges(c)) bytes += (long long)q.second;
  h.bytes = bytes;
  return h;
}

}  // namespace

int fdtd_ctx_state_size(fdtd_ctx* c, long long* bytes) {
  if (!c || !bytes) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  int rc = ensure_traces(c);
  if (rc) return rc;
  *bytes = state_header(c).bytes;
  return FDTD_OK;
}

int fdtd_ctx_save_state(fdtd_ctx* c, void* buf, long long bytes) {
  if (!c || !buf) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  CK(cudaSetDevice(c->device));
  int rc = ensure_traces(c);
  if (rc) return rc;
  const StateHeader h = state_header(c);
  if (bytes != h.bytes) return fail(FDTD_ERR_BADARG, "state buffer of %lld bytes, need %lld", bytes, h.bytes);
  rc = to_dense(c);
  if (rc) return rc;
  char* p = (char*)buf;
  memcpy(p, &h, sizeof(h));
  p += sizeof(h);
  for (auto& q : state_ranges(c)) {
    CK(cudaMemcpyAsync(p, q.first, q.second, cudaMemcpyDeviceToHost, c->stream));
    p += q.second;
  }
  CK(cudaStreamSynchronize(c->stream));
  return FDTD_OK;
}

int fdtd_ctx_load_state(fdtd_ctx* c, const void* buf, long long bytes) {
  if (!c || !buf) return fail(FDTD_ERR_BADARG, "NULL argument");
  Using use(c->mu);
  CK(cudaSetDevice(c->device));
  int rc = ensure_traces(c);
  if (rc) return rc;
  StateHeader mine = state_header(c), theirs;
  if (bytes < (long long)sizeof(StateHeader)) return fail(FDTD_ERR_BADARG, "state buffer too small");
  memcpy(&theirs, buf, sizeof(theirs));
  if (memcmp(theirs.magic, "FDTDST2", 8) != 0) return fail(FDTD_ERR_BADARG, "not an engine state");
  mine.ts = theirs.ts;  // the step is what loading changes
  if (theirs.setup != mine.setup)
    return fail(FDTD_ERR_BADARG, "state was saved from a handle set up with other data (grid, dt, coefficients, "
                                 "faces, sources, probes or far field)");
  if (memcmp(&mine, &theirs, sizeof(StateHeader)) != 0 || bytes != theirs.bytes)
    return fail(FDTD_ERR_BADARG, "state was saved from a problem of another shape, precision or probe set");
  if (theirs.ts < 0 || theirs.ts > c->nsteps) return fail(FDTD_ERR_BADARG, "state step %d out of range", theirs.ts);
  const char* p = (const char*)buf + sizeof(StateHeader);
  c->dense_valid = true;   // every value of the state is replaced
  c->fs.valid = false;
  for (auto& q : state_ranges(c)) {
    CK(cudaMemcpyAsync(q.first, p, q.second, cudaMemcpyHostToDevice, c->stream));
    p += q.second;
  }
  const int dts = theirs.ts - 1;  // the device counter holds the index of the last step run
  CK(cudaMemcpyAsync(c->d_ts, &dts, sizeof(int), cudaMemcpyHostToDevice, c->stream));
  if (c->d_dft_done)  // a saved state has no open DFT block
    CK(cudaMemcpyAsync(c->d_dft_done, &theirs.ts, sizeof(int), cudaMemcpyHostToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  c->ts = theirs.ts;
  return FDTD_OK;
}

int fdtd_ctx_set_dft_block(fdtd_ctx* c, int steps) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (steps < 0 || steps == 1 || steps > 1024) return fail(FDTD_ERR_BADARG, "DFT block of %d steps not in {0, 2..1024}", steps);
  if (steps && c->prec == FDTD_PREC_F64) return fail(FDTD_ERR_BADARG, "FP64 problems keep the per-step DFT");
  if (steps && c->nFreq == 0) return fail(FDTD_ERR_STATE, "no far field set up");
  CK(cudaSetDevice(c->device));
  // without a block until the buffer is there: no graph keeps the old one's address
  c->dft_block = 0;
  invalidate(c);
  if (steps) {
    dfree(c, c->dft_samples);
    c->dft_samples = nullptr;
    const long long npts = c->ffsz[0] + c->ffsz[1] + c->ffsz[2];
    int rc = dalloc(c, (void**)&c->dft_samples, sizeof(float) * (size_t)steps * npts * 8);
    if (!rc && !c->d_dft_done) rc = dalloc(c, (void**)&c->d_dft_done, sizeof(int));
    if (rc) return rc;
    // every earlier step is already in the accumulators
    CK(xfer(c, c->d_dft_done, &c->ts, sizeof(int), cudaMemcpyHostToDevice));
  }
  c->dft_block = steps;
  return FDTD_OK;
}

int fdtd_ctx_set_dft_accumulator(fdtd_ctx* c, int kahan_fp32) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (kahan_fp32 != 0 && kahan_fp32 != 1) return fail(FDTD_ERR_BADARG, "accumulator mode %d not in {0,1}", kahan_fp32);
  if (kahan_fp32 && c->prec == FDTD_PREC_F64) return fail(FDTD_ERR_BADARG, "FP64 problems keep FP64 accumulators");
  if (c->ts != 0) return fail(FDTD_ERR_STATE, "the accumulator mode is set before the first step");
  c->acc_kahan = kahan_fp32;
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_set_x_wall(fdtd_ctx* c, int wall) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (wall != 0 && wall != 1) return fail(FDTD_ERR_BADARG, "x wall mode %d not in {0,1}", wall);
  c->x_wall = wall;
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_set_step_path(fdtd_ctx* c, int path) {
  if (!c) return fail(FDTD_ERR_BADARG, "NULL handle");
  Using use(c->mu);
  if (path != 0 && path != 1) return fail(FDTD_ERR_BADARG, "step path %d not in {0,1}", path);
  CK(cudaSetDevice(c->device));
  if (path == 1)
    if (int rc = fused_drop(c)) return rc;
  c->half_steps = path == 1;
  invalidate(c);
  return FDTD_OK;
}

int fdtd_ctx_get_step_path(const fdtd_ctx* c, int* path) {
  if (!c || !path) return fail(FDTD_ERR_BADARG, "NULL argument");
  *path = c->half_steps;
  return FDTD_OK;
}

int fdtd_ctx_get_x_wall(const fdtd_ctx* c, int* wall) {
  if (!c || !wall) return fail(FDTD_ERR_BADARG, "NULL argument");
  *wall = c->x_wall;
  return FDTD_OK;
}

// Direct time-to-frequency transform (dft.js:17-38); one block per frequency.
__global__ void __launch_bounds__(256) k_dft(const double* x, int N, double dt, const double* f, double shift,
                                             double* re, double* im) {
  __shared__ double sr[256], si[256];
  const int m = blockIdx.x;
  const double w = 2 * M_PI * f[m];
  double r = 0.0, q = 0.0;
  for (int n = threadIdx.x; n < N; n += blockDim.x) {
    const double ph = w * ((n + 1) * dt + shift);
    double s, c;
    sincos(ph, &s, &c);
    r += x[n] * c;
    q -= x[n] * s;
  }
  sr[threadIdx.x] = r;
  si[threadIdx.x] = q;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sr[threadIdx.x] += sr[threadIdx.x + o];
      si[threadIdx.x] += si[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    re[m] = sr[0] * dt;
    im[m] = si[0] * dt;
  }
}

int fdtd_dft(const double* x, int N, double dt, const double* freqs, int M, double shift, double* re, double* im) {
  if (!x || !freqs || !re || !im || N <= 0 || M <= 0) return fail(FDTD_ERR_BADARG, "bad DFT arguments");
  double *dx_ = nullptr, *df = nullptr, *dr = nullptr;
  int rc = FDTD_OK, dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev_malloc(dev, (void**)&dx_, N * sizeof(double)) != cudaSuccess ||
      dev_malloc(dev, (void**)&df, M * sizeof(double)) != cudaSuccess ||
      dev_malloc(dev, (void**)&dr, 2 * M * sizeof(double)) != cudaSuccess) {
    rc = fail(FDTD_ERR_OOM, "DFT buffers");
  } else if (cudaMemcpy(dx_, x, N * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
             cudaMemcpy(df, freqs, M * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) {
    rc = fail(FDTD_ERR_CUDA, "DFT upload");
  } else {
    k_dft<<<M, 256>>>(dx_, N, dt, df, shift, dr, dr + M);
    if (cudaMemcpy(re, dr, M * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(im, dr + M, M * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = fail(FDTD_ERR_CUDA, "DFT: %s", cudaGetErrorString(cudaGetLastError()));
  }
  cudaFree(dx_);
  cudaFree(df);
  cudaFree(dr);
  return rc;
}

// A run of directions [a0, a1) of a far-field call and the distinct values among
// their thetas, [t0, t1) of the call's list.
struct FFRun {
  int a0, a1, t0, t1;
};

// Cuts the directions into runs of at most `most` distinct thetas; cth: their
// cosines, ith: each direction's place among its run's.
static std::vector<FFRun> ff_runs(const double* theta, int nang, int most, std::vector<double>* cth,
                                  std::vector<int>* ith) {
  size_t slots = 16;
  while (slots < 2 * (size_t)std::min(most, nang)) slots *= 2;
  std::vector<int> slot(slots, -1);
  std::vector<double> val;  // of the current run
  std::vector<FFRun> runs;
  cth->clear();
  ith->resize(nang);
  auto cut = [&](int a1) {
    const int a0 = runs.empty() ? 0 : runs.back().a1, t0 = (int)cth->size();
    for (double t : val) cth->push_back(cos(t));
    runs.push_back({a0, a1, t0, (int)cth->size()});
    val.clear();
    std::fill(slot.begin(), slot.end(), -1);
  };
  for (int q = 0; q < nang; q++) {
    unsigned long long bits;
    memcpy(&bits, theta + q, sizeof(bits));
    size_t h = 0;
    auto find = [&] {
      h = (bits * 0x9E3779B97F4A7C15ull >> 32) & (slots - 1);
      while (slot[h] >= 0 && memcmp(&val[slot[h]], &bits, sizeof(bits))) h = (h + 1) & (slots - 1);
      return slot[h] >= 0;
    };
    if (!find()) {
      if ((int)val.size() >= most) {
        cut(q);
        find();
      }
      slot[h] = (int)val.size();
      val.push_back(theta[q]);
    }
    (*ith)[q] = slot[h];
  }
  if (nang > 0) cut(nang);
  return runs;
}

int fdtd_ctx_farfield_post(fdtd_ctx* c, const double* theta, const double* phi, int nang, double* radp,
                           double* d_theta, double* d_phi) {
  if (!c || !radp || (nang > 0 && (!theta || !phi || !d_theta || !d_phi)) || nang < 0)
    return fail(FDTD_ERR_BADARG, "bad far-field post arguments");
  if (c->nFreq == 0) return fail(FDTD_ERR_STATE, "no far field set up");
  CK(cudaSetDevice(c->device));
  FFPost P{};
  P.acc = c->acc;
  double* conv = nullptr;
  if (c->acc_kahan) {
    const long long n = c->ffoff[23] + 2LL * c->nFreq * c->ffsz[2];
    if (dev_malloc(c, &conv, n * sizeof(double)) != cudaSuccess) return fail(FDTD_ERR_OOM, "far-field post buffer");
    k_kahan_to_f64<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(c->acc, conv, n);
    P.acc = conv;
  }
  for (int a = 0; a < 24; a++) P.off[a] = c->ffoff[a];
  for (int a = 0; a < 3; a++) P.sz[a] = c->ffsz[a];
  P.nFreq = c->nFreq;
  P.ni = c->ui - c->li;
  P.nj = c->uj - c->lj;
  P.nk = c->uk - c->lk;
  const double d[3] = {c->dx, c->dy, c->dz};
  const int lo[3] = {c->li, c->lj, c->lk}, hi[3] = {c->ui, c->uj, c->uk};
  for (int a = 0; a < 3; a++) {
    const double centre = 0.5 * (hi[a] + lo[a]);
    P.d[a] = d[a];
    P.pos0[a] = ((lo[a] - 1) - centre + 0.5) * d[a];
    P.face[a][0] = (hi[a] - centre) * d[a];
    P.face[a][1] = (lo[a] - centre) * d[a];
  }
  const int F = c->nFreq;
  const size_t na = (size_t)nang;
  const size_t R = 2 * (size_t)(P.ni + P.nj);
  std::vector<double> cth;
  std::vector<int> ith;
  std::vector<FFRun> runs;
  // one buffer: frequencies, radiated power, angles, results, then the row sums
  // of one run of directions, for as many frequencies as fit `room` values; with
  // less memory left, shorter runs and fewer frequencies at a time
  const size_t n_out = 8 * (size_t)F + 2 * na + 2 * F * na;
  size_t n_rows = 0, n_z = 0;
  int parts = 1, fb = 1;
  double* buf = nullptr;
  int rc = FDTD_OK;
  for (size_t room = (size_t)128 << 20; !buf; room /= 8) {
    const int most = (int)std::max<size_t>(64, std::min<size_t>(1 << 20, room / 2 / (8 * R)));
    try {
      runs = ff_runs(theta, nang, most, &cth, &ith);
    } catch (const std::bad_alloc&) {
      rc = fail(FDTD_ERR_OOM, "far-field post: host memory for %d directions", nang);
      break;
    }
    int ang = 0, th = 0;
    for (const FFRun& u : runs) {
      ang = std::max(ang, u.a1 - u.a0);
      th = std::max(th, u.t1 - u.t0);
    }
    // z-face rows in parts, for some eight blocks of k_ff_zrows a multiprocessor
    const int ztiles = ang / (kFFZThreads * kFFZAng) + 1;
    parts = std::max(1, std::min(P.ni, 8 * 148 / (ztiles * F)));
    n_rows = R * 8 * th;
    n_z = (size_t)parts * 8 * ang;
    fb = (int)std::min<size_t>(F, std::max<size_t>(1, room / std::max<size_t>(1, n_rows + n_z)));
    // the smallest form is worth other handles' padded state, the larger ones are not
    const size_t bytes = (n_out + fb * (n_rows + n_z) + cth.size() + na) * sizeof(double);
    const bool least = room < 65536;
    if ((least ? dev_malloc(c, &buf, bytes) : cudaMalloc(&buf, bytes)) != cudaSuccess) {
      cudaGetLastError();
      buf = nullptr;
      if (least) {
        rc = fail(FDTD_ERR_OOM, "far-field post buffers");
        break;
      }
    }
  }
  if (!rc) {
    double *dfreq = buf, *dradp = dfreq + F, *dpow = dradp + F, *dang = dpow + 6 * F, *dout = dang + 2 * na;
    double *dth = dout + 2 * F * na, *drows = dth + cth.size(), *dz = drows + fb * n_rows;
    int* dith = (int*)(dz + fb * n_z);
    auto up = [&](void* d, const void* h, size_t bytes) {
      return bytes ? cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, c->stream) : cudaSuccess;
    };
    cudaError_t e = up(dfreq, c->ffreq.data(), F * sizeof(double));
    if (e == cudaSuccess) e = up(dang, theta, na * sizeof(double));
    if (e == cudaSuccess) e = up(dang + na, phi, na * sizeof(double));
    if (e == cudaSuccess) e = up(dth, cth.data(), cth.size() * sizeof(double));
    if (e == cudaSuccess) e = up(dith, ith.data(), na * sizeof(int));
    if (e == cudaSuccess) {
      k_ff_power<<<dim3(F, 6), 256, 0, c->stream>>>(P, dpow);
      k_ff_power_sum<<<(F + 127) / 128, 128, 0, c->stream>>>(dpow, F, dradp);
      for (const FFRun& u : runs)
        for (int f0 = 0; f0 < F; f0 += fb) {
          const int per = kFFRowThreads * kFFRowAng, zper = kFFZThreads * kFFZAng, nth = u.t1 - u.t0, ang = u.a1 - u.a0;
          const unsigned nf = (unsigned)std::min(fb, F - f0);
          const FFSums W{f0,  nth,   dth + u.t0, dith + u.a0, dang + u.a0, dang + na + u.a0,
                         ang, drows, dz,         parts};
          k_ff_rows<<<dim3((unsigned)R, (nth + per - 1) / per, nf), kFFRowThreads, 0, c->stream>>>(P, W, dfreq);
          k_ff_zrows<<<dim3((ang + zper - 1) / zper, parts, nf), kFFZThreads, 0, c->stream>>>(P, W, dfreq);
          k_ff_pattern<<<dim3((ang + 127) / 128, nf), 128, 0, c->stream>>>(P, W, dfreq, dradp, (long long)na, dout + u.a0,
                                                                          dout + F * na + u.a0);
        }
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(radp, dradp, F * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess && nang > 0)
      e = cudaMemcpyAsync(d_theta, dout, F * na * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess && nang > 0)
      e = cudaMemcpyAsync(d_phi, dout + F * na, F * na * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) rc = fail(FDTD_ERR_CUDA, "far-field post: %s", cudaGetErrorString(e));
  }
  cudaFree(buf);
  cudaFree(conv);
  return rc;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of fdtd_dft.  Its device staging area is this
// file-scope array instead of cudaMalloc'd buffers, so a call allocates and
// frees nothing.  Every GPU that loads the library holds the array until the
// process exits.  Layout: samples | frequencies | re | im.
// ---------------------------------------------------------------------------
constexpr int kDftNoAllocMaxSamples = 32768;
constexpr int kDftNoAllocMaxFreqs = 4096;
static __device__ __align__(256) double g_dft_scratch[kDftNoAllocMaxSamples + 3 * kDftNoAllocMaxFreqs];

// The array's device address, looked up once per device with that device
// current.  In host code `g_dft_scratch` only names a host-side stand-in, so
// the kernel must be given this address, never the symbol itself.
static int dft_scratch_address(double** out) {
  constexpr int kMaxDevices = 64;
  static double* addr[kMaxDevices] = {};
  static std::mutex lock;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(FDTD_ERR_CUDA, "device ordinal %d not supported", dev);
  std::lock_guard<std::mutex> g(lock);
  if (!addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_dft_scratch);
    if (e != cudaSuccess) return fail(FDTD_ERR_CUDA, "cudaGetSymbolAddress(dft scratch): %s", cudaGetErrorString(e));
    addr[dev] = (double*)p;
  }
  *out = addr[dev];
  return FDTD_OK;
}

int fdtd_dft_noalloc(const double* x, int N, double dt, const double* freqs, int M, double shift, double* re,
                     double* im) {
  if (!x || !freqs || !re || !im) return fail(FDTD_ERR_BADARG, "NULL argument");
  if (N <= 0 || N > kDftNoAllocMaxSamples)
    return fail(FDTD_ERR_BADARG, "fdtd_dft_noalloc: %d samples, must be 1..%d", N, kDftNoAllocMaxSamples);
  if (M <= 0 || M > kDftNoAllocMaxFreqs)
    return fail(FDTD_ERR_BADARG, "fdtd_dft_noalloc: %d frequencies, must be 1..%d", M, kDftNoAllocMaxFreqs);
  double* s = nullptr;
  int rc = dft_scratch_address(&s);
  if (rc) return rc;
  double* d_x = s;
  double* d_f = s + kDftNoAllocMaxSamples;
  double* d_re = d_f + kDftNoAllocMaxFreqs;
  double* d_im = d_re + kDftNoAllocMaxFreqs;
  // Every value the kernel reads is written by this call and every output is
  // fully overwritten, so nothing left by an earlier call needs clearing.
  CK(cudaMemcpy(d_x, x, N * sizeof(double), cudaMemcpyHostToDevice));
  CK(cudaMemcpy(d_f, freqs, M * sizeof(double), cudaMemcpyHostToDevice));
  k_dft<<<M, 256>>>(d_x, N, dt, d_f, shift, d_re, d_im);
  CK(cudaGetLastError());
  CK(cudaMemcpy(re, d_re, M * sizeof(double), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(im, d_im, M * sizeof(double), cudaMemcpyDeviceToHost));
  return FDTD_OK;
}

}  // extern "C"

// ===========================================================================
// Batches: member handles advanced together, one launch per kernel kind per
// step for all of them (fdtd_batch.cuh).
// ===========================================================================
struct fdtd_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  int prec = FDTD_PREC_F32_TABLE;
  std::vector<fdtd_ctx*> m;
  int ichunk = 8, block_rows = 4, prefetch = 1, group = 0;
  int block_w = 32;
  void* d_inst = nullptr;
  size_t inst_size = 0;  // bytes of one Instance
  BatchTile* d_tiles = nullptr;
  BatchBlock* d_mid = nullptr;
  BatchBlock* d_epi = nullptr;
  BatchCtl* d_ctl = nullptr;
  std::vector<BatchTile> tiles;
  std::vector<BatchBlock> mid, epi, flush;
  BatchBlock* d_flush = nullptr;
  int grid_h = 0, grid_e = 0;  // persistent grid sizes
  RunGraphs graphs;
  // member-kernel mode (streams > 0): each member's own step kernels, members
  // spread over `streams` worker streams joined to `stream`
  int streams = 0;
  std::vector<cudaStream_t> ws;
  std::vector<cudaEvent_t> wev;
  cudaEvent_t fork_ev = nullptr;
  // grouped mode (members_per_launch > 0, streams == 0): the members'
  // parameter blocks travel as kernel parameters, `members_per_launch` per
  // launch; the launches of one half-step run side by side on worker streams
  int members_per_launch = 0;
  std::vector<unsigned char> groups;  // host copies of the BatchGroup parameter structs
  int ngroups = 0;
  size_t group_size = 0;
  // what the cached graphs were captured from, see batch_take_path
  std::vector<long long> graph_key;
};

namespace {

void batch_drop_graph(fdtd_batch* b) { b->graphs.clear(); }

// How a run of a batch advances its members.
enum BatchPath { kTileList, kMemberKernels, kChains };

// Graphs of one path are cached by step count and place in a DFT block, which
// say nothing about the path, nor about what the launches of member kernels and
// chains carry of the members themselves: their set-up, and the copies of the
// state that chains start from, relative to the first member's.  Graphs captured
// from anything else are dropped.  (The tile list reads the members' parameters
// from device memory; batch_prepare drops its graphs where the lists, or the
// grouped launches' parameters, change.)
void batch_take_path(fdtd_batch* b, BatchPath path) {
  std::vector<long long> key{path};
  for (const fdtd_ctx* c : b->m) {
    if (path == kTileList) break;
    key.push_back(c->graphs.rev);
    key.push_back(path == kChains ? c->fs.cur ^ b->m[0]->fs.cur : 0);
  }
  if (key == b->graph_key) return;
  batch_drop_graph(b);
  b->graph_key.swap(key);
}

template <class V>
int upload_vec(fdtd_batch* b, V** dst, const std::vector<V>& v) {
  if (*dst) cudaFree(*dst);
  *dst = nullptr;
  const size_t bytes = std::max<size_t>(v.size(), 1) * sizeof(V);
  CK(dev_malloc(b->device, (void**)dst, bytes));
  if (!v.empty()) CK(cudaMemcpyAsync(*dst, v.data(), v.size() * sizeof(V), cudaMemcpyHostToDevice, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  return FDTD_OK;
}

int batch_worker_streams(fdtd_batch* b, int count);

// One half-step of every group: the groups' launches fork from the batch's
// stream onto worker streams and join back into it (also under capture).
template <typename T, class C, bool EXACT>
int batch_group_half(fdtd_batch* b, bool electric, size_t smem) {
  using G = BatchGroup<T, C>;
  auto k = batch_group_kernel<T, C, EXACT>(electric, b->prefetch);
  const dim3 blk(b->block_w, b->block_rows);
  CK(cudaEventRecord(b->fork_ev, b->stream));
  for (int g = 0; g < b->ngroups; g++) {
    const G& grp = *reinterpret_cast<const G*>(b->groups.data() + (size_t)g * sizeof(G));
    cudaStream_t st = b->ngroups == 1 ? b->stream : b->ws[g];
    if (st != b->stream) CK(cudaStreamWaitEvent(st, b->fork_ev, 0));
    k<<<(unsigned)grp.first[grp.n], blk, smem, st>>>(grp);
    if (st != b->stream) {
      CK(cudaEventRecord(b->wev[g], st));
      CK(cudaStreamWaitEvent(b->stream, b->wev[g], 0));
    }
  }
  CK(cudaGetLastError());
  return FDTD_OK;
}

// The parameter blocks of every member (member state may have moved since the
// last run: traces, tables) and, when the work lists changed, the lists.
template <typename T, class C, bool EXACT>
int batch_prepare(fdtd_batch* b, C (*coef_of)(fdtd_ctx*)) {
  using In = Instance<T, C>;
  const int n = (int)b->m.size();
  std::vector<unsigned char> host((size_t)n * sizeof(In), 0);
  std::vector<BatchTile> tiles;
  std::vector<BatchBlock> mid, epi, flush;
  for (int q = 0; q < n; q++) {
    fdtd_ctx* c = b->m[q];
    In in;
    memset(&in, 0, sizeof(In));
    in.sp = step_params<T, C>(c, coef_of(c));
    in.sp.ichunk = b->ichunk;
    in.sp.ts = &b->d_ctl->ts;
    in.pr = dev_probes(c);
    in.ff = dev_ff(c);
    memcpy(host.data() + (size_t)q * sizeof(In), &in, sizeof(In));
    const int gx = (c->nz + b->block_w) / b->block_w, gy = (c->ny + b->block_rows) / b->block_rows,
              gz = (c->nx + 1 + b->ichunk - 1) / b->ichunk;
    if (gx > 65535 || gy > 65535 || gz > 65535)
      return fail(FDTD_ERR_BADARG, "batch member %d: %dx%dx%d tiles exceed the tile index range", q, gx, gy, gz);
    for (int z = 0; z < gz; z++)
      for (int y = 0; y < gy; y++)
        for (int x = 0; x < gx; x++)
          tiles.push_back(BatchTile{(unsigned short)q, (unsigned short)x, (unsigned short)y, (unsigned short)z});
    const long long nmid = (long long)c->ny * (c->nz + 1) + in.pr.n_i;
    for (long long s = 0; s < (nmid + 255) / 256; s++) mid.push_back(BatchBlock{q, (int)s});
    const long long nff = (c->nFreq > 0) ? c->ffsz[0] + c->ffsz[1] + c->ffsz[2] : 0;
    for (long long s = 0; s < (nff + in.pr.n_v + 255) / 256; s++) epi.push_back(BatchBlock{q, (int)s});
    if (c->dft_block > 0)
      for (long long s = 0; s < flush_blocks(nff, c->nFreq); s++) flush.push_back(BatchBlock{q, (int)s});
  }
  if (tiles.size() > (size_t)INT32_MAX) return fail(FDTD_ERR_BADARG, "batch has too many tiles");
  if (b->members_per_launch > 0) {
    // grouped mode: consecutive members, members_per_launch per launch
    using G = BatchGroup<T, C>;
    const int per = b->members_per_launch;
    const int ng = (n + per - 1) / per;
    std::vector<unsigned char> gbytes((size_t)ng * sizeof(G), 0);
    for (int g = 0; g < ng; g++) {
      G grp;
      memset(&grp, 0, sizeof(G));
      grp.ts = g == 0 ? &b->d_ctl->ts : nullptr;
      long long blocks = 0;
      for (int q = g * per; q < std::min(n, (g + 1) * per); q++) {
        fdtd_ctx* c = b->m[q];
        const int k = q - g * per;
        const int gx = (c->nz + b->block_w) / b->block_w, gy = (c->ny + b->block_rows) / b->block_rows,
                  gz = (c->nx + 1 + b->ichunk - 1) / b->ichunk;
        grp.first[k] = (int)blocks;
        grp.gx[k] = gx;
        grp.gy[k] = gy;
        memcpy(&grp.sp[k], host.data() + (size_t)q * sizeof(In) + offsetof(In, sp), sizeof(grp.sp[k]));
        blocks += (long long)gx * gy * gz;
        grp.n = k + 1;
      }
      if (blocks > INT32_MAX) return fail(FDTD_ERR_BADARG, "batch group %d has too many blocks", g);
      grp.first[grp.n] = (int)blocks;
      memcpy(gbytes.data() + (size_t)g * sizeof(G), &grp, sizeof(G));
    }
    if (gbytes != b->groups) batch_drop_graph(b);
    b->groups.swap(gbytes);
    b->ngroups = ng;
    b->group_size = sizeof(G);
  } else {
    b->groups.clear();
    b->ngroups = 0;
  }
  if (!b->d_inst || b->inst_size != sizeof(In)) {
    if (b->d_inst) cudaFree(b->d_inst);
    b->d_inst = nullptr;
    CK(dev_malloc(b->device, &b->d_inst, host.size()));
    b->inst_size = sizeof(In);
  }
  CK(cudaMemcpyAsync(b->d_inst, host.data(), host.size(), cudaMemcpyHostToDevice, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  auto same = [](const std::vector<BatchBlock>& u, const std::vector<BatchBlock>& v) {
    return u.size() == v.size() && (u.empty() || !memcmp(u.data(), v.data(), u.size() * sizeof(BatchBlock)));
  };
  const bool same_tiles = tiles.size() == b->tiles.size() &&
                          (tiles.empty() || !memcmp(tiles.data(), b->tiles.data(), tiles.size() * sizeof(BatchTile)));
  if (!same_tiles || !same(mid, b->mid) || !same(epi, b->epi) || !same(flush, b->flush) || !b->d_tiles) {
    batch_drop_graph(b);
    b->tiles.swap(tiles);
    b->mid.swap(mid);
    b->epi.swap(epi);
    b->flush.swap(flush);
    int rc = upload_vec(b, &b->d_tiles, b->tiles);
    if (!rc) rc = upload_vec(b, &b->d_mid, b->mid);
    if (!rc) rc = upload_vec(b, &b->d_epi, b->epi);
    if (!rc) rc = upload_vec(b, &b->d_flush, b->flush);
    if (rc) return rc;
  }
  // persistent grids: as many blocks as fit on the device at once
  int sms = 0, per_h = 0, per_e = 0;
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device));
  int rc0 = check_block(b->block_w, b->block_rows);
  if (rc0) return rc0;
  const int threads = b->block_w * b->block_rows;
  size_t smem = 0;
  auto kh = batch_kernel<T, C, EXACT>(false, b->prefetch, true);
  auto ke = batch_kernel<T, C, EXACT>(true, b->prefetch, true);
  int rc = stage_smem(kh, b->prefetch, threads, &smem);
  if (!rc) rc = stage_smem(ke, b->prefetch, threads, &smem);
  if (rc) return rc;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_h, kh, threads, smem));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_e, ke, threads, smem));
  b->grid_h = std::max(1, per_h) * sms;
  b->grid_e = std::max(1, per_e) * sms;
  return FDTD_OK;
}

template <typename T, class C, bool EXACT>
int batch_enqueue(fdtd_batch* b, int count, KernelTimer* tm = nullptr) {
  const Instance<T, C>* in = (const Instance<T, C>*)b->d_inst;
  const int nt = (int)b->tiles.size();
  const dim3 blk(b->block_w, b->block_rows);
  const unsigned gh = b->group ? (unsigned)std::min(b->grid_h, (nt + b->group - 1) / b->group) : (unsigned)nt;
  const unsigned ge = b->group ? (unsigned)std::min(b->grid_e, (nt + b->group - 1) / b->group) : (unsigned)nt;
  auto kh = batch_kernel<T, C, EXACT>(false, b->prefetch, b->group != 0);
  auto ke = batch_kernel<T, C, EXACT>(true, b->prefetch, b->group != 0);
  size_t smem = 0;
  int rc = stage_smem(kh, b->prefetch, b->block_w * b->block_rows, &smem);
  if (!rc) rc = stage_smem(ke, b->prefetch, b->block_w * b->block_rows, &smem);
  if (rc) return rc;
  const bool grouped = b->ngroups > 0;
  size_t gsmem = 0;
  if (grouped) {
    rc = batch_worker_streams(b, b->ngroups);
    if (!rc) rc = stage_smem(batch_group_kernel<T, C, EXACT>(false, b->prefetch), b->prefetch,
                             b->block_w * b->block_rows, &gsmem);
    if (!rc) rc = stage_smem(batch_group_kernel<T, C, EXACT>(true, b->prefetch), b->prefetch,
                             b->block_w * b->block_rows, &gsmem);
    if (rc) return rc;
  }
  for (int s = 0; s < count; s++) {
    if (tm) CK(cudaEventRecord(tm->ev[0], b->stream));
    if (grouped) {
      rc = batch_group_half<T, C, EXACT>(b, false, gsmem);
      if (rc) return rc;
    } else {
      kh<<<gh, blk, smem, b->stream>>>(in, b->d_tiles, nt, b->d_ctl, b->group);
    }
    if (tm) CK(cudaEventRecord(tm->ev[1], b->stream));
    k_batch_mid<T, C, EXACT><<<(unsigned)b->mid.size(), 256, 0, b->stream>>>(in, b->d_mid, b->d_ctl,
                                                                             (int)b->m.size());
    if (tm) CK(cudaEventRecord(tm->ev[2], b->stream));
    if (grouped) {
      rc = batch_group_half<T, C, EXACT>(b, true, gsmem);
      if (rc) return rc;
    } else {
      ke<<<ge, blk, smem, b->stream>>>(in, b->d_tiles, nt, b->d_ctl, b->group);
    }
    if (tm) CK(cudaEventRecord(tm->ev[3], b->stream));
    if (!b->epi.empty()) k_batch_epilogue<T, C><<<(unsigned)b->epi.size(), 256, 0, b->stream>>>(in, b->d_epi);
    if (!b->flush.empty())
      k_batch_flush<T, C><<<(unsigned)b->flush.size(), 256, 0, b->stream>>>(in, b->d_flush, -1);
    if (tm) {
      CK(cudaEventRecord(tm->ev[4], b->stream));
      CK(cudaEventSynchronize(tm->ev[4]));
      for (int q = 0; q < 4; q++) {
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, tm->ev[q], tm->ev[q + 1]));
        tm->ms[q] += ms;
      }
    }
  }
  CK(cudaGetLastError());
  return FDTD_OK;
}

ArrayCoef<double> coef_f64(fdtd_ctx* c) { return array_coef<double>(c); }
ArrayCoef<float> coef_f32(fdtd_ctx* c) { return array_coef<float>(c); }
TableCoef coef_table(fdtd_ctx* c) { return c->tcoef; }

int batch_prepare_any(fdtd_batch* b) {
  if (b->prec == FDTD_PREC_F64) return batch_prepare<double, ArrayCoef<double>, true>(b, coef_f64);
  if (b->prec == FDTD_PREC_F32) return batch_prepare<float, ArrayCoef<float>, true>(b, coef_f32);
  return batch_prepare<float, TableCoef, false>(b, coef_table);
}

// Closes the members' open DFT blocks at the end of a run reaching `upto`.
template <typename T, class C>
int batch_close_blocks(fdtd_batch* b, int upto) {
  if (b->flush.empty()) return FDTD_OK;
  k_batch_flush<T, C><<<(unsigned)b->flush.size(), 256, 0, b->stream>>>((const Instance<T, C>*)b->d_inst, b->d_flush,
                                                                        upto);
  CK(cudaGetLastError());
  for (fdtd_ctx* c : b->m)
    if (c->dft_block > 0) CK(cudaMemcpyAsync(c->d_dft_done, &upto, sizeof(int), cudaMemcpyHostToDevice, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  return FDTD_OK;
}

int batch_close_any(fdtd_batch* b, int upto) {
  if (b->prec == FDTD_PREC_F64) return batch_close_blocks<double, ArrayCoef<double>>(b, upto);
  if (b->prec == FDTD_PREC_F32) return batch_close_blocks<float, ArrayCoef<float>>(b, upto);
  return batch_close_blocks<float, TableCoef>(b, upto);
}

int batch_enqueue_any(fdtd_batch* b, int count, KernelTimer* tm = nullptr) {
  if (b->prec == FDTD_PREC_F64) return batch_enqueue<double, ArrayCoef<double>, true>(b, count, tm);
  if (b->prec == FDTD_PREC_F32) return batch_enqueue<float, ArrayCoef<float>, true>(b, count, tm);
  return batch_enqueue<float, TableCoef, false>(b, count, tm);
}

// Member-kernel mode.  Sets a member's launch shape to the batch's for the
// duration of a scope (its own shape comes back afterwards).
struct MemberShape {
  fdtd_ctx* c;
  int ichunk, rows, pf, w;
  MemberShape(fdtd_ctx* m, const fdtd_batch* b)
      : c(m), ichunk(m->ichunk), rows(m->block_rows), pf(m->prefetch), w(m->block_w) {
    m->ichunk = b->ichunk;
    m->block_rows = b->block_rows;
    m->prefetch = b->prefetch;
    m->block_w = b->block_w;
  }
  ~MemberShape() {
    c->ichunk = ichunk;
    c->block_rows = rows;
    c->prefetch = pf;
    c->block_w = w;
  }
};

int batch_worker_streams(fdtd_batch* b, int count) {
  while ((int)b->ws.size() < count) {
    cudaStream_t st = nullptr;
    cudaEvent_t ev = nullptr;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    b->ws.push_back(st);
    CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
    b->wev.push_back(ev);
  }
  if (!b->fork_ev) CK(cudaEventCreateWithFlags(&b->fork_ev, cudaEventDisableTiming));
  return FDTD_OK;
}

// `count` steps of every member, member-major: worker stream s steps members
// s, s + S, s + 2S, ... one after another, all `count` steps of one member
// before the next, so a member's arrays are still in L2 at its next step.
// The worker streams fork from and join back into the batch's stream (also
// under stream capture), and are joined even when an enqueue fails.
int batch_member_enqueue(fdtd_batch* b, int count) {
  const int S = b->streams;
  CK(cudaEventRecord(b->fork_ev, b->stream));
  for (int q = 0; q < S; q++) CK(cudaStreamWaitEvent(b->ws[q], b->fork_ev, 0));
  int rc = FDTD_OK;
  for (size_t q = 0; q < b->m.size() && !rc; q++) {
    MemberShape shape(b->m[q], b);
    rc = enqueue(b->m[q], count, nullptr, b->ws[q % S]);
  }
  for (int q = 0; q < S; q++) {
    CK(cudaEventRecord(b->wev[q], b->ws[q]));
    CK(cudaStreamWaitEvent(b->stream, b->wev[q], 0));
  }
  return rc;
}

// One-pass mode.  A member's steps are a chain of launches that needs none of
// the other members', so the chains run side by side, each on its worker stream
// (member-major, as above), with blocks for its share of the device: no launch
// waits for the slowest member, and a member's last blocks overlap the others'
// first.  160 steps of 32 antennas of 1.1 M cells (material table), half-step
// tile list 224.5 ms; chains on 2, 4, 8, 16, 32 streams 200, 161, 139, 133,
// 132 ms.  6 FP64 antennas 53.9 ms; 34.0, 33.0, 29.3 ms on 2, 4, 6.
// Launches of a chain graph: 32 members' graphs of 32 steps run as fast as of
// 160 (132.3 ms), and the first run, which captures them, took 264 ms for 342.
constexpr int kChainNodes = 4096;
int batch_chain_streams(const fdtd_batch* b) { return std::min((int)b->m.size(), kMaxBatchStreams); }

int batch_chain_enqueue(fdtd_batch* b, int at, int count) {
  const int S = batch_chain_streams(b);
  CK(cudaEventRecord(b->fork_ev, b->stream));
  for (int q = 0; q < S; q++) CK(cudaStreamWaitEvent(b->ws[q], b->fork_ev, 0));
  int rc = FDTD_OK;
  for (size_t q = 0; q < b->m.size() && !rc; q++)
    rc = fused_enqueue(b->m[q], at, count, nullptr, b->ws[q % S], S > 1 ? 1.0 / S : 1);
  for (int q = 0; q < S; q++) {
    CK(cudaEventRecord(b->wev[q], b->ws[q]));
    CK(cudaStreamWaitEvent(b->stream, b->wev[q], 0));
  }
  return rc;
}

// Whether no other mode was chosen and every member can run the one-pass step
// (their DFT blocks closing together); then makes them hold the current state in
// that form.
int batch_chain_ready(fdtd_batch* b, bool* use) {
  *use = b->streams == 0 && b->group == 0 && b->members_per_launch == 0;
  for (const fdtd_ctx* c : b->m)
    *use = *use && !c->half_steps && c->dft_block == b->m[0]->dft_block && (c->fs.ok || !c->fs.tried || fused_retry(c));
  std::vector<fdtd_ctx*> order = b->m, built;  // those refused before first: they may be again
  std::stable_partition(order.begin(), order.end(), fused_retry);
  for (size_t q = 0; q < order.size() && *use; q++) {
    const bool had = order[q]->fs.ok;
    int rc = fused_usable(order[q], use);
    if (rc) return rc;
    if (!had && *use) built.push_back(order[q]);
  }
  if (!*use)  // built in vain
    for (fdtd_ctx* c : built)
      if (int rc = fused_drop(c)) return rc;
  for (size_t q = 0; q < b->m.size() && *use; q++) {
    fdtd_ctx* c = b->m[q];
    int rc = fused_ready(c, use);
    if (rc) return rc;
    CK(cudaStreamSynchronize(c->stream));
    if (c->dirty) {
      c->graphs.clear();
      c->dirty = false;
    }
  }
  return FDTD_OK;
}

// The first member that a run left with a status.
int batch_status(const fdtd_batch* b) {
  for (size_t q = 0; q < b->m.size(); q++)
    if (int rc = check_status(b->m[q], b->stream, "batch member " + std::to_string(q) + ": ")) return rc;
  return FDTD_OK;
}

// Runs the members: by their own step kernels on worker streams, or (chain) as
// one-pass chains.
int batch_run_members(fdtd_batch* b, int count, bool chain, float* elapsed_ms, KernelTimer* tm) {
  const int ts = b->m[0]->ts;
  int rc = batch_worker_streams(b, chain ? batch_chain_streams(b) : b->streams);
  if (rc) return rc;
  batch_take_path(b, chain ? kChains : kMemberKernels);
  // the whole run as cached graphs, captured before the first launch
  std::vector<cudaGraphExec_t> plan;
  if (!tm) {
    int per_step = 0;
    for (fdtd_ctx* c : b->m) per_step += c->dft_block > 0 ? 5 : 4;
    if (chain)
      rc = run_plan(b->graphs, b->stream, count, per_step, fused_start(b->m[0]),
                    [b](int at, int n) { return batch_chain_enqueue(b, at, n); }, &plan,
                    std::max(1, kChainNodes / per_step));
    else
      rc = run_plan(b->graphs, b->stream, count, per_step, RunStart(),
                    [b](int, int n) { return batch_member_enqueue(b, n); }, &plan);
    if (rc) return rc;
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  if (elapsed_ms) {
    CK(cudaEventCreate(&ev0));
    CK(cudaEventCreate(&ev1));
    CK(cudaEventRecord(ev0, b->stream));
  }
  if (tm) {
    // one member at a time on the batch's stream: per-kernel times summed over members
    for (size_t q = 0; q < b->m.size() && !rc; q++) {
      MemberShape shape(b->m[q], b);
      rc = chain ? fused_enqueue(b->m[q], 0, count, tm, b->stream) : enqueue(b->m[q], count, tm, b->stream);
    }
    if (rc) return rc;
  }
  if (chain && count > 0)  // from here the padded states run ahead of the dense ones
    for (fdtd_ctx* c : b->m) c->dense_valid = false;
  for (cudaGraphExec_t ge : plan) CK(cudaGraphLaunch(ge, b->stream));
  if (chain)
    for (fdtd_ctx* c : b->m) {
      c->fs.cur ^= count & 1;
      c->fs.ts_at = ts + count;
    }
  if (elapsed_ms) {
    CK(cudaEventRecord(ev1, b->stream));
    CK(cudaEventSynchronize(ev1));
    CK(cudaEventElapsedTime(elapsed_ms, ev0, ev1));
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
  }
  for (fdtd_ctx* c : b->m) {
    rc = count > 0 ? close_dft_block(c, ts + count, b->stream) : FDTD_OK;
    if (rc) return rc;
  }
  CK(cudaStreamSynchronize(b->stream));
  for (fdtd_ctx* c : b->m) c->ts += count;
  return batch_status(b);
}

int batch_run(fdtd_batch* b, int count, float* elapsed_ms = nullptr, KernelTimer* tm = nullptr) {
  if (count < 0) return fail(FDTD_ERR_BADARG, "negative step count %d", count);
  // in one order for all batches, as two with members in common may run at once
  std::vector<fdtd_ctx*> order = b->m;
  std::sort(order.begin(), order.end(), std::less<fdtd_ctx*>());
  std::vector<std::unique_lock<std::recursive_mutex>> use;
  for (fdtd_ctx* c : order) use.emplace_back(c->mu);
  const int ts = b->m[0]->ts;
  for (size_t q = 0; q < b->m.size(); q++) {
    fdtd_ctx* c = b->m[q];
    if (c->ts != ts) return fail(FDTD_ERR_STATE, "batch member %zu is at step %d, member 0 at step %d", q, c->ts, ts);
    if (ts + count > c->nsteps)
      return fail(FDTD_ERR_BADARG, "batch member %zu: running %d steps from step %d exceeds numberOfTimeSteps=%d", q,
                  count, ts, c->nsteps);
    int rc = check_ready(c);
    if (!rc) rc = ensure_traces(c);
    if (!rc && c->prec == FDTD_PREC_F32_TABLE && c->table_dirty) rc = prepare_table(c, &c->tcoef);
    if (rc) {
      std::string msg = g_err;
      return fail(rc, "batch member %zu: %s", q, msg.c_str());
    }
  }
  CK(cudaSetDevice(b->device));
  bool chain = false;
  int rc = count > 0 ? batch_chain_ready(b, &chain) : FDTD_OK;
  if (rc) return rc;
  if (chain) return batch_run_members(b, count, true, elapsed_ms, tm);
  for (size_t q = 0; q < b->m.size() && count > 0; q++)
    if ((rc = claim_dense(b->m[q]))) {
      std::string msg = g_err;
      return fail(rc, "batch member %zu: %s", q, msg.c_str());
    }
  if (b->streams > 0) return batch_run_members(b, count, false, elapsed_ms, tm);
  batch_take_path(b, kTileList);
  rc = batch_prepare_any(b);
  if (rc) return rc;
  const int ctl_ts = ts - 1;
  CK(cudaMemcpyAsync(&b->d_ctl->ts, &ctl_ts, sizeof(int), cudaMemcpyHostToDevice, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  // the whole run as cached graphs, captured before the first launch
  std::vector<cudaGraphExec_t> plan;
  if (!tm) {
    const int per_step = (b->flush.empty() ? 2 : 3) + (b->ngroups > 0 ? 2 * b->ngroups : 2);
    rc = run_plan(b->graphs, b->stream, count, per_step, RunStart(),
                  [b](int, int n) { return batch_enqueue_any(b, n); }, &plan);
    if (rc) return rc;
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  if (elapsed_ms) {
    CK(cudaEventCreate(&ev0));
    CK(cudaEventCreate(&ev1));
    CK(cudaEventRecord(ev0, b->stream));
  }
  if (tm) {
    rc = batch_enqueue_any(b, count, tm);
    if (rc) return rc;
  }
  for (cudaGraphExec_t ge : plan) CK(cudaGraphLaunch(ge, b->stream));
  if (elapsed_ms) {
    CK(cudaEventRecord(ev1, b->stream));
    CK(cudaEventSynchronize(ev1));
    CK(cudaEventElapsedTime(elapsed_ms, ev0, ev1));
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
  }
  if (count > 0) {
    rc = batch_close_any(b, ts + count);
    if (rc) return rc;
  }
  // hand the shared step counter back to every member
  for (fdtd_ctx* c : b->m) CK(cudaMemcpyAsync(c->d_ts, &b->d_ctl->ts, sizeof(int), cudaMemcpyDeviceToDevice, b->stream));
  CK(cudaStreamSynchronize(b->stream));
  for (fdtd_ctx* c : b->m) c->ts += count;
  return batch_status(b);
}

}  // namespace

extern "C" {

int fdtd_batch_create(fdtd_ctx* const* members, int count, fdtd_batch** out) {
  if (!members || !out || count < 1) return fail(FDTD_ERR_BADARG, "bad batch arguments");
  *out = nullptr;
  if (count > 65535) return fail(FDTD_ERR_BADARG, "a batch holds at most 65535 members");
  for (int q = 0; q < count; q++) {
    if (!members[q]) return fail(FDTD_ERR_BADARG, "batch member %d is NULL", q);
    if (members[q]->device != members[0]->device || members[q]->prec != members[0]->prec)
      return fail(FDTD_ERR_BADARG, "batch member %d differs from member 0 in device or precision", q);
    for (int r = 0; r < q; r++)
      if (members[r] == members[q]) return fail(FDTD_ERR_BADARG, "batch member %d repeats member %d", q, r);
  }
  fdtd_batch* b = new fdtd_batch();
  b->device = members[0]->device;
  b->prec = members[0]->prec;
  b->m.assign(members, members + count);
  if (cudaSetDevice(b->device) != cudaSuccess ||
      cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete b;
    return fail(FDTD_ERR_CUDA, "cannot create a stream on device %d", members[0]->device);
  }
  BatchCtl zero{};
  if (dev_malloc(b->device, (void**)&b->d_ctl, sizeof(BatchCtl)) != cudaSuccess ||
      cudaMemcpyAsync(b->d_ctl, &zero, sizeof(BatchCtl), cudaMemcpyHostToDevice, b->stream) != cudaSuccess ||
      cudaStreamSynchronize(b->stream) != cudaSuccess) {
    fdtd_batch_free(b);
    return fail(FDTD_ERR_CUDA, "cannot allocate the batch control block");
  }
  *out = b;
  return FDTD_OK;
}

void fdtd_batch_free(fdtd_batch* b) {
  if (!b) return;
  cudaSetDevice(b->device);
  if (b->stream) cudaStreamSynchronize(b->stream);
  batch_drop_graph(b);
  cudaFree(b->d_inst);
  cudaFree(b->d_tiles);
  cudaFree(b->d_mid);
  cudaFree(b->d_epi);
  cudaFree(b->d_flush);
  cudaFree(b->d_ctl);
  for (cudaStream_t st : b->ws) {
    cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
  }
  for (cudaEvent_t ev : b->wev) cudaEventDestroy(ev);
  if (b->fork_ev) cudaEventDestroy(b->fork_ev);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

int fdtd_batch_set_tiling(fdtd_batch* b, int x_planes_per_thread, int block_rows, int prefetch, int group) {
  if (!b) return fail(FDTD_ERR_BADARG, "NULL batch");
  if (x_planes_per_thread < 1 || x_planes_per_thread > 1024)
    return fail(FDTD_ERR_BADARG, "x planes per thread %d outside 1..1024", x_planes_per_thread);
  if (block_rows != 1 && block_rows != 2 && block_rows != 4 && block_rows != 8 && block_rows != 16)
    return fail(FDTD_ERR_BADARG, "block rows %d not in {1,2,4,8,16}", block_rows);
  if (prefetch < 1 || prefetch > 4) return fail(FDTD_ERR_BADARG, "prefetch depth %d not in 1..4", prefetch);
  if (prefetch > 2 && b->prec != FDTD_PREC_F32_TABLE)
    return fail(FDTD_ERR_BADARG, "prefetch depths 3 and 4 (shared-memory stages) need material-table members");
  if (group < 0 || group > 4096) return fail(FDTD_ERR_BADARG, "tile group %d outside 0..4096", group);
  if (b->ichunk != x_planes_per_thread || b->block_rows != block_rows || b->prefetch != prefetch ||
      b->group != group)
    batch_drop_graph(b);
  b->ichunk = x_planes_per_thread;
  b->block_rows = block_rows;
  b->prefetch = prefetch;
  b->group = group;
  return FDTD_OK;
}

int fdtd_batch_set_block_width(fdtd_batch* b, int threads_along_k) {
  if (!b) return fail(FDTD_ERR_BADARG, "NULL batch");
  if (threads_along_k != 16 && threads_along_k != 32)
    return fail(FDTD_ERR_BADARG, "block width %d not 16 or 32", threads_along_k);
  if (threads_along_k != b->block_w) batch_drop_graph(b);
  b->block_w = threads_along_k;
  return FDTD_OK;
}

int fdtd_batch_get_block_width(const fdtd_batch* b, int* threads_along_k) {
  if (!b || !threads_along_k) return fail(FDTD_ERR_BADARG, "NULL argument");
  *threads_along_k = b->block_w;
  return FDTD_OK;
}

int fdtd_batch_get_tiling(const fdtd_batch* b, int* x_planes_per_thread, int* block_rows, int* prefetch,
                          int* group) {
  if (!b || !x_planes_per_thread || !block_rows || !prefetch || !group) return fail(FDTD_ERR_BADARG, "NULL argument");
  *x_planes_per_thread = b->ichunk;
  *block_rows = b->block_rows;
  *prefetch = b->prefetch;
  *group = b->group;
  return FDTD_OK;
}

int fdtd_batch_set_streams(fdtd_batch* b, int streams) {
  if (!b) return fail(FDTD_ERR_BADARG, "NULL batch");
  if (streams < 0 || streams > kMaxBatchStreams)
    return fail(FDTD_ERR_BADARG, "worker streams %d outside 0..%d", streams, kMaxBatchStreams);
  if (streams != b->streams) batch_drop_graph(b);
  b->streams = streams;
  return FDTD_OK;
}

int fdtd_batch_set_members_per_launch(fdtd_batch* b, int members) {
  if (!b) return fail(FDTD_ERR_BADARG, "NULL batch");
  if (members < 0 || members > kGroupMembers)
    return fail(FDTD_ERR_BADARG, "members per launch %d outside 0..%d", members, kGroupMembers);
  if (members != b->members_per_launch) batch_drop_graph(b);
  b->members_per_launch = members;
  return FDTD_OK;
}

int fdtd_batch_get_members_per_launch(const fdtd_batch* b, int* members) {
  if (!b || !members) return fail(FDTD_ERR_BADARG, "NULL argument");
  *members = b->members_per_launch;
  return FDTD_OK;
}

int fdtd_batch_get_streams(const fdtd_batch* b, int* streams) {
  if (!b || !streams) return fail(FDTD_ERR_BADARG, "NULL argument");
  *streams = b->streams;
  return FDTD_OK;
}

int fdtd_batch_run(fdtd_batch* b, int count) {
  if (!b) return fail(FDTD_ERR_BADARG, "NULL batch");
  return batch_run(b, count);
}

int fdtd_batch_run_timed(fdtd_batch* b, int count, float* ms) {
  if (!b || !ms) return fail(FDTD_ERR_BADARG, "NULL argument");
  return batch_run(b, count, ms);
}

int fdtd_batch_profile_kernels(fdtd_batch* b, int count, double* avg_ms) {
  if (!b || !avg_ms || count < 1) return fail(FDTD_ERR_BADARG, "bad arguments");
  KernelTimer tm;
  CK(cudaSetDevice(b->device));
  for (int q = 0; q < 5; q++) CK(cudaEventCreate(&tm.ev[q]));
  int rc = batch_run(b, count, nullptr, &tm);
  for (int q = 0; q < 5; q++) cudaEventDestroy(tm.ev[q]);
  if (rc) return rc;
  for (int q = 0; q < 4; q++) avg_ms[q] = tm.ms[q] / count;
  return FDTD_OK;
}

int fdtd_batch_size(const fdtd_batch* b) { return b ? (int)b->m.size() : -1; }

// ===========================================================================
// Legacy global-context API (fdtd_cuda.h), FP32 per-cell coefficients.
// ===========================================================================
static fdtd_ctx* g_legacy = nullptr;

int fdtd_init(const FdtdDims* d) {
  if (!d) return fail(FDTD_ERR_BADARG, "NULL dims");
  fdtd_free(g_legacy);
  g_legacy = nullptr;
  FdtdConfig cfg{d->nx, d->ny, d->nz, d->dx, d->dy, d->dz, d->dt, d->numberOfTimeSteps, FDTD_PREC_F32, 0};
  return fdtd_create(&cfg, &g_legacy);
}

static std::vector<double> widen(const float* p, long long n) {
  std::vector<double> v(std::max<long long>(n, 0));
  for (long long q = 0; q < n; q++) v[q] = p[q];
  return v;
}

int fdtd_upload_coeff(int which, const float* host, int n) {
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  if (!host) return fail(FDTD_ERR_BADARG, "NULL array");
  auto v = widen(host, n);
  return fdtd_ctx_upload_coeff(g_legacy, which, v.data(), n);
}

int fdtd_upload_cpml(int faceId, int nc, const float* b_e, const float* a_e, const float* b_m, const float* a_m,
                     const float* CPsi0, int n0, const float* CPsi1, int n1, const float* CPsi2, int n2,
                     const float* CPsi3, int n3, int m_start, int e_start, int ascending) {
  (void)ascending;  // the band starts carry the same information
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  if (nc > 0 && (!b_e || !a_e || !b_m || !a_m)) return fail(FDTD_ERR_BADARG, "missing b/a profile");
  auto be = nc > 0 ? widen(b_e, nc) : std::vector<double>(), ae = nc > 0 ? widen(a_e, nc) : std::vector<double>();
  auto bm = nc > 0 ? widen(b_m, nc) : std::vector<double>(), am = nc > 0 ? widen(a_m, nc) : std::vector<double>();
  auto c0 = CPsi0 ? widen(CPsi0, n0) : std::vector<double>(), c1 = CPsi1 ? widen(CPsi1, n1) : std::vector<double>();
  auto c2 = CPsi2 ? widen(CPsi2, n2) : std::vector<double>(), c3 = CPsi3 ? widen(CPsi3, n3) : std::vector<double>();
  return fdtd_ctx_upload_cpml(g_legacy, faceId, nc, be.data(), ae.data(), bm.data(), am.data(), nullptr, nullptr,
                              CPsi0 ? c0.data() : nullptr, n0, CPsi1 ? c1.data() : nullptr, n1,
                              CPsi2 ? c2.data() : nullptr, n2, CPsi3 ? c3.data() : nullptr, n3, m_start, e_start);
}

int fdtd_upload_vsource(int dir, const int* idx, const float* coef, int count, const float* waveform, int nSteps) {
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  if (!coef || !waveform) return fail(FDTD_ERR_BADARG, "NULL array");
  auto cs = widen(coef, count), wv = widen(waveform, nSteps);
  return fdtd_ctx_add_vsource(g_legacy, dir, idx, cs.data(), count, wv.data(), nSteps);
}

int fdtd_upload_svoltage(int dir, const int* idx, int count, float Csvf) {
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  return fdtd_ctx_add_svoltage(g_legacy, dir, idx, count, Csvf);
}

int fdtd_upload_scurrent(const int* hxIdx, const float* hxW, int hxN, const int* hyIdx, const float* hyW, int hyN,
                         const int* hzIdx, const float* hzW, int hzN) {
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  std::vector<int> comp, idx;
  std::vector<double> w;
  const int* I[3] = {hxIdx, hyIdx, hzIdx};
  const float* W[3] = {hxW, hyW, hzW};
  const int N[3] = {hxN, hyN, hzN};
  for (int c = 0; c < 3; c++) {
    if (N[c] > 0 && (!I[c] || !W[c])) return fail(FDTD_ERR_BADARG, "NULL gather list");
    for (int q = 0; q < N[c]; q++) {
      comp.push_back(c);
      idx.push_back(I[c][q]);
      w.push_back(W[c][q]);
    }
  }
  return fdtd_ctx_add_scurrent(g_legacy, comp.data(), idx.data(), w.data(), (int)comp.size());
}

int fdtd_run_batch(int tsStart, int count, float* svOut, float* siOut) {
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  if (tsStart != g_legacy->ts) return fail(FDTD_ERR_BADARG, "batch starts at %d, the problem is at step %d", tsStart, g_legacy->ts);
  int rc = fdtd_ctx_run(g_legacy, count);
  if (rc && rc != FDTD_ERR_NONFINITE) return rc;
  std::vector<double> tmp(g_legacy->nsteps);
  if (svOut && !g_legacy->vprobe.empty()) {
    int r2 = fdtd_ctx_read_trace(g_legacy, 0, 0, tmp.data(), tsStart + count);
    if (r2) return r2;
    for (int q = 0; q < count; q++) svOut[q] = (float)tmp[tsStart + q];
  }
  if (siOut && !g_legacy->iprobe.empty()) {
    int r2 = fdtd_ctx_read_trace(g_legacy, 1, 0, tmp.data(), tsStart + count);
    if (r2) return r2;
    for (int q = 0; q < count; q++) siOut[q] = (float)tmp[tsStart + q];
  }
  return rc;
}

int fdtd_read_field(int which, float* host, int n) {
  if (!g_legacy) return fail(FDTD_ERR_STATE, "fdtd_init not called");
  if (!host) return fail(FDTD_ERR_BADARG, "NULL array");
  std::vector<double> tmp(std::max(n, 0));
  int rc = fdtd_ctx_read_field(g_legacy, which, tmp.data(), n);
  if (rc) return rc;
  for (int q = 0; q < n; q++) host[q] = (float)tmp[q];
  return FDTD_OK;
}

void fdtd_destroy(void) {
  fdtd_free(g_legacy);
  g_legacy = nullptr;
}

}  // extern "C"
