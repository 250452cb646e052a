// es_net.cu -- the learned early-stop network: a 1-D convolutional stack and
// an MLP head over the early port transient, with hand-written training and
// inference kernels.  Weights live as FP32 master values plus BF16 copies; the
// forward and backward passes read the BF16 copies and accumulate in FP32.
//
// Every layer is one GEMM: a convolution is
// out[(b,t)][co] = sum_{k,ci} in[b][t*stride+k-pad][ci] * W[co][k][ci], a dense
// layer is out[b][o] = sum_i in[b][i] * W[o][i].  Activations are stored time
// major with the channel fastest, so a convolution's GEMM output is directly
// the next layer's input, and the inputs of one output (its row of the GEMM) are
// one run of ksz*cin values, cut off at the ends of the sample: the GEMM reads
// them in place.  All reductions run in a fixed order (split sums are
// combined by a second pass, never by atomics), so training is reproducible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/fdtd_b200.h"
#include "fdtd_internal.h"

namespace {

int es_fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  return fdtd_internal_fail(code, buf);
}

#define ES_CK(call)                                                                                    \
  do {                                                                                                 \
    cudaError_t e_ = (call);                                                                           \
    if (e_ != cudaSuccess) return es_fail(FDTD_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_));     \
  } while (0)

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ float ld(const float* p) { return *p; }
__device__ __forceinline__ float ld(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// The rows of inputs that a layer's outputs read: row r = (b, t) is `kdim`
// values from in[b * width + off], off = (t * step - pad), zero where off + k
// leaves [0, width).  Dense: lout = 1, pad = 0, width = kdim.
struct Rows {
  const float* in;
  int lout, step, pad, width;
  __device__ __forceinline__ void at(int r, const float*& p, int& off) const {
    const int b = r / lout;
    off = (r - b * lout) * step - pad;
    p = in + (long long)b * width + off;
  }
};

// Three products, FP32 accumulation in order of k within a slice of the k range
// (kchunk wide, blockIdx.z):
//   kForward:  C[m][n] = sum_k rows(m, k) W[n][k]     (rows of inputs, BF16 weights)
//   kInput:    C[m][n] = sum_k Y[m][k] W[k][n]        (gradient with respect to the inputs)
//   kWeights:  C[n][m] = sum_k rows(k, m) Y[k][n], and bsum[n] = sum_k Y[k][n]
// With one slice (kForward, kInput) bias and ReLU, or the derivative of the ReLU
// whose output `post` is, are applied here, otherwise the slices' partial results
// go to C + z c_split for k_sum_slices.
//
// A tile is 128 x 64 x 16 with 8 x 4 results a thread, 3 shared-memory loads of
// 16 bytes per 32 multiply-adds, and the next tile's values are in flight while
// this one's are used.  The 64 x 64 tile with 4 x 4 results, scalar loads and no
// prefetch, over an im2col matrix in memory, took 1.7 ms of a 256-sample
// gradient's 2.1; these take 0.5 ms of 0.6.  (FP32 activations times BF16 weights on
// the tensor cores would need three products each, and round their sums
// otherwise.)
enum GemmForm { kForward, kInput, kWeights };
constexpr int kTM = 128, kTN = 64, kTK = 16;

template <GemmForm F>
__global__ void __launch_bounds__(256)
    k_gemm(int M, int N, int K, Rows rows, const float* __restrict__ Y, const __nv_bfloat16* __restrict__ W, int ldw,
           float* __restrict__ Cm, int ldc, long long c_split, int kchunk, const float* __restrict__ bias, int relu,
           const float* __restrict__ post, float* __restrict__ bsum) {
  __shared__ __align__(16) float As[2][kTK][kTM + 4];
  __shared__ __align__(16) float Bs[2][kTK][kTN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
  const int kbeg = blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
  // a thread's places in the tiles: kWeights walks m along a row, the others k
  const int ak = F == kWeights ? tid / kTM : tid % kTK, am = F == kWeights ? tid % kTM : tid / kTK;
  const int bk = F == kForward ? tid % kTK : tid / kTN, bn = F == kForward ? tid / kTK : tid % kTN;
  const float* ap[8];
  int aoff[8];
  if (F == kForward) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int m = m0 + am + 16 * q;
      ap[q] = nullptr;
      aoff[q] = 0;
      if (m < M) rows.at(m, ap[q], aoff[q]);
    }
  }
  float ra[8], rb[4];
  auto load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      ra[q] = 0.f;
      if (F == kForward) {
        const int k = k0 + ak;
        if (ap[q] && k < kend && (unsigned)(aoff[q] + k) < (unsigned)rows.width) ra[q] = ap[q][k];
      } else if (F == kInput) {
        const int k = k0 + ak, m = m0 + am + 16 * q;
        if (m < M && k < kend) ra[q] = Y[(long long)m * K + k];
      } else {
        const int k = k0 + ak + 2 * q, m = m0 + am;
        if (m < M && k < kend) {
          const float* p;
          int off;
          rows.at(k, p, off);
          if ((unsigned)(off + m) < (unsigned)rows.width) ra[q] = p[m];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      rb[q] = 0.f;
      if (F == kForward) {
        const int k = k0 + bk, n = n0 + bn + 16 * q;
        if (n < N && k < kend) rb[q] = __bfloat162float(W[(long long)n * ldw + k]);
      } else {
        const int k = k0 + bk + 4 * q, n = n0 + bn;
        if (n < N && k < kend)
          rb[q] = F == kInput ? __bfloat162float(W[(long long)k * ldw + n]) : Y[(long long)k * N + n];
      }
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 8; q++) As[buf][F == kWeights ? ak + 2 * q : ak][F == kWeights ? am : am + 16 * q] = ra[q];
#pragma unroll
    for (int q = 0; q < 4; q++) Bs[buf][F == kForward ? bk : bk + 4 * q][F == kForward ? bn + 16 * q : bn] = rb[q];
  };
  const int tx = tid % 16, ty = tid / 16;
  float acc[8][4];
#pragma unroll
  for (int a = 0; a < 8; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) acc[a][b] = 0.f;
  float bs = 0.f;
  const bool sums = F == kWeights && blockIdx.y == 0 && tid < kTN;
  load(kbeg);
  store(0);
  __syncthreads();
  for (int k0 = kbeg, buf = 0; k0 < kend; k0 += kTK, buf ^= 1) {
    const bool more = k0 + kTK < kend;
    if (more) load(k0 + kTK);
#pragma unroll
    for (int kk = 0; kk < kTK; kk++) {
      float a[8], b[4];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[buf][kk][4 * ty]);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&As[buf][kk][64 + 4 * ty]);
      *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&Bs[buf][kk][4 * tx]);
#pragma unroll
      for (int p = 0; p < 8; p++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[p][q] = fmaf(a[p], b[q], acc[p][q]);
    }
    if (sums) {
      float t = 0.f;
#pragma unroll
      for (int kk = 0; kk < kTK; kk++) t += Bs[buf][kk][tid];
      bs += t;
    }
    if (more) store(buf ^ 1);
    __syncthreads();
  }
  float* C = Cm + (long long)blockIdx.z * c_split;
  const bool single = gridDim.z == 1;
#pragma unroll
  for (int p = 0; p < 8; p++) {
    const int m = m0 + (p < 4 ? 0 : 60) + 4 * ty + p;
    if (m >= M) continue;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int n = n0 + 4 * tx + q;
      if (n >= N) continue;
      float v = acc[p][q];
      if (F == kWeights) {
        C[(long long)n * ldc + m] = v;
        continue;
      }
      if (single) {
        if (bias) v += bias[n];
        if (relu) v = fmaxf(v, 0.f);
        if (post && !(post[(long long)m * ldc + n] > 0.f)) v = 0.f;
      }
      C[(long long)m * ldc + n] = v;
    }
  }
  if (sums && n0 + tid < N) bsum[(long long)blockIdx.z * c_split + n0 + tid] = bs;
}

// out[i] = sum over s of part[s*n + i] (+ bias of column i % cols, ReLU, or the
// derivative of the ReLU whose output `post` is).  A block has 256 / Y values and
// Y threads each: thread y sums slices y, y + Y, ... in order, then the Y sums are
// added in order.  Y = 8 where there are many slices of few values: 296 slices of
// 704 values took 25 us with one thread each.
template <int Y>
__global__ void __launch_bounds__(256)
    k_sum_slices(const float* __restrict__ part, int slices, long long n, const float* __restrict__ bias, int cols,
                 int relu, const float* __restrict__ post, float* __restrict__ out) {
  constexpr int X = 256 / Y;
  __shared__ float red[Y][X];
  const int x = threadIdx.x % X, y = threadIdx.x / X;
  const long long i = (long long)blockIdx.x * X + x;
  float s = 0.f;
  if (i < n) {
#pragma unroll 8
    for (int q = y; q < slices; q += Y) s += part[(long long)q * n + i];
  }
  if constexpr (Y > 1) {
    red[y][x] = s;
    __syncthreads();
    if (y > 0) return;
    for (int q = 1; q < Y; q++) s += red[q][x];
  }
  if (i >= n) return;
  if (bias) s += bias[i % cols];
  if (relu) s = fmaxf(s, 0.f);
  if (post && !(post[i] > 0.f)) s = 0.f;
  out[i] = s;
}

// Adjoint of the rows' reads: din[b][s][c] = sum_k dcols[(b*lout + t)][k*cin + c],
// t = (s + pad - k) / stride where that is a whole number in [0, lout); times the
// derivative of the ReLU whose output `post` is.
__global__ void k_col2im(const float* __restrict__ dcols, int B, int lin, int cin, int lout, int ksz, int stride,
                         int pad, const float* __restrict__ post, float* __restrict__ din) {
  const int width = lin * cin;  // a sample's values; one per thread along x, samples along y
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= width) return;
  const int s = e / cin, c = e - s * cin;
  for (int b = blockIdx.y; b < B; b += gridDim.y) {
    const long long at = (long long)b * width + e;
    float acc = 0.f;
    for (int k = (s + pad) % stride; k < ksz; k += stride) {
      const int t = (s + pad - k) / stride;
      if (s + pad < k) break;
      if (t >= lout) continue;
      acc += dcols[((long long)b * lout + t) * (ksz * cin) + k * cin + c];
    }
    din[at] = post && !(post[at] > 0.f) ? 0.f : acc;
  }
}

// Per-sample weighted squared error and dL/dy = 2 w (y - t) / B.
__global__ void k_loss(const float* __restrict__ y, const float* __restrict__ t, const float* __restrict__ w, int B,
                       int D, float* __restrict__ dy, float* __restrict__ per) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  float s = 0.f;
  for (int o = 0; o < D; o++) {
    const float r = y[b * D + o] - t[b * D + o];
    s += w[o] * r * r;
    dy[b * D + o] = 2.f * w[o] * r / (float)B;
  }
  per[b] = s;
}

// Mean of per-sample losses (one block, fixed order).
__global__ void __launch_bounds__(256) k_mean(const float* __restrict__ per, int B, float* __restrict__ out) {
  __shared__ float red[256];
  float s = 0.f;
  for (int b = threadIdx.x; b < B; b += 256) s += per[b];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0] / (float)B;
}

// Adam with decoupled weight decay; refreshes the BF16 compute copy.
__global__ void k_adam(float* __restrict__ p, __nv_bfloat16* __restrict__ p16, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, long long n, float lr, float b1, float b2,
                       float eps, float wd, float c1, float c2) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  float pi = p[i];
  pi -= lr * wd * pi;
  pi -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  p[i] = pi;
  p16[i] = __float2bfloat16_rn(pi);
}

__global__ void k_to_bf16(const float* __restrict__ p, __nv_bfloat16* __restrict__ p16, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p16[i] = __float2bfloat16_rn(p[i]);
}

// Minibatch gather from the resident set (block row b = sample b of the batch).
__global__ void k_gather(const float* __restrict__ x, const float* __restrict__ y, const int* __restrict__ idx,
                         int B, int xw, int yw, float* __restrict__ bx, float* __restrict__ by) {
  const int b = blockIdx.y;
  if (b >= B) return;
  const long long s = idx[b];
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < xw; e += gridDim.x * blockDim.x)
    bx[(long long)b * xw + e] = x[s * xw + e];
  if (blockIdx.x == 0)
    for (int e = threadIdx.x; e < yw; e += blockDim.x) by[(long long)b * yw + e] = y[s * yw + e];
}

// Network input from the port traces of handle b (block b).
__global__ void __launch_bounds__(256) k_trace_inputs(const double* const* __restrict__ V,
                                                      const double* const* __restrict__ I, int L, int decim,
                                                      float* __restrict__ x, float* __restrict__ scales) {
  __shared__ float red[2][256];
  const int b = blockIdx.x;
  const double* src[2] = {V[b], I[b]};
  float mx[2] = {0.f, 0.f};
  for (int t = threadIdx.x; t < L; t += 256) {
    for (int ch = 0; ch < 2; ch++) {
      double s = 0.0;
      for (int q = 0; q < decim; q++) s += src[ch][(long long)t * decim + q];
      const float v = (float)(s / decim);
      x[((long long)b * L + t) * 2 + ch] = v;
      mx[ch] = fmaxf(mx[ch], fabsf(v));
    }
  }
  red[0][threadIdx.x] = mx[0];
  red[1][threadIdx.x] = mx[1];
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      red[0][threadIdx.x] = fmaxf(red[0][threadIdx.x], red[0][threadIdx.x + w]);
      red[1][threadIdx.x] = fmaxf(red[1][threadIdx.x], red[1][threadIdx.x + w]);
    }
    __syncthreads();
  }
  const float s0 = red[0][0] > 0.f ? red[0][0] : 1.f, s1 = red[1][0] > 0.f ? red[1][0] : 1.f;
  for (int t = threadIdx.x; t < L; t += 256) {
    x[((long long)b * L + t) * 2 + 0] /= s0;
    x[((long long)b * L + t) * 2 + 1] /= s1;
  }
  if (threadIdx.x == 0) {
    scales[2 * b] = s0;
    scales[2 * b + 1] = s1;
  }
}

unsigned blocks_for(long long n, int threads = 256) {
  return (unsigned)std::max<long long>(1, std::min<long long>((n + threads - 1) / threads, 1 << 20));
}

// One GEMM layer of the network.
struct Layer {
  bool conv;
  int cin, cout, lin, lout;  // conv: channels and lengths; dense: lin = lout = 1
  int ksz, stride, pad;
  bool relu;
  long long w_off, b_off;
  long long kdim() const { return conv ? (long long)ksz * cin : cin; }
  long long in_width() const { return (long long)lin * cin; }    // per-sample input values
  long long out_width() const { return (long long)lout * cout; }  // per-sample output values
};

}  // namespace

struct fdtd_es_net {
  FdtdEsConfig cfg{};
  cudaStream_t stream = nullptr;
  std::vector<Layer> layers;
  long long nparam = 0;
  float* p32 = nullptr;
  __nv_bfloat16* p16 = nullptr;
  float *grad = nullptr, *m = nullptr, *v = nullptr;
  std::vector<float*> act;  // act[0] input, act[l+1] output of layer l (max_batch samples)
  float *dcols = nullptr, *da = nullptr, *db = nullptr, *ws = nullptr;
  float *target = nullptr, *wout = nullptr, *dy = nullptr, *per = nullptr, *loss = nullptr;
  float *dset_x = nullptr, *dset_y = nullptr;
  int* d_perm = nullptr;  // shuffled sample order of the current epoch
  long long nsamples = 0;
  float* scales = nullptr;
  const double** d_traces = nullptr;  // [2][max_batch] device pointers
  long long adam_t = 0;
  std::vector<void*> owned;
};

namespace {

int es_alloc(fdtd_es_net* n, void** p, size_t bytes) {
  if (bytes == 0) bytes = 16;
  cudaError_t e = fdtd_internal_malloc(n->cfg.device, p, bytes);
  if (e != cudaSuccess) return es_fail(FDTD_ERR_OOM, "cudaMalloc(%zu bytes): %s", bytes, cudaGetErrorString(e));
  n->owned.push_back(*p);
  e = cudaMemsetAsync(*p, 0, bytes, n->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(n->stream);
  if (e != cudaSuccess) return es_fail(FDTD_ERR_CUDA, "zeroing: %s", cudaGetErrorString(e));
  return FDTD_OK;
}

void es_release(fdtd_es_net* n, void* p) {
  if (!p) return;
  cudaFree(p);
  n->owned.erase(std::remove(n->owned.begin(), n->owned.end(), p), n->owned.end());
}

Rows layer_rows(const Layer& L, const float* in) {
  return Rows{in, L.lout, L.stride * L.cin, L.conv ? L.pad * L.cin : 0, (int)L.in_width()};
}

// One product of the given form in `slices` slices of the k range.
template <GemmForm F>
void gemm(fdtd_es_net* n, int M, int N, int K, const Rows& rows, const float* Y, const __nv_bfloat16* W, int ldw,
          float* C, int ldc, const float* bias, bool relu, const float* post, int slices, long long c_split, float* bsum) {
  const int kchunk = ((K + slices - 1) / slices + kTK - 1) / kTK * kTK;
  const dim3 grd((N + kTN - 1) / kTN, (M + kTM - 1) / kTM, slices);
  k_gemm<F><<<grd, 256, 0, n->stream>>>(M, N, K, rows, Y, W, ldw, C, ldc, c_split, kchunk, bias, relu ? 1 : 0, post,
                                         bsum);
}

// Slices of a dense layer's k range: its few rows fill few tiles.  Never a
// function of the batch, so a sample's outputs do not depend on the others.
int dense_slices(long long k) { return (int)std::max<long long>(1, std::min<long long>(16, k / 128)); }

void sum_slices(fdtd_es_net* n, int slices, long long e, const float* bias, int cols, bool relu, const float* post,
                float* out) {
  if (slices >= 32)
    k_sum_slices<8><<<(unsigned)((e + 31) / 32), 256, 0, n->stream>>>(n->ws, slices, e, bias, cols, relu, post, out);
  else
    k_sum_slices<1><<<(unsigned)((e + 255) / 256), 256, 0, n->stream>>>(n->ws, slices, e, bias, cols, relu, post, out);
}

// rows x width results of kForward or kInput, through the slices' sums if need be.
template <GemmForm F>
void product(fdtd_es_net* n, const Layer& L, int M, int N, int K, const Rows& rows, const float* Y, float* C,
             const float* bias, bool relu, const float* post) {
  const int slices = L.conv ? 1 : dense_slices(K), ldw = (int)L.kdim();
  const __nv_bfloat16* W = n->p16 + L.w_off;
  if (slices == 1) {
    gemm<F>(n, M, N, K, rows, Y, W, ldw, C, N, bias, relu, post, 1, 0, nullptr);
  } else {
    const long long e = (long long)M * N;
    gemm<F>(n, M, N, K, rows, Y, W, ldw, n->ws, N, nullptr, false, nullptr, slices, e, nullptr);
    sum_slices(n, slices, e, bias, N, relu, post, C);
  }
}

// Forward pass of B samples already in act[0].
void forward(fdtd_es_net* n, int B) {
  for (size_t l = 0; l < n->layers.size(); l++) {
    const Layer& L = n->layers[l];
    product<kForward>(n, L, L.conv ? B * L.lout : B, L.cout, (int)L.kdim(), layer_rows(L, n->act[l]), nullptr,
                      n->act[l + 1], n->p32 + L.b_off, L.relu, nullptr);  // biases stay FP32
  }
}

// Slices of the weight-gradient reduction over `rows`: two blocks a
// multiprocessor, none below 64 rows.
int grad_slices(const Layer& L, long long rows) {
  const long long tiles = (L.kdim() + kTM - 1) / kTM * ((L.cout + kTN - 1) / kTN);
  return (int)std::max<long long>(1, std::min<long long>(296 / tiles, (rows + 63) / 64));
}

// dW and db of one layer from dpre (rows x cout) and its input: slice s sums its
// own range of rows; the slices are then added in order.
void weight_grads(fdtd_es_net* n, const Layer& L, const float* dpre, const float* in, int rows) {
  const int N = L.cout, K = (int)L.kdim(), slices = grad_slices(L, rows);
  const long long e = (long long)N * K + N;  // a slice: dW, then db, as in the gradient
  gemm<kWeights>(n, K, N, rows, layer_rows(L, in), dpre, nullptr, 0, n->ws, K, nullptr, false, nullptr, slices,
                 e, n->ws + (long long)N * K);
  sum_slices(n, slices, e, nullptr, 1, false, nullptr, n->grad + L.w_off);
}

// Backward pass: dy (B x out_dim) -> n->grad.  Activations of the forward pass
// are still in act[].
void backward(fdtd_es_net* n, int B) {
  float* dcur = n->dy;  // gradient with respect to the current layer's output
  float* bufs[2] = {n->da, n->db};
  int flip = 0;
  for (int l = (int)n->layers.size() - 1; l >= 0; l--) {
    const Layer& L = n->layers[l];
    const int rows = L.conv ? B * L.lout : B;
    float* dnext = bufs[flip];
    weight_grads(n, L, dcur, n->act[l], rows);
    if (l > 0) {
      const float* post = n->layers[l - 1].relu ? n->act[l] : nullptr;  // the gradient passes its ReLU too
      product<kInput>(n, L, rows, (int)L.kdim(), L.cout, Rows{}, dcur, L.conv ? n->dcols : dnext, nullptr, false,
                      L.conv ? nullptr : post);
      if (L.conv)
        k_col2im<<<dim3((L.lin * L.cin + 255) / 256, std::min(B, 1024)), 256, 0, n->stream>>>(
            n->dcols, B, L.lin, L.cin, L.lout, L.ksz, L.stride, L.pad, post, dnext);
    }
    dcur = dnext;
    flip ^= 1;
  }
}

int check_batch(const fdtd_es_net* n, int B) {
  if (B < 1 || B > n->cfg.max_batch)
    return es_fail(FDTD_ERR_BADARG, "batch %d outside 1..%d (max_batch)", B, n->cfg.max_batch);
  return FDTD_OK;
}

long long in_width(const fdtd_es_net* n) { return (long long)n->cfg.in_length * n->cfg.in_channels; }

// Loss of the batch in act[0] against n->target (both on the device).
int loss_and_grad(fdtd_es_net* n, int B, float* loss_host, bool want_grad) {
  forward(n, B);
  const int D = n->cfg.out_dim;
  k_loss<<<(B + 127) / 128, 128, 0, n->stream>>>(n->act.back(), n->target, n->wout, B, D, n->dy, n->per);
  k_mean<<<1, 256, 0, n->stream>>>(n->per, B, n->loss);
  if (want_grad) backward(n, B);
  ES_CK(cudaGetLastError());
  if (loss_host) {
    ES_CK(cudaMemcpyAsync(loss_host, n->loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    ES_CK(cudaStreamSynchronize(n->stream));
  }
  return FDTD_OK;
}

// xorshift64* stream for initialisation and shuffling.
struct Rng {
  unsigned long long s;
  explicit Rng(unsigned long long seed) : s(seed * 0x9E3779B97F4A7C15ull + 0x2545F4914F6CDD1Dull) {
    if (!s) s = 1;
  }
  unsigned long long next() {
    s ^= s >> 12;
    s ^= s << 25;
    s ^= s >> 27;
    return s * 0x2545F4914F6CDD1Dull;
  }
  double uniform() { return (next() >> 11) * (1.0 / 9007199254740992.0); }
};

int upload_params(fdtd_es_net* n, const float* host) {
  ES_CK(cudaMemcpyAsync(n->p32, host, n->nparam * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  k_to_bf16<<<blocks_for(n->nparam), 256, 0, n->stream>>>(n->p32, n->p16, n->nparam);
  ES_CK(cudaGetLastError());
  ES_CK(cudaStreamSynchronize(n->stream));
  return FDTD_OK;
}

int reset_optimizer(fdtd_es_net* n) {
  n->adam_t = 0;
  ES_CK(cudaMemsetAsync(n->m, 0, n->nparam * sizeof(float), n->stream));
  ES_CK(cudaMemsetAsync(n->v, 0, n->nparam * sizeof(float), n->stream));
  return FDTD_OK;
}

int trace_inputs(fdtd_es_net* n, fdtd_ctx* const* members, int count, int decim, float* scales) {
  if (!members || decim < 1) return es_fail(FDTD_ERR_BADARG, "bad member arguments");
  int rc = check_batch(n, count);
  if (rc) return rc;
  if (n->cfg.in_channels != 2) return es_fail(FDTD_ERR_STATE, "member inputs need in_channels == 2");
  const long long need = (long long)n->cfg.in_length * decim;
  std::vector<const double*> ptr(2 * count);
  for (int b = 0; b < count; b++) {
    if (!members[b]) return es_fail(FDTD_ERR_BADARG, "member %d is NULL", b);
    const double *V, *I;
    int nsteps, steps, dev;
    rc = fdtd_internal_traces(members[b], &V, &I, &nsteps, &steps, &dev);
    if (rc) return rc;
    if (dev != n->cfg.device)
      return es_fail(FDTD_ERR_BADARG, "member %d is on device %d, the network on %d", b, dev, n->cfg.device);
    if (steps < need) return es_fail(FDTD_ERR_STATE, "member %d has run %d steps, the input needs %lld", b, steps, need);
    ptr[b] = V;          // voltage probe 0
    ptr[count + b] = I;  // current probe 0
  }
  ES_CK(cudaMemcpyAsync(n->d_traces, ptr.data(), ptr.size() * sizeof(double*), cudaMemcpyHostToDevice, n->stream));
  k_trace_inputs<<<count, 256, 0, n->stream>>>(n->d_traces, n->d_traces + count, n->cfg.in_length, decim, n->act[0],
                                               n->scales);
  ES_CK(cudaGetLastError());
  if (scales)
    ES_CK(cudaMemcpyAsync(scales, n->scales, 2 * count * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
  ES_CK(cudaStreamSynchronize(n->stream));
  return FDTD_OK;
}

}  // namespace

extern "C" {

int fdtd_es_create(const FdtdEsConfig* cfg, fdtd_es_net** out) {
  if (!cfg || !out) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  *out = nullptr;
  const FdtdEsConfig& c = *cfg;
  if (c.in_channels < 1 || c.in_length < 1 || c.conv_layers < 0 || c.channels < 1 || c.kernel < 1 ||
      c.kernel % 2 == 0 || c.stride < 1 || c.mlp_layers < 0 || c.mlp_width < 1 || c.out_dim < 1 ||
      c.max_batch < 1 || c.max_batch > 65535)
    return es_fail(FDTD_ERR_BADARG, "invalid network configuration");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || c.device < 0 || c.device >= ndev)
    return es_fail(FDTD_ERR_CUDA, "CUDA device %d not available", c.device);
  fdtd_es_net* n = new fdtd_es_net();
  n->cfg = c;
  long long off = 0;
  int len = c.in_length, ch = c.in_channels;
  for (int l = 0; l < c.conv_layers; l++) {
    Layer L{};
    L.conv = true;
    L.cin = ch;
    L.cout = c.channels;
    L.lin = len;
    L.ksz = c.kernel;
    L.stride = c.stride;
    L.pad = c.kernel / 2;
    L.lout = (len + 2 * L.pad - L.ksz) / L.stride + 1;
    L.relu = true;
    L.w_off = off;
    off += (long long)L.cout * L.ksz * L.cin;
    L.b_off = off;
    off += L.cout;
    n->layers.push_back(L);
    len = L.lout;
    ch = L.cout;
  }
  int feat = len * ch;
  for (int l = 0; l <= c.mlp_layers; l++) {
    Layer L{};
    L.conv = false;
    L.cin = feat;
    L.cout = l < c.mlp_layers ? c.mlp_width : c.out_dim;
    L.lin = L.lout = 1;
    L.ksz = L.stride = 1;
    L.relu = l < c.mlp_layers;
    L.w_off = off;
    off += (long long)L.cout * L.cin;
    L.b_off = off;
    off += L.cout;
    n->layers.push_back(L);
    feat = L.cout;
  }
  n->nparam = off;
  if (cudaSetDevice(c.device) != cudaSuccess ||
      cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete n;
    return es_fail(FDTD_ERR_CUDA, "cannot create a stream on device %d", c.device);
  }
  const long long B = c.max_batch;
  long long max_act = in_width(n), max_cols = 1, max_ws = 1;
  n->act.assign(n->layers.size() + 1, nullptr);
  for (const Layer& L : n->layers) {
    max_act = std::max(max_act, std::max(L.in_width(), L.out_width()));
    const long long rows = L.conv ? B * L.lout : B;
    if (L.conv) max_cols = std::max(max_cols, rows * L.kdim());
    max_ws = std::max(max_ws, grad_slices(L, rows) * (L.cout * L.kdim() + L.cout));
    if (!L.conv) max_ws = std::max(max_ws, rows * std::max(dense_slices(L.cin) * L.cout, dense_slices(L.cout) * L.cin));
  }
  int rc = es_alloc(n, (void**)&n->p32, n->nparam * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->p16, n->nparam * sizeof(__nv_bfloat16));
  if (!rc) rc = es_alloc(n, (void**)&n->grad, n->nparam * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->m, n->nparam * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->v, n->nparam * sizeof(float));
  for (size_t l = 0; l <= n->layers.size() && !rc; l++) {
    const long long w = l == 0 ? in_width(n) : n->layers[l - 1].out_width();
    rc = es_alloc(n, (void**)&n->act[l], B * w * sizeof(float));
  }
  if (!rc) rc = es_alloc(n, (void**)&n->dcols, max_cols * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->da, B * max_act * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->db, B * max_act * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->ws, max_ws * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->target, B * c.out_dim * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->wout, c.out_dim * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->dy, B * c.out_dim * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->per, B * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->loss, sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->scales, 2 * B * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->d_traces, 2 * B * sizeof(double*));
  if (rc) {
    fdtd_es_free(n);
    return rc;
  }
  *out = n;
  return FDTD_OK;
}

void fdtd_es_free(fdtd_es_net* n) {
  if (!n) return;
  cudaSetDevice(n->cfg.device);
  if (n->stream) cudaStreamSynchronize(n->stream);
  for (void* p : n->owned) cudaFree(p);
  if (n->stream) cudaStreamDestroy(n->stream);
  delete n;
}

int fdtd_es_param_count(const fdtd_es_net* n, long* count) {
  if (!n || !count) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  *count = (long)n->nparam;
  return FDTD_OK;
}

int fdtd_es_init_params(fdtd_es_net* n, unsigned long long seed) {
  if (!n) return es_fail(FDTD_ERR_BADARG, "NULL network");
  std::vector<float> h(n->nparam);
  Rng r(seed);
  for (const Layer& L : n->layers) {
    const double bound = 1.0 / std::sqrt((double)L.kdim());
    for (long long q = L.w_off; q < L.b_off + L.cout; q++) h[q] = (float)((2.0 * r.uniform() - 1.0) * bound);
  }
  ES_CK(cudaSetDevice(n->cfg.device));
  int rc = reset_optimizer(n);
  return rc ? rc : upload_params(n, h.data());
}

int fdtd_es_set_params(fdtd_es_net* n, const float* params, long count) {
  if (!n || !params) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  if (count != n->nparam)
    return es_fail(FDTD_ERR_BADARG, "%ld parameters given, the network has %lld", count, n->nparam);
  ES_CK(cudaSetDevice(n->cfg.device));
  int rc = reset_optimizer(n);
  return rc ? rc : upload_params(n, params);
}

int fdtd_es_get_params(fdtd_es_net* n, float* params, long count) {
  if (!n || !params) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  if (count != n->nparam)
    return es_fail(FDTD_ERR_BADARG, "%ld parameters asked, the network has %lld", count, n->nparam);
  ES_CK(cudaSetDevice(n->cfg.device));
  ES_CK(cudaMemcpyAsync(params, n->p32, n->nparam * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
  ES_CK(cudaStreamSynchronize(n->stream));
  return FDTD_OK;
}

int fdtd_es_forward(fdtd_es_net* n, const float* x, int batch, float* y) {
  if (!n || !x || !y) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  int rc = check_batch(n, batch);
  if (rc) return rc;
  ES_CK(cudaSetDevice(n->cfg.device));
  ES_CK(cudaMemcpyAsync(n->act[0], x, batch * in_width(n) * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  forward(n, batch);
  ES_CK(cudaGetLastError());
  ES_CK(cudaMemcpyAsync(y, n->act.back(), (size_t)batch * n->cfg.out_dim * sizeof(float), cudaMemcpyDeviceToHost,
                        n->stream));
  ES_CK(cudaStreamSynchronize(n->stream));
  return FDTD_OK;
}

int fdtd_es_loss_grad(fdtd_es_net* n, const float* x, const float* target, const float* w, int batch, float* loss,
                      float* grad, long count) {
  if (!n || !x || !target || !w || !loss) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  int rc = check_batch(n, batch);
  if (rc) return rc;
  if (grad && count != n->nparam)
    return es_fail(FDTD_ERR_BADARG, "gradient buffer of %ld, the network has %lld", count, n->nparam);
  ES_CK(cudaSetDevice(n->cfg.device));
  const int D = n->cfg.out_dim;
  ES_CK(cudaMemcpyAsync(n->act[0], x, batch * in_width(n) * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  ES_CK(cudaMemcpyAsync(n->target, target, (size_t)batch * D * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  ES_CK(cudaMemcpyAsync(n->wout, w, D * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  rc = loss_and_grad(n, batch, loss, grad != nullptr);
  if (rc) return rc;
  if (grad) {
    ES_CK(cudaMemcpyAsync(grad, n->grad, n->nparam * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    ES_CK(cudaStreamSynchronize(n->stream));
  }
  return FDTD_OK;
}

int fdtd_es_set_data(fdtd_es_net* n, const float* x, const float* target, long count) {
  if (!n || !x || !target || count < 1) return es_fail(FDTD_ERR_BADARG, "bad training set");
  ES_CK(cudaSetDevice(n->cfg.device));
  es_release(n, n->dset_x);
  es_release(n, n->dset_y);
  es_release(n, n->d_perm);
  n->dset_x = n->dset_y = nullptr;
  n->d_perm = nullptr;
  n->nsamples = 0;
  int rc = es_alloc(n, (void**)&n->dset_x, count * in_width(n) * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->dset_y, (size_t)count * n->cfg.out_dim * sizeof(float));
  if (!rc) rc = es_alloc(n, (void**)&n->d_perm, count * sizeof(int));
  if (rc) return rc;
  ES_CK(cudaMemcpyAsync(n->dset_x, x, count * in_width(n) * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  ES_CK(cudaMemcpyAsync(n->dset_y, target, (size_t)count * n->cfg.out_dim * sizeof(float), cudaMemcpyHostToDevice,
                        n->stream));
  ES_CK(cudaStreamSynchronize(n->stream));
  n->nsamples = count;
  return FDTD_OK;
}

int fdtd_es_train(fdtd_es_net* n, int epochs, int batch, const float* w, float lr, float beta1, float beta2,
                  float eps, float weight_decay, unsigned long long seed, float* epoch_loss) {
  if (!n || !w || epochs < 0) return es_fail(FDTD_ERR_BADARG, "bad training arguments");
  int rc = check_batch(n, batch);
  if (rc) return rc;
  if (!n->dset_x) return es_fail(FDTD_ERR_STATE, "no training set (fdtd_es_set_data)");
  if (batch > n->nsamples) return es_fail(FDTD_ERR_BADARG, "batch %d larger than the training set", batch);
  ES_CK(cudaSetDevice(n->cfg.device));
  const int D = n->cfg.out_dim;
  ES_CK(cudaMemcpyAsync(n->wout, w, D * sizeof(float), cudaMemcpyHostToDevice, n->stream));
  const long long steps = n->nsamples / batch;
  std::vector<int> perm(n->nsamples);
  std::vector<float> losses(steps);
  Rng r(seed);
  float* d_losses = nullptr;
  rc = es_alloc(n, (void**)&d_losses, steps * sizeof(float));
  if (rc) return rc;
  for (int ep = 0; ep < epochs && !rc; ep++) {
    for (long long q = 0; q < n->nsamples; q++) perm[q] = (int)q;
    for (long long q = n->nsamples - 1; q > 0; q--) std::swap(perm[q], perm[r.next() % (q + 1)]);
    // the previous epoch ended with a stream wait, so no copy still reads perm
    ES_CK(cudaMemcpyAsync(n->d_perm, perm.data(), n->nsamples * sizeof(int), cudaMemcpyHostToDevice, n->stream));
    for (long long s = 0; s < steps && !rc; s++) {
      const dim3 g((unsigned)std::min<long long>(64, (in_width(n) + 255) / 256), batch);
      k_gather<<<g, 256, 0, n->stream>>>(n->dset_x, n->dset_y, n->d_perm + s * batch, batch, (int)in_width(n), D,
                                          n->act[0], n->target);
      rc = loss_and_grad(n, batch, nullptr, true);
      if (rc) break;
      ES_CK(cudaMemcpyAsync(d_losses + s, n->loss, sizeof(float), cudaMemcpyDeviceToDevice, n->stream));
      n->adam_t++;
      const double c1 = 1.0 / (1.0 - std::pow((double)beta1, (double)n->adam_t));
      const double c2 = 1.0 / (1.0 - std::pow((double)beta2, (double)n->adam_t));
      k_adam<<<blocks_for(n->nparam), 256, 0, n->stream>>>(n->p32, n->p16, n->grad, n->m, n->v, n->nparam, lr, beta1,
                                                           beta2, eps, weight_decay, (float)c1, (float)c2);
      ES_CK(cudaGetLastError());
    }
    if (rc) break;
    ES_CK(cudaMemcpyAsync(losses.data(), d_losses, steps * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    ES_CK(cudaStreamSynchronize(n->stream));
    if (epoch_loss) {
      double s = 0;
      for (float v : losses) s += v;
      epoch_loss[ep] = (float)(s / std::max<long long>(1, steps));
    }
  }
  cudaStreamSynchronize(n->stream);
  es_release(n, d_losses);
  return rc;
}

int fdtd_es_member_inputs(fdtd_es_net* n, fdtd_ctx* const* members, int count, int decim, float* scales,
                          float* x) {
  if (!n) return es_fail(FDTD_ERR_BADARG, "NULL network");
  ES_CK(cudaSetDevice(n->cfg.device));
  int rc = trace_inputs(n, members, count, decim, scales);
  if (rc) return rc;
  if (x) {
    ES_CK(cudaMemcpyAsync(x, n->act[0], count * in_width(n) * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    ES_CK(cudaStreamSynchronize(n->stream));
  }
  return FDTD_OK;
}

int fdtd_es_predict_members(fdtd_es_net* n, fdtd_ctx* const* members, int count, int decim, float* scales,
                            float* y) {
  if (!n || !y) return es_fail(FDTD_ERR_BADARG, "NULL argument");
  ES_CK(cudaSetDevice(n->cfg.device));
  int rc = trace_inputs(n, members, count, decim, scales);
  if (rc) return rc;
  forward(n, count);
  ES_CK(cudaGetLastError());
  ES_CK(cudaMemcpyAsync(y, n->act.back(), (size_t)count * n->cfg.out_dim * sizeof(float), cudaMemcpyDeviceToHost,
                        n->stream));
  ES_CK(cudaStreamSynchronize(n->stream));
  return FDTD_OK;
}

}  // extern "C"
