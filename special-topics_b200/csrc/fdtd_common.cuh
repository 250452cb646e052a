// fdtd_common.cuh -- shared device types and the per-step epilogue (port
// voltages + running far-field DFT) used by every field layout.
#pragma once
#include <type_traits>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fdtd {

constexpr int kMaxSources = 8;
constexpr int kMaxProbes = 8;

// Exactly rounded arithmetic that nvcc may not contract into FMA.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }

struct GridDims {
  int nx, ny, nz;
};

// The padded layout of fdtd_fused.cuh: one index for all six components.
struct PaddedGrid {
  int pitch, rows;
};

// Index of component c (0..5 = Hx Hy Hz Ex Ey Ez) at (i, j, k) in either layout.
__device__ __forceinline__ long long field_index(const GridDims& g, int c, int i, int j, int k) {
  const int rows = c == 1 || c == 3 || c == 5 ? g.ny + 1 : g.ny, cols = c >= 2 && c <= 4 ? g.nz + 1 : g.nz;
  return ((long long)i * rows + j) * cols + k;
}
__device__ __forceinline__ long long field_index(const PaddedGrid& g, int, int i, int j, int k) {
  return ((long long)i * g.rows + j) * g.pitch + k;
}

template <typename T>
struct Fields {
  T *Hx, *Hy, *Hz, *Ex, *Ey, *Ez;
};

// One CPML face.  Psi slots: x face 0=hyx 1=hzx 2=eyx 3=ezx; y face 0=hxy 1=hzy
// 2=ezy 3=exy; z face 0=hxz 1=hyz 2=exz 3=eyz (js_fdtd/src/cpml.js:147-448).
template <typename T>
struct Face {
  int nc;       // 0 when the face is not a CPML
  int m_start;  // first H index of the band along the face axis
  int e_start;  // first E index of the band along the face axis
  const T *b_e, *a_e, *b_m, *a_m;
  const float *inv_ke, *inv_km;  // 1/kappa per band cell (material-table problems only)
  T* psi[4];
  const T* cpsi[4];
};

struct SourceBox {
  int comp;                    // 0=Ex 1=Ey 2=Ez
  int i0, i1, j0, j1, k0, k1;  // inclusive component-index box
};

template <typename T>
struct Sources {
  int n;
  SourceBox box[kMaxSources];
  const T* cs[kMaxSources];    // per-cell source coefficient (Cexs / Ceys / Cezs)
  const T* wave[kMaxSources];  // voltage_per_e_field, one value per step
};

struct Probes {
  int n_v, n_i;
  int v_comp[kMaxProbes];
  int v_count[kMaxProbes];
  const int* v_idx[kMaxProbes];
  double v_csvf[kMaxProbes];
  int i_count[kMaxProbes];
  const int* i_comp[kMaxProbes];
  const int* i_idx[kMaxProbes];
  const double* i_w[kMaxProbes];
  double* V;   // [n_v][nsteps]
  double* I;   // [n_i][nsteps]
  int nsteps;
  int* status; // [0] = watchdog code, [1] = first non-finite step
};

struct FarField {
  int nFreq;
  int LI, LJ, LK, UI, UJ, UK;  // 0-based box planes
  int ni, nj, nk;              // box extents in cells
  const double* ph;            // [nsteps][nFreq][4] = cos_h, -sin_h, cos_e, -sin_e
  double* acc;                 // 24 arrays, each re[nFreq][sz] then im[nFreq][sz]
  long long off[24];
  long long sz[3];             // x-, y-, z-face point counts
  int kahan;                   // accumulators are FP32 (sum, compensation) pairs, not FP64
  int block;                   // > 0: steps per time block (samples buffered, accumulated by dft_flush)
  float* samples;              // [block][8][points] surface samples of the open block
  const int* done;             // steps already accumulated
};



// Lumped source on the cell this thread owns (sources.js:271-288).
template <typename T>
__device__ __forceinline__ void inject_sources(const Sources<T>& s, int comp, int i, int j, int k, int ts, T& e) {
  for (int q = 0; q < s.n; q++) {
    const SourceBox& b = s.box[q];
    if (b.comp == comp && i >= b.i0 && i <= b.i1 && j >= b.j0 && j <= b.j1 && k >= b.k0 && k <= b.k1) {
      const int ni = b.i1 - b.i0 + 1, nj = b.j1 - b.j0 + 1;
      const int n = ((k - b.k0) * nj + (j - b.j0)) * ni + (i - b.i0);
      e = add(e, mul(s.cs[q][n], s.wave[q][ts]));
    }
  }
}

template <typename T>
__device__ __forceinline__ const T* comp_ptr(const Fields<T>& f, int c) {
  return c == 0 ? f.Hx : c == 1 ? f.Hy : c == 2 ? f.Hz : c == 3 ? f.Ex : c == 4 ? f.Ey : f.Ez;
}

// Port current: ordered weighted sum of H samples (sampling.js:204-245).
template <typename T>
__device__ void current_probe(const Fields<T>& f, const Probes& pr, int q, int ts) {
  double sv = 0.0;
  const int n = pr.i_count[q];
  for (int m = 0; m < n; m++) {
    const double h = (double)comp_ptr(f, pr.i_comp[q][m])[pr.i_idx[q][m]];
    sv = add(sv, mul(pr.i_w[q][m], h));
  }
  pr.I[(long long)q * pr.nsteps + ts] = sv;
}

// Port voltage: V = Csvf * (sequential sum of the gap samples) (sampling.js:295-307).
template <typename T>
__device__ void voltage_probe(const Fields<T>& f, const Probes& pr, int q, int ts) {
  const T* F = comp_ptr(f, 3 + pr.v_comp[q]);
  double sum = 0.0;
  const int n = pr.v_count[q];
  for (int m = 0; m < n; m++) sum = add(sum, (double)F[pr.v_idx[q][m]]);
  const double v = mul(pr.v_csvf[q], sum);
  pr.V[(long long)q * pr.nsteps + ts] = v;
  if (!isfinite(v)) {
    atomicCAS(&pr.status[0], 0, 5);  // a wait that ran out stays the cause
    atomicMin(&pr.status[1], ts);
  }
}

// The same probes by a warp: the lanes fetch 32 samples at a time, every lane
// then adds them in list order (one thread's chain of dependent loads, an index
// and a sample per cell, took 15 us for a 15-cell port).
template <typename T>
__device__ void probe_warp(const Fields<T>& f, const Probes& pr, int q, int ts, int lane) {
  const bool volt = q < pr.n_v;
  const int u = volt ? q : q - pr.n_v, n = volt ? pr.v_count[u] : pr.i_count[u];
  double sum = 0.0;
  for (int m0 = 0; m0 < n; m0 += 32) {
    const int m = m0 + lane;
    double x = 0.0;
    if (m < n)
      x = volt ? (double)comp_ptr(f, 3 + pr.v_comp[u])[pr.v_idx[u][m]]
               : mul(pr.i_w[u][m], (double)comp_ptr(f, pr.i_comp[u][m])[pr.i_idx[u][m]]);
    for (int l = 0; l < min(32, n - m0); l++) sum = add(sum, __shfl_sync(0xffffffffu, x, l));
  }
  if (lane) return;
  if (volt) {
    const double v = mul(pr.v_csvf[u], sum);
    pr.V[(long long)u * pr.nsteps + ts] = v;
    if (!isfinite(v)) {
      atomicCAS(&pr.status[0], 0, 5);  // a wait that ran out stays the cause
      atomicMin(&pr.status[1], ts);
    }
  } else {
    pr.I[(long long)u * pr.nsteps + ts] = sum;
  }
}

// Names of the 24 accumulator arrays, in FarField::off order.
enum {
  CJYXP, CJZXP, CJYXN, CJZXN, CJXYP, CJZYP, CJXYN, CJZYN, CJXZP, CJYZP, CJXZN, CJYZN,
  CMYXP, CMZXP, CMYXN, CMZXN, CMXYP, CMZYP, CMXYN, CMZYN, CMXZP, CMYZP, CMXZN, CMYZN
};

// The 8 accumulator arrays a surface point feeds, in sample order, for the
// x-face (0), y-face (1) and z-face (2) point pairs.
__device__ __forceinline__ int sample_array(int group, int a) {
  static constexpr int tab[3][8] = {{CMYXP, CMZXP, CJYXP, CJZXP, CMYXN, CMZXN, CJYXN, CJZXN},
                                    {CMXYP, CMZYP, CJZYP, CJXYP, CMXYN, CMZYN, CJZYN, CJXYN},
                                    {CMXZP, CMYZP, CJXZP, CJYZP, CMXZN, CMYZN, CJXZN, CJYZN}};
  return tab[group][a];
}

// Time-blocked DFT: the epilogue stores a step's 8 samples per point in slot
// ts % block; this writes them into the running accumulators.
__device__ __forceinline__ void store_samples(const FarField& ff, long long t, int ts, const double* v) {
  const long long npts = ff.sz[0] + ff.sz[1] + ff.sz[2];
  float* s = ff.samples + (long long)(ts % ff.block) * 8 * npts + t;
#pragma unroll
  for (int a = 0; a < 8; a++) s[a * npts] = (float)v[a];
}

// One Kahan-compensated FP32 step: v = (sum, compensation), sum += x.
__device__ __forceinline__ void kahan_add(float2* v, float x) {
  float2 a = *v;
  const float y = __fsub_rn(x, a.y);
  const float t = __fadd_rn(a.x, y);
  a.y = __fsub_rn(__fsub_rn(t, a.x), y);
  a.x = t;
  *v = a;
}

// One step of the running DFT at a surface point: its 8 samples into the 8
// arrays of its group.  Every accumulator is loaded before the first is stored:
// in load-store pairs the chain of 8 memory latencies per frequency was the
// epilogue's time (20 us for 15,000 points; 8 us this way).
__device__ __forceinline__ void accumulate(const FarField& ff, int group, long long pt, int ts, const double* v) {
  const long long sz = ff.sz[group], im = ff.nFreq * sz;
  const double* ph = ff.ph + (long long)ts * ff.nFreq * 4;
  double* re[8];
#pragma unroll
  for (int a = 0; a < 8; a++) re[a] = ff.acc + ff.off[sample_array(group, a)] + pt;
  for (int m = 0; m < ff.nFreq; m++, ph += 4) {
    const double c[2] = {ph[0], ph[2]}, s[2] = {ph[1], ph[3]};  // H-time, E-time
    double r[8], i[8];
#pragma unroll
    for (int a = 0; a < 8; a++) {
      r[a] = re[a][0];
      i[a] = re[a][im];
    }
#pragma unroll
    for (int a = 0; a < 8; a++) {
      const int e = (a & 2) == 0;  // sample order: two magnetic (E-time), two electric (H-time), twice
      if (ff.kahan) {
        const float tf = (float)v[a];
        kahan_add(reinterpret_cast<float2*>(&r[a]), __fmul_rn((float)c[e], tf));
        kahan_add(reinterpret_cast<float2*>(&i[a]), __fmul_rn((float)s[e], tf));
      } else if (group == 2 && a == 2) {
        // zp Jx: the reference adds the Hx average (sample 3), then swaps it for
        // the Hy average in a second statement (farfield.js:211-225); keep both
        // roundings (with compensated FP32 only the net Hy term is added)
        const double r1 = add(r[a], mul(c[0], v[3])), i1 = add(i[a], mul(s[0], v[3]));
        r[a] = add(sub(r1, mul(c[0], v[3])), mul(c[0], v[2]));
        i[a] = add(sub(i1, mul(s[0], v[3])), mul(s[0], v[2]));
      } else {
        r[a] = add(r[a], mul(c[e], v[a]));
        i[a] = add(i[a], mul(s[e], v[a]));
      }
    }
#pragma unroll
    for (int a = 0; a < 8; a++) {
      re[a][0] = r[a];
      re[a][im] = i[a];
      re[a] += sz;
    }
  }
}

// ---------------------------------------------------------------------------
// Epilogue: running NF-FF DFT (farfield.js:90-248) on the six Huygens faces,
// then the port voltages and, in the padded layout (whose step has no mid
// launch), the port currents, a warp each.  One thread per surface point
// (xp/xn, yp/yn and zp/zn pairs share the point), looping over frequencies.
// ---------------------------------------------------------------------------
template <class G>
constexpr bool kWarpProbes = false;
template <>
constexpr bool kWarpProbes<PaddedGrid> = true;

// Threads of an epilogue in the padded layout.
inline long long epilogue_threads(long long points, int probes) { return ((points + 31) / 32 + probes) * 32; }

template <typename T, class G>
__device__ __forceinline__ void epilogue_thread(const Fields<T>& f, const G& g, const FarField& ff,
                                                const Probes& probes, int ts, long long t) {
  const long long nff = ff.nFreq > 0 ? ff.sz[0] + ff.sz[1] + ff.sz[2] : 0;
  if constexpr (kWarpProbes<G>) {  // whole warps after the points' last one
    const long long w = t / 32 - (nff + 31) / 32;
    if (w >= 0) {
      if (w < probes.n_v + probes.n_i) probe_warp(f, probes, (int)w, ts, (int)(t % 32));
      return;
    }
    if (t >= nff) return;
  } else if (t >= nff) {
    const long long q = t - nff;
    if (q < probes.n_v) voltage_probe(f, probes, (int)q, ts);
    return;
  }
#define HX(i, j, k) (double)f.Hx[field_index(g, 0, i, j, k)]
#define HY(i, j, k) (double)f.Hy[field_index(g, 1, i, j, k)]
#define HZ(i, j, k) (double)f.Hz[field_index(g, 2, i, j, k)]
#define EX(i, j, k) (double)f.Ex[field_index(g, 3, i, j, k)]
#define EY(i, j, k) (double)f.Ey[field_index(g, 4, i, j, k)]
#define EZ(i, j, k) (double)f.Ez[field_index(g, 5, i, j, k)]
  double v[8];
  int group;
  long long pt = t;
  if (t < ff.sz[0]) {
    group = 0;
    const int nj = (int)pt / ff.nk, nk = (int)pt % ff.nk;
    const int j0 = ff.LJ + nj, k0 = ff.LK + nk, UI = ff.UI, LI = ff.LI;
    v[0] = mul(0.5, add(EZ(UI, j0, k0), EZ(UI, j0 + 1, k0)));
    v[1] = mul(-0.5, add(EY(UI, j0, k0), EY(UI, j0, k0 + 1)));
    v[2] = mul(-0.25, add(add(add(HZ(UI, j0, k0), HZ(UI, j0, k0 + 1)), HZ(UI - 1, j0, k0)), HZ(UI - 1, j0, k0 + 1)));
    v[3] = mul(0.25, add(add(add(HY(UI, j0, k0), HY(UI, j0 + 1, k0)), HY(UI - 1, j0, k0)), HY(UI - 1, j0 + 1, k0)));
    v[4] = mul(-0.5, add(EZ(LI, j0, k0), EZ(LI, j0 + 1, k0)));
    v[5] = mul(0.5, add(EY(LI, j0, k0), EY(LI, j0, k0 + 1)));
    v[6] = mul(0.25, add(add(add(HZ(LI, j0, k0), HZ(LI, j0, k0 + 1)), HZ(LI - 1, j0, k0)), HZ(LI - 1, j0, k0 + 1)));
    v[7] = mul(-0.25, add(add(add(HY(LI, j0, k0), HY(LI, j0 + 1, k0)), HY(LI - 1, j0, k0)), HY(LI - 1, j0 + 1, k0)));
  } else if (t < ff.sz[0] + ff.sz[1]) {
    group = 1;
    pt = t - ff.sz[0];
    const int ni = (int)pt / ff.nk, nk = (int)pt % ff.nk;
    const int i0 = ff.LI + ni, k0 = ff.LK + nk, UJ = ff.UJ, LJ = ff.LJ;
    v[0] = mul(-0.5, add(EZ(i0, UJ, k0), EZ(i0 + 1, UJ, k0)));
    v[1] = mul(0.5, add(EX(i0, UJ, k0), EX(i0, UJ, k0 + 1)));
    v[2] = mul(-0.25, add(add(add(HX(i0, UJ, k0), HX(i0 + 1, UJ, k0)), HX(i0, UJ - 1, k0)), HX(i0 + 1, UJ - 1, k0)));
    v[3] = mul(0.25, add(add(add(HZ(i0, UJ, k0), HZ(i0, UJ, k0 + 1)), HZ(i0, UJ - 1, k0)), HZ(i0, UJ - 1, k0 + 1)));
    v[4] = mul(0.5, add(EZ(i0, LJ, k0), EZ(i0 + 1, LJ, k0)));
    v[5] = mul(-0.5, add(EX(i0, LJ, k0), EX(i0, LJ, k0 + 1)));
    v[6] = mul(0.25, add(add(add(HX(i0, LJ, k0), HX(i0 + 1, LJ, k0)), HX(i0, LJ - 1, k0)), HX(i0 + 1, LJ - 1, k0)));
    v[7] = mul(-0.25, add(add(add(HZ(i0, LJ, k0), HZ(i0, LJ, k0 + 1)), HZ(i0, LJ - 1, k0)), HZ(i0, LJ - 1, k0 + 1)));
  } else {
    group = 2;
    pt = t - ff.sz[0] - ff.sz[1];
    const int ni = (int)pt / ff.nj, nj = (int)pt % ff.nj;
    const int i0 = ff.LI + ni, j0 = ff.LJ + nj, UK = ff.UK, LK = ff.LK;
    v[0] = mul(0.5, add(EY(i0, j0, UK), EY(i0 + 1, j0, UK)));
    v[1] = mul(-0.5, add(EX(i0, j0, UK), EX(i0, j0 + 1, UK)));
    // zp: the reference's Jx is the Hy average, its Jy the Hx average
    v[3] = mul(0.25, add(add(add(HX(i0, j0, UK), HX(i0 + 1, j0, UK)), HX(i0, j0, UK - 1)), HX(i0 + 1, j0, UK - 1)));
    v[2] = mul(-0.25, add(add(add(HY(i0, j0, UK), HY(i0, j0 + 1, UK)), HY(i0, j0, UK - 1)), HY(i0, j0 + 1, UK - 1)));
    v[4] = mul(-0.5, add(EY(i0, j0, LK), EY(i0 + 1, j0, LK)));
    v[5] = mul(0.5, add(EX(i0, j0, LK), EX(i0, j0 + 1, LK)));
    v[6] = mul(0.25, add(add(add(HY(i0, j0, LK), HY(i0, j0 + 1, LK)), HY(i0, j0, LK - 1)), HY(i0, j0 + 1, LK - 1)));
    v[7] = mul(-0.25, add(add(add(HX(i0, j0, LK), HX(i0 + 1, j0, LK)), HX(i0, j0, LK - 1)), HX(i0 + 1, j0, LK - 1)));
  }
  if (ff.block)  // time-blocked: buffer the samples, dft_flush accumulates them
    store_samples(ff, t, ts, v);
  else
    accumulate(ff, group, pt, ts, v);
#undef HX
#undef HY
#undef HZ
#undef EX
#undef EY
#undef EZ
}

template <typename T>
__global__ void __launch_bounds__(256) k_epilogue(Fields<T> f, GridDims g, FarField ff, Probes probes,
                                                  const int* ts_ptr) {
  epilogue_thread<T>(f, g, ff, probes, *ts_ptr, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// Accumulates the buffered samples of the steps before `upto` that are not in
// the running DFT yet (from the block's first step, or *ff.done when a run
// started inside the block), steps in order.
//
// A block holds the accumulators of 32 surface points and NF frequencies in
// registers over all those steps (a warp per sample array, a point a thread), so
// an accumulator is read and written once and a sample is read once per NF
// frequencies; the phasors of kFlushSteps steps wait in shared memory.  One
// thread per (point, frequency), which read every sample and phasor again for
// each frequency, was bound by those loads: 16 steps of 93 k point pairs at 64
// frequencies took 888 us, now 341 us (of which the accumulators' own traffic is
// 235 us).  Two points a thread, or 4 or 16 frequencies, leave too few warps or
// loads in flight (484, 460, 371 us); few frequencies take a smaller NF, whose
// blocks need fewer registers.
constexpr int kFlushPoints = 32, kFlushSteps = 32;
__host__ __device__ inline int flush_freqs(int freqs) { return freqs <= 2 ? 2 : freqs <= 4 ? 4 : 8; }  // NF
__host__ __device__ inline long long flush_blocks(long long points, int freqs) {
  const int nf = flush_freqs(freqs);
  return (points + kFlushPoints - 1) / kFlushPoints * ((freqs + nf - 1) / nf);
}

template <bool KAHAN, int NF>
__device__ __forceinline__ void dft_flush_block(const FarField& ff, int upto, long long b) {
  using A = std::conditional_t<KAHAN, float2, double>;   // an accumulator
  using P = std::conditional_t<KAHAN, float2, double2>;  // a phasor
  __shared__ P ph[kFlushSteps][NF][2];          // H-time, E-time
  const long long npts = ff.sz[0] + ff.sz[1] + ff.sz[2];
  const int chunks = (ff.nFreq + NF - 1) / NF;
  const int m0 = (int)(b % chunks) * NF, nf = min(NF, ff.nFreq - m0);
  const int a = threadIdx.x / 32;
  const int first = (upto - 1) / ff.block * ff.block, from = max(*ff.done, first);
  const long long t = b / chunks * kFlushPoints + threadIdx.x % 32;
  const bool has = t < npts;
  const int group = t < ff.sz[0] ? 0 : t < ff.sz[0] + ff.sz[1] ? 1 : 2;
  const long long sz = ff.sz[group];
  A* const acc = reinterpret_cast<A*>(ff.acc + ff.off[sample_array(group, a)]) + m0 * sz +
                 (group == 0 ? t : group == 1 ? t - ff.sz[0] : t - ff.sz[0] - ff.sz[1]);
  A re[NF], im[NF];
#pragma unroll
  for (int f = 0; f < NF; f++)
    if (has && f < nf) {
      re[f] = acc[f * sz];
      im[f] = acc[(ff.nFreq + f) * sz];
    }
  const int e = (a & 2) == 0;  // magnetic currents take the E-time phasor
  for (int s0 = from; s0 < upto; s0 += kFlushSteps) {
    const int ns = min(kFlushSteps, upto - s0);
    __syncthreads();
    for (int w = threadIdx.x; w < ns * NF * 2; w += 256) {
      const int s = w / (2 * NF), f = w / 2 % NF;
      if (f < nf) {
        const double* src = ff.ph + ((long long)(s0 + s) * ff.nFreq + m0 + f) * 4 + w % 2 * 2;
        ph[s][f][w % 2].x = src[0];
        ph[s][f][w % 2].y = src[1];
      }
    }
    __syncthreads();
    const float* smp = ff.samples + ((long long)(s0 - first) * 8 + a) * npts + t;
#pragma unroll 8
    for (int s = 0; s < ns; s++) {
      const float v = has ? smp[s * 8 * npts] : 0.0f;
#pragma unroll
      for (int f = 0; f < NF; f++)
        if (f < nf) {
          const P c = ph[s][f][e];
          if constexpr (KAHAN) {
            kahan_add(&re[f], __fmul_rn(c.x, v));
            kahan_add(&im[f], __fmul_rn(c.y, v));
          } else {
            re[f] += c.x * v;
            im[f] += c.y * v;
          }
        }
    }
  }
#pragma unroll
  for (int f = 0; f < NF; f++)
    if (has && f < nf) {
      acc[f * sz] = re[f];
      acc[(ff.nFreq + f) * sz] = im[f];
    }
}

// With NF as flush_blocks counts the blocks.
template <bool KAHAN>
__device__ __forceinline__ void dft_flush_any(const FarField& ff, int upto, long long b) {
  const int nf = flush_freqs(ff.nFreq);
  if (nf == 2)
    dft_flush_block<KAHAN, 2>(ff, upto, b);
  else if (nf == 4)
    dft_flush_block<KAHAN, 4>(ff, upto, b);
  else
    dft_flush_block<KAHAN, 8>(ff, upto, b);
}

// The steps a flush covers: upto >= 0, the end of a run (nothing to do when a
// block closed there); -1, a launch inside every step of a graph, which acts
// only when the step just finished, *ts_ptr, closes a block; -2, the same where
// *ts_ptr is the step after it.
__device__ __forceinline__ bool flush_upto(const FarField& ff, const int* ts_ptr, int& upto) {
  if (ff.block <= 0) return false;
  if (upto >= 0) return upto % ff.block != 0;
  upto = *ts_ptr + (upto == -1 ? 1 : 0);
  return upto % ff.block == 0;
}

// 256 threads; flush_blocks() of them.
template <bool KAHAN, int NF>
static __global__ void __launch_bounds__(256) k_dft_flush(FarField ff, const int* ts_ptr, int upto) {
  if (flush_upto(ff, ts_ptr, upto)) dft_flush_block<KAHAN, NF>(ff, upto, blockIdx.x);
}
template <int NF>
cudaError_t dft_flush_launch(const FarField& ff, const int* ts_ptr, int upto, cudaStream_t st) {
  const unsigned n = (unsigned)flush_blocks(ff.sz[0] + ff.sz[1] + ff.sz[2], ff.nFreq);
  if (ff.kahan)
    k_dft_flush<true, NF><<<n, 256, 0, st>>>(ff, ts_ptr, upto);
  else
    k_dft_flush<false, NF><<<n, 256, 0, st>>>(ff, ts_ptr, upto);
  return cudaGetLastError();
}
inline cudaError_t dft_flush(const FarField& ff, const int* ts_ptr, int upto, cudaStream_t st) {
  const int nf = flush_freqs(ff.nFreq);
  return nf == 2 ? dft_flush_launch<2>(ff, ts_ptr, upto, st)
         : nf == 4 ? dft_flush_launch<4>(ff, ts_ptr, upto, st)
                   : dft_flush_launch<8>(ff, ts_ptr, upto, st);
}

}  // namespace fdtd
