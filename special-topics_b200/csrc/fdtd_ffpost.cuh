// fdtd_ffpost.cuh -- far-field post-processing on the device: radiated power
// and directivity from the running NF-FF DFT accumulators
// (js_fdtd/src/farfield.js:257-607, restated in postproc.py for the host).
//
// Radiated power: per frequency, the surface integral of the Poynting flux
// of the equivalent currents, sum over faces and points of
// sign * area * (M1.J1 - M2.J2) / 2 (farfield.js:257-325).
//
// Directivity: for each frequency and direction (theta, phi), the radiation
// vectors N = sum J exp(jk r'.r) dA and L = sum M exp(jk r'.r) dA over the six
// faces, projected on theta/phi (farfield.js:328-607), then
// D_theta = k^2 |L_phi + eta N_theta|^2 / (8 pi eta P_rad), and D_phi alike
// with |L_theta - eta N_phi|^2.
//
// Face points lie on a regular grid, so along a row of points the phase factor
// advances by one complex multiply per point; one sincos starts each run.  The
// points of a row are taken in pairs about its middle: with u and v the sum and
// the difference of a pair's currents, the pair adds cos(x) u + j sin(x) v, half
// the multiplications of two single points.  All of it is FP64 arithmetic on the
// CUDA cores, and that bounds it, so the rows are summed where they need be:
//   * along z the phase depends on theta alone.  The rows of the x and y faces
//     run along z, so k_ff_rows sums each of them once per distinct theta, and
//     a direction (k_ff_pattern) sums the row sums;
//   * the rows of the z faces run along y, and k_ff_zrows sums them for every
//     direction, both faces together as they share the phase in the plane.
// Summing every point for every direction (4.4 ms for up to 2,000 directions,
// 13.8 ms for 16,380, on a 13 x 110 x 110 box at 12 frequencies) was slower for
// one direction (0.26 ms), for a 2-degree grid (2.4 ms, of which the kernels 1.3)
// and for 16,000 directions without a theta in common (9.6 ms).
#pragma once
#include "fdtd_common.cuh"

namespace fdtd {

struct FFPost {
  const double* acc;
  long long off[24];
  long long sz[3];
  int nFreq;
  int ni, nj, nk;        // box extents in cells
  double pos0[3];        // first face point along x, y, z relative to the box centre
  double face[3][2];     // face planes (p, n) along x, y, z relative to the centre
  double d[3];           // cell sizes
};

constexpr double kC0 = 2.99792458e8;
constexpr double kEta0 = 376.73031346177066;
constexpr double kPi = 3.141592653589793;

// Accumulator names of face f (0..5 = xp xn yp yn zp zn): J1, J2, M1, M2.
__device__ __forceinline__ void face_arrays(int f, int& j1, int& j2, int& m1, int& m2) {
  static constexpr int tab[6][4] = {{CJYXP, CJZXP, CMYXP, CMZXP}, {CJYXN, CJZXN, CMYXN, CMZXN},
                                    {CJXYP, CJZYP, CMXYP, CMZYP}, {CJXYN, CJZYN, CMXYN, CMZYN},
                                    {CJXZP, CJYZP, CMXZP, CMYZP}, {CJXZN, CJYZN, CMXZN, CMYZN}};
  j1 = tab[f][0];
  j2 = tab[f][1];
  m1 = tab[f][2];
  m2 = tab[f][3];
}

// Compensated FP32 accumulator pairs (sum, compensation) -> FP64 values.
__global__ void k_kahan_to_f64(const double* __restrict__ acc, double* __restrict__ out, long long n) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const float2 v = reinterpret_cast<const float2*>(acc)[q];
  out[q] = (double)v.x - (double)v.y;
}

// Radiated power: the sum of each face pair's points, a block per (frequency,
// term), fixed-order reduction; k_ff_power_sum adds a frequency's terms.
__global__ void __launch_bounds__(256) k_ff_power(FFPost P, double* __restrict__ part) {
  __shared__ double red[256];
  const int f = blockIdx.x, t = blockIdx.y;
  // (face, area, M1, J1, M2, J2, sign) as farfield.js:257-325 pairs them
  const int terms[6][5] = {{CMYZP, CJXZP, CMXZP, CJYZP, 1},  {CMYZN, CJXZN, CMXZN, CJYZN, -1},
                           {CMXYP, CJZYP, CMZYP, CJXYP, 1},  {CMXYN, CJZYN, CMZYN, CJXYN, -1},
                           {CMZXP, CJYXP, CMYXP, CJZXP, 1},  {CMZXN, CJYXN, CMYXN, CJZXN, -1}};
  const int a = 2 - t / 2;
  const long long n = P.sz[a];
  const double area = a == 0 ? P.d[1] * P.d[2] : a == 1 ? P.d[0] * P.d[2] : P.d[0] * P.d[1];
  const double* m1 = P.acc + P.off[terms[t][0]] + (long long)f * n;
  const double* j1 = P.acc + P.off[terms[t][1]] + (long long)f * n;
  const double* m2 = P.acc + P.off[terms[t][2]] + (long long)f * n;
  const double* j2 = P.acc + P.off[terms[t][3]] + (long long)f * n;
  const long long im = (long long)P.nFreq * n;  // imaginary parts follow the real ones
  double fs = 0.0;
#pragma unroll 4
  for (long long p = threadIdx.x; p < n; p += 256)
    fs += m1[p] * j1[p] + m1[p + im] * j1[p + im] - m2[p] * j2[p] - m2[p + im] * j2[p + im];
  red[threadIdx.x] = terms[t][4] * area * fs;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[f * 6 + t] = red[0];
}
__global__ void k_ff_power_sum(const double* __restrict__ part, int F, double* __restrict__ radp) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= F) return;
  double s = 0.0;
  for (int t = 0; t < 6; t++) s += part[f * 6 + t];
  radp[f] = 0.5 * s;
}

struct Cplx {
  double re, im;
};
__device__ __forceinline__ Cplx cmul(Cplx a, Cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ void cmac(Cplx& s, Cplx e, double re, double im) {
  s.re += e.re * re - e.im * im;
  s.im += e.re * im + e.im * re;
}
__device__ __forceinline__ Cplx cexpj(double phase) {
  double s, c;
  sincos(phase, &s, &c);
  return {c, s};
}

// Rows of points along axis `n` of a face, summed for one thread's directions.
// Stages the pairs of `rows` rows (the same row of that many faces) in shared
// memory and adds their sums, phases relative to the rows' middles.
constexpr int kFFPairs = 64;  // pairs staged at a time
template <int ANG, int ROWS>
struct FFRows {
  double (*sm)[kFFPairs][16];  // [ROWS]: u then v of J1 J2 M1 M2 (re, im)
  // arr[row][w]: current w of the row's first point; its imaginary part `im` on
  __device__ __forceinline__ void sum(const double* const (*arr)[4], long long im, int nn, const double* kx, double d,
                                      Cplx (*S)[ROWS][4]) const {
    const int half = nn / 2, odd = nn & 1, np = half + odd;
    for (int t0 = 0; t0 < np; t0 += kFFPairs) {
      const int cnt = min(kFFPairs, np - t0);
      __syncthreads();
      for (int x = threadIdx.x; x < ROWS * 8 * cnt; x += blockDim.x) {
        const int t = x % cnt, w = x / cnt % 8, row = x / cnt / 8;
        const double* A = arr[row][w / 2] + (w & 1 ? im : 0);
        const int hi = half + t0 + t;          // the pair's upper point; of an odd row the middle comes first
        const int lo = nn - 1 - hi;
        const double p = A[hi], m = lo == hi ? 0.0 : A[lo];
        sm[row][t][w] = p + m;
        sm[row][t][8 + w] = lo == hi ? 0.0 : p - m;
      }
      __syncthreads();
      Cplx e[ANG], step[ANG];
#pragma unroll
      for (int q = 0; q < ANG; q++) {
        e[q] = cexpj(kx[q] * d * (t0 + (odd ? 0.0 : 0.5)));
        step[q] = cexpj(kx[q] * d);
      }
      for (int t = 0; t < cnt; t++) {
#pragma unroll
        for (int row = 0; row < ROWS; row++)
#pragma unroll
          for (int w = 0; w < 4; w++) {
            const double2 u = *reinterpret_cast<const double2*>(&sm[row][t][2 * w]);
            const double2 v = *reinterpret_cast<const double2*>(&sm[row][t][8 + 2 * w]);
#pragma unroll
            for (int q = 0; q < ANG; q++) {
              Cplx& s = S[q][row][w];
              s.re += e[q].re * u.x - e[q].im * v.y;
              s.im += e[q].re * u.y + e[q].im * v.x;
            }
          }
#pragma unroll
        for (int q = 0; q < ANG; q++) e[q] = cmul(e[q], step[q]);
      }
    }
  }
};

// Workspace of the row sums.
struct FFSums {
  int f0;             // first frequency
  int nth;            // distinct thetas of the directions
  const double* cth;  // their cosines
  const int* ith;     // [directions] which of them
  const double *theta, *phi;
  int nang;           // directions
  double* rows;       // [freq][row][8][theta]: rows of xp, xn (nj each), yp, yn (ni each)
  double* z;          // [freq][part][8][direction]: the z faces' sums
  int parts;          // each of a part of their rows
};

// A block per (row, run of thetas, frequency); the rows along the grid's first axis,
// as a long thin problem has more of them than the others hold (65,535).
constexpr int kFFRowThreads = 64, kFFRowAng = 2;
__global__ void __launch_bounds__(kFFRowThreads)
    k_ff_rows(FFPost P, FFSums W, const double* __restrict__ freqs) {
  __shared__ __align__(16) double sm[1][kFFPairs][16];
  const int f = W.f0 + blockIdx.z;
  int r = blockIdx.x, fc = 0;
  for (; fc < 3 && r >= (fc < 2 ? P.nj : P.ni); fc++) r -= fc < 2 ? P.nj : P.ni;
  const int a = fc / 2, nn = P.nk;
  const double k = 2.0 * kPi * freqs[f] / kC0;
  int c[4];
  face_arrays(fc, c[0], c[1], c[2], c[3]);
  const double* arr[1][4];
  for (int w = 0; w < 4; w++) arr[0][w] = P.acc + P.off[c[w]] + (long long)f * P.sz[a] + (long long)r * nn;
  double kx[kFFRowAng];
  Cplx S[kFFRowAng][1][4] = {};
  const int th0 = blockIdx.y * kFFRowThreads * kFFRowAng + threadIdx.x;
  for (int q = 0; q < kFFRowAng; q++) {
    const int th = th0 + q * kFFRowThreads;
    kx[q] = th < W.nth ? k * W.cth[th] : 0.0;
  }
  FFRows<kFFRowAng, 1>{sm}.sum(arr, (long long)P.nFreq * P.sz[a], nn, kx, P.d[2], S);
  const int R = 2 * (P.ni + P.nj);
  for (int q = 0; q < kFFRowAng; q++) {
    const int th = th0 + q * kFFRowThreads;
    if (th >= W.nth) continue;
    const Cplx mid = cexpj(kx[q] * (P.pos0[2] + 0.5 * (nn - 1) * P.d[2]));
    double* out = W.rows + ((long long)blockIdx.z * R + blockIdx.x) * 8 * W.nth + th;
    for (int w = 0; w < 4; w++) {
      const Cplx v = cmul(mid, S[q][0][w]);
      out[2 * w * (long long)W.nth] = v.re;
      out[(2 * w + 1) * (long long)W.nth] = v.im;
    }
  }
}

// Directions: (sin theta cos phi, sin theta sin phi, cos theta).
constexpr int kFFZThreads = 64, kFFZAng = 2;
__global__ void __launch_bounds__(kFFZThreads) k_ff_zrows(FFPost P, FFSums W, const double* __restrict__ freqs) {
  __shared__ __align__(16) double sm[2][kFFPairs][16];
  const int f = W.f0 + blockIdx.z, part = blockIdx.y, nn = P.nj;
  const double k = 2.0 * kPi * freqs[f] / kC0;
  double dx[kFFZAng], kx[kFFZAng];
  Cplx side[kFFZAng][2];
  int c[2][4];
  for (int s = 0; s < 2; s++) face_arrays(4 + s, c[s][0], c[s][1], c[s][2], c[s][3]);
  const int ang0 = blockIdx.x * kFFZThreads * kFFZAng + threadIdx.x;
  for (int q = 0; q < kFFZAng; q++) {
    const int ang = ang0 + q * kFFZThreads;
    const double th = ang < W.nang ? W.theta[ang] : 0.0, ph = ang < W.nang ? W.phi[ang] : 0.0;
    double st, ct, sp, cp;
    sincos(th, &st, &ct);
    sincos(ph, &sp, &cp);
    const double dy = st * sp;
    dx[q] = st * cp;
    kx[q] = k * dy;
    for (int s = 0; s < 2; s++) side[q][s] = cexpj(k * (P.face[2][s] * ct + (P.pos0[1] + 0.5 * (nn - 1) * P.d[1]) * dy));
  }
  Cplx T[kFFZAng][4] = {};
  const int r0 = (int)((long long)part * P.ni / W.parts), r1 = (int)((long long)(part + 1) * P.ni / W.parts);
  for (int r = r0; r < r1; r++) {
    const double* arr[2][4];
    for (int s = 0; s < 2; s++)
      for (int w = 0; w < 4; w++) arr[s][w] = P.acc + P.off[c[s][w]] + (long long)f * P.sz[2] + (long long)r * nn;
    Cplx S[kFFZAng][2][4] = {};
    FFRows<kFFZAng, 2>{sm}.sum(arr, (long long)P.nFreq * P.sz[2], nn, kx, P.d[1], S);
    for (int q = 0; q < kFFZAng; q++) {
      const Cplx e = cexpj(k * (P.pos0[0] + r * P.d[0]) * dx[q]);
      for (int s = 0; s < 2; s++) {
        const Cplx es = cmul(e, side[q][s]);
        for (int w = 0; w < 4; w++) cmac(T[q][w], es, S[q][s][w].re, S[q][s][w].im);
      }
    }
  }
  for (int q = 0; q < kFFZAng; q++) {
    const int ang = ang0 + q * kFFZThreads;
    if (ang >= W.nang) continue;
    double* out = W.z + ((long long)blockIdx.z * W.parts + part) * 8 * W.nang + ang;
    for (int w = 0; w < 4; w++) {
      out[2 * w * (long long)W.nang] = T[q][w].re;
      out[(2 * w + 1) * (long long)W.nang] = T[q][w].im;
    }
  }
}

// A direction's radiation vectors.
struct FFVectors {
  double st, ct, sp, cp;
  Cplx Nt{0.0, 0.0}, Np{0.0, 0.0}, Lt{0.0, 0.0}, Lp{0.0, 0.0};
  // adds a face's sums, or several of one axis's (farfield.js:328-607)
  __device__ __forceinline__ void add(int a, double A, const Cplx* S) {
    const Cplx J1 = S[0], J2 = S[1], M1 = S[2], M2 = S[3];
    double t1, t2, p1, p2;  // N_theta = t1 J1 + t2 J2, N_phi = p1 J1 + p2 J2 (same for L with M)
    if (a == 0) {           // J1 = Jy, J2 = Jz
      t1 = A * ct * sp; t2 = -A * st; p1 = A * cp; p2 = 0.0;
    } else if (a == 1) {    // J1 = Jx, J2 = Jz
      t1 = A * ct * cp; t2 = -A * st; p1 = -A * sp; p2 = 0.0;
    } else {                // J1 = Jx, J2 = Jy
      t1 = A * ct * cp; t2 = A * ct * sp; p1 = -A * sp; p2 = A * cp;
    }
    Nt.re += t1 * J1.re + t2 * J2.re;
    Nt.im += t1 * J1.im + t2 * J2.im;
    Np.re += p1 * J1.re + p2 * J2.re;
    Np.im += p1 * J1.im + p2 * J2.im;
    Lt.re += t1 * M1.re + t2 * M2.re;
    Lt.im += t1 * M1.im + t2 * M2.im;
    Lp.re += p1 * M1.re + p2 * M2.re;
    Lp.im += p1 * M1.im + p2 * M2.im;
  }
  __device__ __forceinline__ void out(double k, double radp, double& dth, double& dph) const {
    const double scale = k * k / (8.0 * kPi * kEta0 * radp);
    const double ar = Lp.re + kEta0 * Nt.re, ai = Lp.im + kEta0 * Nt.im;
    const double br = Lt.re - kEta0 * Np.re, bi = Lt.im - kEta0 * Np.im;
    dth = scale * (ar * ar + ai * ai);
    dph = scale * (br * br + bi * bi);
  }
};

// Directions from the row sums: one thread per (direction, frequency).  dth and
// dph: [freq][stride], from the first direction.
__global__ void __launch_bounds__(128)
    k_ff_pattern(FFPost P, FFSums W, const double* __restrict__ freqs, const double* __restrict__ radp, long long stride,
                 double* __restrict__ dth, double* __restrict__ dph) {
  const int f = W.f0 + blockIdx.y, ang = blockIdx.x * 128 + threadIdx.x, nang = W.nang;
  if (ang >= nang) return;
  const double k = 2.0 * kPi * freqs[f] / kC0;
  FFVectors V;
  sincos(W.theta[ang], &V.st, &V.ct);
  sincos(W.phi[ang], &V.sp, &V.cp);
  const double dir[2] = {V.st * V.cp, V.st * V.sp};
  const double* g = W.rows + (long long)blockIdx.y * 2 * (P.ni + P.nj) * 8 * W.nth + W.ith[ang];
  for (int fc = 0; fc < 4; fc++) {
    const int a = fc / 2, o = 1 - a, no = a == 0 ? P.nj : P.ni;
    Cplx S[4] = {};
    const Cplx step = cexpj(k * P.d[o] * dir[o]);
    for (int r0 = 0; r0 < no; r0 += 64) {
      Cplx e = cexpj(k * (P.face[a][fc % 2] * dir[a] + (P.pos0[o] + r0 * P.d[o]) * dir[o]));
      const int r1 = min(r0 + 64, no);
#pragma unroll 1  // the loads of more rows cost registers, and so warps: 430 us for 341 when unrolled by two
      for (int r = r0; r < r1; r++) {
#pragma unroll
        for (int w = 0; w < 4; w++)
          cmac(S[w], e, __ldg(g + 2 * w * (long long)W.nth), __ldg(g + (2 * w + 1) * (long long)W.nth));
        e = cmul(e, step);
        g += 8 * (long long)W.nth;
      }
    }
    V.add(a, a == 0 ? P.d[1] * P.d[2] : P.d[0] * P.d[2], S);
  }
  Cplx S[4] = {};
  for (int part = 0; part < W.parts; part++) {
    const double* z = W.z + ((long long)blockIdx.y * W.parts + part) * 8 * nang + ang;
    for (int w = 0; w < 4; w++) {
      S[w].re += z[2 * w * (long long)nang];
      S[w].im += z[(2 * w + 1) * (long long)nang];
    }
  }
  V.add(2, P.d[0] * P.d[1], S);
  V.out(k, radp[f], dth[f * stride + ang], dph[f * stride + ang]);
}

}  // namespace fdtd
