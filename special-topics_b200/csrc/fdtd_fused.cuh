// fdtd_fused.cuh -- one launch per time step: the H and the E half-step of
// fdtd_step.cuh in a single pass over the fields.
//
// What bounds the step is memory traffic, the latency of the loads and the
// integer work around them.  Two half-step launches read every field value
// twice and write it once, and in the reference layout (rows of nz or nz + 1
// values) every component has its own index and no row is aligned.  Here
//   * the state lives in two padded copies.  A step reads one and writes the
//     other, so a block may recompute the H values its tile's E update needs
//     from its neighbours (one row, one column, one x plane) instead of waiting
//     for them, and each field is read once and written once;
//   * all six components share one index (rows of `pitch` values, 32-byte
//     aligned), so the tiles of a plane come into shared memory by tensor-map
//     copies, kFusedStages planes deep, with no per-thread loads or addresses,
//     and zeros where the grid ends;
//   * a 16-bit class per cell names its coefficients in a table.  A class is
//     what a cell's coefficients are apart from the CPML kappa: it holds the
//     18 update coefficients, the 12 CPsi, and, for each of the 12 curl
//     coefficients, its values along the band positions of its axis.  Classes
//     and table are filled on the device from the problem's own coefficients
//     and every cell is compared with its lookup bit for bit, so the table form
//     loses nothing.  Values a step leaves alone, or that do not exist at a
//     cell, are classes too (coefficients 1,0,0 and 0,0,0); held values are kept
//     by a select besides, as 0 times an infinity is not 0.  A thread keeps its
//     coefficients in registers along x and reads the table only where the class
//     changes.
// The arithmetic of a value is that of fdtd_step.cuh, in the same order.
//
// A block owns six rows of up to 72 columns (with a halo row and, where a row
// takes more than one tile, a halo group of columns), one thread per group of V
// columns and row, and walks its chunk of x planes.  Per plane: H of the tile
// and its halo, exchanged through shared memory; one barrier; E of the owned
// cells from the new H.
//
// Measured per step in a captured run, before (two half-step launches, a mid
// launch and an epilogue) and now, on one B200:
//   39 x 136 x 136 antenna: material table 52.9 -> 32.0 us, FP64 103.5 -> 65.6 us
//   97 x 131 x 118, FP32 cell by cell: 114.9 -> 66 us
//   256^3: material table 0.403 -> 0.374 ms, FP64 0.873 -> 0.55 ms
//   512 x 512 x 640, material table: 3.22 -> 2.42 ms; without CPML 2.89 -> 1.87,
//   of which the step 1.71 ms: 50 bytes a cell at 4.9 TB/s.
// Of these the selects that keep held values and a slab's other columns as they are
// (0 times an infinity is not 0) cost 0.4 to 1%.
#pragma once
#include <cuda.h>

#include "fdtd_common.cuh"
#include "fdtd_step.cuh"

namespace fdtd {

// Tile shape: 7 rows (one of them halo) of up to 72 columns.  A tile row holds
// 80 values: four columns before the first owned one where there is a halo
// column (tensor copies start on 16 bytes), the owned ones, and four after.
// Rows and tiles have fixed sizes, so every shared-memory access of the step
// has a constant offset.  A thread owns a group of V consecutive columns: 2
// floats or 1 double.  Two floats halve the integer work, the branches and the
// shared-memory instructions per cell, which is what one float per thread was
// bound by; two doubles do not fit the registers.
constexpr int kFusedStages = 4;
constexpr int kPsiAhead = 3;                      // planes between a Psi line's prefetch and its use
constexpr int kTileW = 80, kTileRows = 7, kTileCols = 72;
constexpr int kTileE = (kTileRows + 1) * kTileW;  // values of an E tile
constexpr int kTileH = 576;                       // of an H tile: 7 rows, to a 128-byte boundary
constexpr int kTileC = 88;                        // classes of a tile row, from a multiple of eight columns
constexpr int kTileCBytes = 1280;                 // of a class tile: 7 rows, to a 128-byte boundary
constexpr int kFusedSmemValues =
    kFusedStages * 3 * (kTileE + kTileH) + 2 * 3 * kTileH + 4 * (kTileRows + 1 + kTileW);

template <typename T>
struct FusedShape {
  static constexpr int V = 8 / (int)sizeof(T);
  static constexpr int kThreads = 512 / V;
  static constexpr int kBlocks = V;  // per SM: 128 registers a thread
};

template <typename T>
__host__ __device__ constexpr int fused_smem_bytes() {
  return kFusedStages * (kTileCBytes + 8) + kFusedSmemValues * (int)sizeof(T);
}

// A group's values.
template <typename T, int V = FusedShape<T>::V>
struct Vec {
  T v[V];
};
template <typename T>
__device__ __forceinline__ Vec<T> ldv(const T* p) {  // global, read-only for the launch
  Vec<T> o;
  if constexpr (sizeof(T) == 4) {
    const float2 a = __ldg(reinterpret_cast<const float2*>(p));
    o.v[0] = a.x, o.v[1] = a.y;
  } else {
    o.v[0] = __ldg(p);
  }
  return o;
}
template <typename T>
__device__ __forceinline__ Vec<T> ldw(const T* p) {  // shared memory, and arrays the launch also writes
  Vec<T> o;
  if constexpr (sizeof(T) == 4) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    o.v[0] = a.x, o.v[1] = a.y;
  } else {
    o.v[0] = *p;
  }
  return o;
}
template <typename T>
__device__ __forceinline__ void stv(T* p, const Vec<T>& a) {
  if constexpr (sizeof(T) == 4)
    *reinterpret_cast<float2*>(p) = make_float2(a.v[0], a.v[1]);
  else
    *p = a.v[0];
}
template <typename T>
__device__ __forceinline__ Vec<T> vsub(const Vec<T>& a, const Vec<T>& b) {
  Vec<T> o;
#pragma unroll
  for (int q = 0; q < FusedShape<T>::V; q++) o.v[q] = sub(a.v[q], b.v[q]);
  return o;
}
// differences along k: v[q+1] - v[q], `next` after the last; v[q] - v[q-1], `prev` before the first
template <typename T>
__device__ __forceinline__ Vec<T> vdiff_up(const Vec<T>& a, T next) {
  constexpr int V = FusedShape<T>::V;
  Vec<T> o;
#pragma unroll
  for (int q = 0; q < V; q++) o.v[q] = sub(q + 1 < V ? a.v[(q + 1) % V] : next, a.v[q]);
  return o;
}
template <typename T>
__device__ __forceinline__ Vec<T> vdiff_dn(const Vec<T>& a, T prev) {
  constexpr int V = FusedShape<T>::V;
  Vec<T> o;
#pragma unroll
  for (int q = 0; q < V; q++) o.v[q] = sub(a.v[q], q > 0 ? a.v[(q + V - 1) % V] : prev);
  return o;
}

// c0, c1, c2 of a component.
template <typename T>
struct Row {
  T c0, c1, c2;
};
__device__ __forceinline__ Row<float> ld_row(const float* row, int comp) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(row) + comp);
  return {a.x, a.y, a.z};
}
__device__ __forceinline__ Row<double> ld_row(const double* row, int comp) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(row) + 2 * comp);
  return {a.x, a.y, __ldg(row + 4 * comp + 2)};
}

// The CPML bands of one axis in the padded layout: the n face's cells, then the
// p face's.  Psi of the x axis: [band cell][j][k], of y: [i][band cell][k], of
// z: [i][j][slab cell], where a slab is a band widened to whole groups (zero
// profiles outside the band).  H Psi is recomputed in the halo, so it has two copies
// like the fields; E Psi has one reader and writer and is updated in place.
// (One array for both faces: no pointer of the step depends on the face.)
template <typename T>
struct FusedAxis {
  int nc[2][2], start[2][2];  // [H, E][n, p face]: cells and first position of the band (z: of the slab)
  int nb;                     // cells of both faces (z: room for either half-step's slabs)
  const T* phi[2];         // H Psi (slots 0, 1 of the faces) of the copy read
  T* pho[2];               // and of the copy written
  T* pe[2];                // E Psi (slots 2, 3)
  const T* prof[2][2];     // [H, E][b, a] over the whole axis; outside the bands a is 0 and b -0
};

// Layout of a class's table row, in values: the six components' (c0, c1, c2, -)
// away from the bands, the 12 CPsi (component c: 2 c for the c1 axis, 2 c + 1
// for the c2 axis), then for each axis the band values of its four curl
// coefficients (slots 0, 1 = H, 2, 3 = E, as the face's Psi slots), one per
// band position (n face, then p face; along z one per slab cell).
struct ClassRow {
  int stride;
  int o[3];   // offset of axis a's values
  int n[3];   // values per coefficient: the axis's nb
};
constexpr int kRowCpsi = 24, kRowBands = 36;

template <typename T>
struct FusedParams {
  int nx, ny, nz;
  int pitch;               // values per row
  unsigned plane;          // values per x plane
  CUtensorMap map[7];      // the copy read: Hx Hy Hz Ex Ey Ez, and the classes, as (k, j, i) tiles
  const T* fi[6];          // its arrays
  T* fo[6];                // the copy written
  const unsigned short* cls;
  const T* tab;            // class table, see ClassRow
  ClassRow row;
  FusedAxis<T> axis[3];
  const int* ts;           // step index, see k_fused
  int* ts_next;
  Sources<T> src;
  int* fault;              // the handle's status code word
  int x_wall;
  int rk, halo_k;          // threads along k, 1: column 0 of a tile is halo
  int tk, tj, tx;          // tiles along k, j, x
  int slow_j[2], slow_k[2];  // tiles at the low and high end that meet a y band, a z band
};

// Band cell of axis position `pos` for the H or E update, -1 outside the bands.
template <bool ELECTRIC, typename T>
__device__ __forceinline__ int band_cell(const FusedAxis<T>& x, int pos) {
  const int d0 = pos - x.start[ELECTRIC][0], d1 = pos - x.start[ELECTRIC][1];
  return (unsigned)d0 < (unsigned)x.nc[ELECTRIC][0]   ? d0
         : (unsigned)d1 < (unsigned)x.nc[ELECTRIC][1] ? x.nc[ELECTRIC][0] + d1
                                                      : -1;
}

// Whether a column of a z slab lies in the band.  Outside the bands b is -0 (no
// band's b = exp(-x) is): such a column keeps a zero Psi and takes none of it, as
// 0 times an infinite drive is not 0.  The slabs of one-column groups are the bands.
__device__ __forceinline__ bool in_band(float b) { return __float_as_uint(b) != 0x80000000u; }
__device__ __forceinline__ constexpr bool in_band(double) { return true; }

// Programmatic launches: waits for the launch before this one (at once where
// this is an ordinary launch), and lets the one after it start its blocks.
__device__ __forceinline__ void launch_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Orders what this thread sees of global memory ahead of its tensor copies, which
// read it by another path (the launch before wrote it with ordinary stores).
__device__ __forceinline__ void fence_proxy_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One (k, j, i) tile from the padded array of `map` into shared memory,
// completing on `bar`.  Elements outside the array read zero.
__device__ __forceinline__ void tma_tile(void* dst, const CUtensorMap* map, int k, int j, int i,
                                         unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
          smem_addr(dst)),
      "l"(map), "r"(k), "r"(j), "r"(i), "r"(smem_addr(bar))
      : "memory");
}

// One axis's CPML on a value: Psi = b Psi + a drive, v += CPsi Psi; `in`: see in_band.
template <bool EXACT, typename T>
__device__ __forceinline__ void fused_cpml(T& psi, T b, T a, T cp, T d, T& v, bool in = true) {
  const T n = Ar<T, EXACT>::lin2(b, psi, a, d);
  psi = in ? n : T(0);
  v = Ar<T, EXACT>::axpy(v, cp, psi);
}

// Psi of one plane's half-step.  It is loaded at the head of the half-step, from
// L2: `ahead` planes earlier its line was asked for.  (Holding the next plane's
// values in registers made every wait on shared memory wait for them too.)
template <typename T>
struct FusedPsi {
  Vec<T> x0, x1, y0, y1, z0, z1;
};
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }
template <bool ELECTRIC, typename T>
__device__ __forceinline__ void fused_psi(const FusedAxis<T>& A, unsigned o, unsigned ahead, Vec<T>& s0, Vec<T>& s1) {
  if (ahead) {
    prefetch_l2((ELECTRIC ? A.pe[0] : A.phi[0]) + o + ahead);
    prefetch_l2((ELECTRIC ? A.pe[1] : A.phi[1]) + o + ahead);
  }
  s0 = ELECTRIC ? ldw<T>(A.pe[0] + o) : ldv<T>(A.phi[0] + o);
  s1 = ELECTRIC ? ldw<T>(A.pe[1] + o) : ldv<T>(A.phi[1] + o);
}

// A cell's coefficients for one half-step, the y band's included (yc: the
// column's band cell), and those of its z differences per cell of the group (zc:
// its slab cell).
template <typename T>
struct FusedCoef {
  Row<T> x, y, z;
  Vec<T> z0, z1;  // Hx c1, Hy c2 / Ex c2, Ey c1
};
template <bool ELECTRIC, typename T>
__device__ __forceinline__ void fused_coef(const ClassRow& L, const T* row, int yc, int zc, FusedCoef<T>& n) {
  n.x = ld_row(row, ELECTRIC ? 3 : 0);
  n.y = ld_row(row, ELECTRIC ? 4 : 1);
  n.z = ld_row(row, ELECTRIC ? 5 : 2);
  if (yc >= 0) {
    const T* t = row + L.o[1] + (ELECTRIC ? 2 : 0) * L.n[1] + yc;
    (ELECTRIC ? n.z.c2 : n.x.c2) = __ldg(t);
    (ELECTRIC ? n.x.c1 : n.z.c1) = __ldg(t + L.n[1]);
  }
  if (zc >= 0) {
    const T* t = row + L.o[2] + (ELECTRIC ? 2 : 0) * L.n[2] + zc;
    n.z0 = ldv<T>(t);
    n.z1 = ldv<T>(t + L.n[2]);
  } else {
#pragma unroll
    for (int q = 0; q < FusedShape<T>::V; q++) {
      n.z0.v[q] = ELECTRIC ? n.x.c2 : n.x.c1;
      n.z1.v[q] = ELECTRIC ? n.y.c1 : n.y.c2;
    }
  }
}

// Values the update leaves alone along z: Hx and Hy do not exist at k = nz, Ex
// and Ey are held at k = 0 and k = nz.  They keep their old value here, so that
// the groups at the walls need no class of their own.  `all`: the whole group is
// held by another wall.
template <bool ELECTRIC, typename T>
__device__ __forceinline__ void fused_hold(int k, int nz, bool all, const Vec<T>& old, Vec<T>& v) {
#pragma unroll
  for (int q = 0; q < FusedShape<T>::V; q++)
    if (all || k + q == nz || (ELECTRIC && q == 0 && k == 0)) v.v[q] = old.v[q];
}

// The coefficients of the cells of a group for one half-step.  Cells that share
// a class share the set held in registers.  Where they do not (MIXED, at
// material edges), each cell's set is loaded ahead or its parts are looked up
// where they are used: the sets cost registers, which spill (16 to 28 bytes a
// thread, and a 512 x 512 x 640 table problem without CPML went from 1.71 to
// 2.04 ms), the look-ups time on every mixed plane (a 97 x 131 x 118 problem of
// materials cell by cell: 62 us with sets, 76 us with look-ups).  A material
// table has mixed groups only at the faces of its bodies, and looks up.
enum FusedMix { kSame, kSets, kLookUp };
template <typename T, FusedMix MIX, bool ELECTRIC>
struct FusedCells {
  static constexpr bool MIXED = MIX != kSame;
  const FusedCoef<T>* n;  // one set, or one per cell
  const T* tab;
  const ClassRow& L;
  unsigned id;  // the classes, 16 bits each
  int yc, zc;
  __device__ __forceinline__ const T* row(int q) const {
    return tab + (id >> (MIXED ? 16 * q : 0) & 0xffffu) * (unsigned)L.stride;
  }
  __device__ __forceinline__ T cpsi(int q, int slot) const { return __ldg(row(q) + kRowCpsi + slot); }
  // band value of the axis's Psi slot s (0, 1) at cell c
  __device__ __forceinline__ T band(int q, int axis, int s, int c) const {
    return __ldg(row(q) + L.o[axis] + ((ELECTRIC ? 2 : 0) + s) * L.n[axis] + c);
  }
  __device__ __forceinline__ Row<T> x(int q) const {
    if constexpr (MIX != kLookUp) return n[MIXED ? q : 0].x;
    Row<T> r = ld_row(row(q), ELECTRIC ? 3 : 0);
    if (yc >= 0) (ELECTRIC ? r.c1 : r.c2) = band(q, 1, ELECTRIC ? 1 : 0, yc);
    return r;
  }
  __device__ __forceinline__ Row<T> y(int q) const {
    if constexpr (MIX != kLookUp) return n[MIXED ? q : 0].y;
    return ld_row(row(q), ELECTRIC ? 4 : 1);
  }
  __device__ __forceinline__ Row<T> z(int q) const {
    if constexpr (MIX != kLookUp) return n[MIXED ? q : 0].z;
    Row<T> r = ld_row(row(q), ELECTRIC ? 5 : 2);
    if (yc >= 0) (ELECTRIC ? r.c2 : r.c1) = band(q, 1, ELECTRIC ? 0 : 1, yc);
    return r;
  }
  // coefficients of the z differences: Hx c1 / Ex c2, and Hy c2 / Ey c1
  __device__ __forceinline__ T z0(int q) const {
    if constexpr (MIX != kLookUp) return n[MIXED ? q : 0].z0.v[q];
    if (zc >= 0) return band(q, 2, 0, zc + q);
    const Row<T> r = ld_row(row(q), ELECTRIC ? 3 : 0);
    return ELECTRIC ? r.c2 : r.c1;
  }
  __device__ __forceinline__ T z1(int q) const {
    if constexpr (MIX != kLookUp) return n[MIXED ? q : 0].z1.v[q];
    if (zc >= 0) return band(q, 2, 1, zc + q);
    const Row<T> r = ld_row(row(q), ELECTRIC ? 4 : 1);
    return ELECTRIC ? r.c1 : r.c2;
  }
};

// A thread's column group and its bands on the current plane.
template <typename T>
struct FusedHere {
  int i, j, k;
  int xc;                 // band cell of the plane, -1 outside
  unsigned ox, oy, oz;    // Psi offsets
  const T *prow, *pcol;   // the row's and columns' profiles in shared memory
  bool store;             // Psi goes back to memory
};

// H of a group, from the old E tiles (E, En: planes i and i + 1) and old H.
template <bool EXACT, FusedMix MIX, typename T>
__device__ __forceinline__ void fused_h(const FusedParams<T>& p, const FusedCells<T, MIX, false>& c, const FusedHere<T>& t,
                                        FusedPsi<T>& f, const T* E, const T* H, const Vec<T>& ex, const Vec<T>& ey,
                                        const Vec<T>& ez, const Vec<T>& eyn, const Vec<T>& ezn, Vec<T>& hx, Vec<T>& hy,
                                        Vec<T>& hz) {
  using A = Ar<T, EXACT>;
  constexpr int V = FusedShape<T>::V, W = kTileW, R1 = kTileRows + 1, ES = kTileE, HS = kTileH;
  const Vec<T> dey_z = vdiff_up(ey, E[ES + V]), dez_y = vsub(ldw<T>(E + 2 * ES + W), ez);
  const Vec<T> dez_x = vsub(ezn, ez), dex_z = vdiff_up(ex, E[V]);
  const Vec<T> dex_y = vsub(ldw<T>(E + W), ex), dey_x = vsub(eyn, ey);
  const Vec<T> ox = ldw<T>(H), oy = ldw<T>(H + HS), oz = ldw<T>(H + 2 * HS);
  T cx0 = T(0), cx1 = T(0);
#pragma unroll
  for (int q = 0; q < V; q++) {
    if (t.xc >= 0 && (MIX != kSame || q == 0)) {
      cx0 = c.band(q, 0, 0, t.xc);
      cx1 = c.band(q, 0, 1, t.xc);
    }
    const Row<T> x = c.x(q), y = c.y(q), z = c.z(q);
    hx.v[q] = A::lin3(x.c0, ox.v[q], c.z0(q), dey_z.v[q], x.c2, dez_y.v[q]);
    hy.v[q] = A::lin3(y.c0, oy.v[q], t.xc >= 0 ? cx0 : y.c1, dez_x.v[q], c.z1(q), dex_z.v[q]);
    hz.v[q] = A::lin3(z.c0, oz.v[q], z.c1, dex_y.v[q], t.xc >= 0 ? cx1 : z.c2, dey_x.v[q]);
  }
  fused_hold<false>(t.k, p.nz, false, ox, hx);
  fused_hold<false>(t.k, p.nz, false, oy, hy);
  if (t.xc >= 0) {
    const FusedAxis<T>& X = p.axis[0];
    const T b = __ldg(X.prof[0][0] + t.i), a = __ldg(X.prof[0][1] + t.i);
#pragma unroll
    for (int q = 0; q < V; q++) {
      fused_cpml<EXACT>(f.x0.v[q], b, a, c.cpsi(q, 2), dez_x.v[q], hy.v[q]);
      fused_cpml<EXACT>(f.x1.v[q], b, a, c.cpsi(q, 5), dey_x.v[q], hz.v[q]);
    }
    if (t.store) {
      stv(X.pho[0] + t.ox, f.x0);
      stv(X.pho[1] + t.ox, f.x1);
    }
  }
  if (c.yc >= 0) {
    const FusedAxis<T>& Y = p.axis[1];
    const T b = t.prow[0], a = t.prow[R1];
#pragma unroll
    for (int q = 0; q < V; q++) {
      fused_cpml<EXACT>(f.y0.v[q], b, a, c.cpsi(q, 1), dez_y.v[q], hx.v[q]);
      fused_cpml<EXACT>(f.y1.v[q], b, a, c.cpsi(q, 4), dex_y.v[q], hz.v[q]);
    }
    if (t.store) {
      stv(Y.pho[0] + t.oy, f.y0);
      stv(Y.pho[1] + t.oy, f.y1);
    }
  }
  if (c.zc >= 0) {
    const FusedAxis<T>& Z = p.axis[2];
    const Vec<T> b = ldw<T>(t.pcol), a = ldw<T>(t.pcol + W);
#pragma unroll
    for (int q = 0; q < V; q++) {
      fused_cpml<EXACT>(f.z0.v[q], b.v[q], a.v[q], c.cpsi(q, 0), dey_z.v[q], hx.v[q], in_band(b.v[q]));
      fused_cpml<EXACT>(f.z1.v[q], b.v[q], a.v[q], c.cpsi(q, 3), dex_z.v[q], hy.v[q], in_band(b.v[q]));
    }
    if (t.store) {
      stv(Z.pho[0] + t.oz, f.z0);
      stv(Z.pho[1] + t.oz, f.z1);
    }
  }
}

// E of a group from its new H, that of plane i - 1 (hyp, hzp) and the new H
// around it (N: its place in the exchange tiles).  Ey and Ez at i = nx are held
// (x_wall) or left to k_fused_wall: yz is false there.
template <bool EXACT, FusedMix MIX, typename T>
__device__ __forceinline__ void fused_e(const FusedParams<T>& p, const FusedCells<T, MIX, true>& c, const FusedHere<T>& t,
                                        FusedPsi<T>& f, bool yz, const T* N, const Vec<T>& hx, const Vec<T>& hy,
                                        const Vec<T>& hz, const Vec<T>& hyp, const Vec<T>& hzp, Vec<T>& ex, Vec<T>& ey,
                                        Vec<T>& ez) {
  using A = Ar<T, EXACT>;
  constexpr int V = FusedShape<T>::V, W = kTileW, R1 = kTileRows + 1, HS = kTileH;
  const Vec<T> dhz_y = vsub(hz, ldw<T>(N + 2 * HS - W)), dhy_z = vdiff_dn(hy, N[HS - 1]);
  const Vec<T> dhx_z = vdiff_dn(hx, N[-1]), dhx_y = vsub(hx, ldw<T>(N - W));
  const Vec<T> dhz_x = vsub(hz, hzp), dhy_x = vsub(hy, hyp);
  const Vec<T> oex = ex, oey = ey, oez = ez;
#pragma unroll
  for (int q = 0; q < V; q++) {
    const Row<T> x = c.x(q);
    ex.v[q] = A::lin3(x.c0, ex.v[q], x.c1, dhz_y.v[q], c.z0(q), dhy_z.v[q]);
  }
  // the row of a wall: as one compare it makes the table kernel spill 8 bytes, as two
  // it costs FP64 0.7% of a step (256^3: 555 us for 551)
  const bool wall_j = V > 1 ? t.j == 0 || t.j == p.ny : (unsigned)(t.j - 1) >= (unsigned)(p.ny - 1);
  fused_hold<true>(t.k, p.nz, wall_j, oex, ex);
  if (yz) {
    T cx0 = T(0), cx1 = T(0);
#pragma unroll
    for (int q = 0; q < V; q++) {
      if (t.xc >= 0 && (MIX != kSame || q == 0)) {
        cx0 = c.band(q, 0, 0, t.xc);
        cx1 = c.band(q, 0, 1, t.xc);
      }
      const Row<T> y = c.y(q), z = c.z(q);
      ey.v[q] = A::lin3(y.c0, ey.v[q], c.z1(q), dhx_z.v[q], t.xc >= 0 ? cx0 : y.c2, dhz_x.v[q]);
      ez.v[q] = A::lin3(z.c0, ez.v[q], t.xc >= 0 ? cx1 : z.c1, dhy_x.v[q], z.c2, dhx_y.v[q]);
    }
    fused_hold<true>(t.k, p.nz, t.i == 0, oey, ey);
    if (wall_j || t.i == 0) ez = oez;
    if (t.xc >= 0) {
      const FusedAxis<T>& X = p.axis[0];
      const T b = __ldg(X.prof[1][0] + t.i), a = __ldg(X.prof[1][1] + t.i);
#pragma unroll
      for (int q = 0; q < V; q++) {
        fused_cpml<EXACT>(f.x0.v[q], b, a, c.cpsi(q, 9), dhz_x.v[q], ey.v[q]);
        fused_cpml<EXACT>(f.x1.v[q], b, a, c.cpsi(q, 10), dhy_x.v[q], ez.v[q]);
      }
      stv(X.pe[0] + t.ox, f.x0);
      stv(X.pe[1] + t.ox, f.x1);
    }
  }
  if (c.yc >= 0) {
    const FusedAxis<T>& Y = p.axis[1];
    const T b = t.prow[2 * R1], a = t.prow[3 * R1];
#pragma unroll
    for (int q = 0; q < V; q++) fused_cpml<EXACT>(f.y1.v[q], b, a, c.cpsi(q, 6), dhz_y.v[q], ex.v[q]);
    stv(Y.pe[1] + t.oy, f.y1);
    if (yz) {
#pragma unroll
      for (int q = 0; q < V; q++) fused_cpml<EXACT>(f.y0.v[q], b, a, c.cpsi(q, 11), dhx_y.v[q], ez.v[q]);
      stv(Y.pe[0] + t.oy, f.y0);
    }
  }
  if (c.zc >= 0) {
    const FusedAxis<T>& Z = p.axis[2];
    const Vec<T> b = ldw<T>(t.pcol + 2 * W), a = ldw<T>(t.pcol + 3 * W);
#pragma unroll
    for (int q = 0; q < V; q++) fused_cpml<EXACT>(f.z0.v[q], b.v[q], a.v[q], c.cpsi(q, 7), dhy_z.v[q], ex.v[q], in_band(b.v[q]));
    stv(Z.pe[0] + t.oz, f.z0);
    if (yz) {
#pragma unroll
      for (int q = 0; q < V; q++) fused_cpml<EXACT>(f.z1.v[q], b.v[q], a.v[q], c.cpsi(q, 8), dhx_z.v[q], ey.v[q], in_band(b.v[q]));
      stv(Z.pe[1] + t.oz, f.z1);
    }
  }
}

// One tile of one step.  Load event t of the ring brings the E tiles of plane
// t and the H tiles of plane t - 1 into slots t and t - 1 (mod kFusedStages,
// counted from the chunk's first plane).  A thread keeps its own old E and new
// H of a plane in registers, so after the plane's barrier its E slot and the H
// slot before it are free and the event kFusedStages planes on is issued, two
// planes before its wait.  The block's last warp waits for the next plane's
// event ahead of the barrier that the other warps meet it at.  New H goes
// through two exchange buffers that only threads write (the ring's are written
// by the copies alone, so no proxy fence is needed between them).
template <typename T, bool EXACT>
__device__ __forceinline__ void fused_tile(const FusedParams<T>& p, int bx, int by, int bz,
                                           unsigned char* smem) {
  constexpr int V = FusedShape<T>::V, NT = FusedShape<T>::kThreads;
  constexpr int NS = kFusedStages, W = kTileW, R1 = kTileRows + 1, ES = kTileE, HS = kTileH;
  const int tid = threadIdx.x;
  const int rk = p.rk, hk = p.halo_k;
  const int r = tid / rk, q0 = (tid - r * rk) * V + (4 - V) * hk;  // row and first column in the tiles
  const int j0 = by * (kTileRows - 1) - 1, kb = bx * (rk - hk) * V - 4 * hk;  // first row and column of the tiles
  const int j = j0 + r, k = kb + q0;
  const bool in = r < kTileRows && j >= 0 && j <= p.ny && k >= 0 && k <= p.nz;
  const bool own = in && r >= 1 && (hk == 0 || q0 >= 4);
  const int i0 = (int)((long long)bz * (p.nx + 1) / p.tx), i1 = (int)((long long)(bz + 1) * (p.nx + 1) / p.tx);
  const int ib = i0 > 0 ? i0 - 1 : 0;  // the plane before the chunk: H only, for the x differences of E

  unsigned char* const sc = smem;            // [NS] classes
  T* const se = reinterpret_cast<T*>(smem + NS * kTileCBytes);  // [NS][Ex Ey Ez]
  T* const sh = se + NS * 3 * ES;            // [NS][Hx Hy Hz], old
  T* const sx = sh + NS * 3 * HS;            // [2][Hx Hy Hz], new
  T* const sprof = sx + 2 * 3 * HS;          // profiles of the tile's columns, then rows: [H, E][b, a]
  unsigned long long* const bar = reinterpret_cast<unsigned long long*>(sprof + 4 * (R1 + W));
  constexpr unsigned kEBytes = R1 * W * sizeof(T), kHBytes = kTileRows * (3 * W * sizeof(T) + kTileC * 2);
  const int kc = kb & ~7;  // first column of the class tiles
  const int last = i1 - ib;  // the last event
  auto issue = [&](int m) {  // event of plane ib + m
    const int s = m % NS, sp = (m + NS - 1) % NS;
    mbar_arrive_tx(bar + s, 3 * kEBytes + (m > 0 ? kHBytes : 0));
    for (int c = 0; c < 3; c++) tma_tile(se + (s * 3 + c) * ES, &p.map[3 + c], kb, j0, ib + m, bar + s);
    if (m == 0) return;
    for (int c = 0; c < 3; c++) tma_tile(sh + (sp * 3 + c) * HS, &p.map[c], kb, j0, ib + m - 1, bar + s);
    tma_tile(sc + sp * kTileCBytes, &p.map[6], kc, j0, ib + m - 1, bar + s);
  };
  if (tid == 0) {
    for (int s = 0; s < NS; s++) mbar_init(bar + s, 1);
    mbar_fence_init();
  }
  for (int w = tid; w < 4 * (R1 + W); w += NT) {
    const bool row = w >= 4 * W;
    const int u = row ? w - 4 * W : w, len = row ? R1 : W;
    const int c = u / len, pos = (row ? j0 : kb) + u % len;  // c: 2 electric + (b, a)
    const bool fits = pos >= 0 && pos <= (row ? p.ny : p.nz);
    sprof[w] = fits ? __ldg(p.axis[row ? 1 : 2].prof[c / 2][c % 2] + pos) : T(0);
  }
  // All above overlaps the launch before; all it wrote is read from here on.
  launch_wait();
  launch_next();
  if (tid == 0) {
    if (bx + by + bz == 0) *p.ts_next = *p.ts + 1;
    fence_proxy_global();
    for (int m = 0; m <= min(NS - 1, last); m++) issue(m);
  }
  // H where the grid has none is read into differences that nothing uses
  for (int w = tid; w < 2 * 3 * HS; w += NT) sx[w] = T(0);

  const unsigned plane = p.plane, jk = in ? (unsigned)(j * p.pitch + k) : 0u;
  unsigned off = (unsigned)ib * plane + jk;
  const FusedAxis<T>&X = p.axis[0], &Y = p.axis[1], &Z = p.axis[2];
  const int yh = in ? band_cell<false>(Y, j) : -1, zh = in ? band_cell<false>(Z, k) : -1;
  const int ye = own ? band_cell<true>(Y, j) : -1, ze = own ? band_cell<true>(Z, k) : -1;
  // Psi offsets, and their steps from plane to plane
  const unsigned dy = (unsigned)(Y.nb * p.pitch), dz = (unsigned)((p.ny + 1) * Z.nb);
  auto oy_at = [&](int c, int i) { return (unsigned)((i * Y.nb + c) * p.pitch + k); };
  auto oz_at = [&](int c, int i) { return (unsigned)((i * (p.ny + 1) + j) * Z.nb + c); };
  // uniform over the block: the chunk meets an x band; a source box meets the tile
  bool xband = false, src_here = false;
  for (int e = 0; e < 2; e++)
    for (int f = 0; f < 2; f++) xband |= X.nc[e][f] > 0 && X.start[e][f] < i1 && X.start[e][f] + X.nc[e][f] > ib;
  for (int s = 0; s < p.src.n; s++) {
    const SourceBox& b = p.src.box[s];
    src_here |= b.i1 >= i0 && b.i0 < i1 && b.j1 > j0 && b.j0 < j0 + kTileRows && b.k1 >= kb && b.k0 < kb + W;
  }
  // Psi of plane i for the next half-step of each kind
  FusedPsi<T> ph{}, pe{};
  auto psi_h = [&](int i) {
    const unsigned far = i + kPsiAhead < i1 ? kPsiAhead : 0;
    if (xband) {
      const int c = band_cell<false>(X, i);
      if (c >= 0) fused_psi<false>(X, (unsigned)c * plane + jk, c + 2 < X.nb ? 2 * plane : 0, ph.x0, ph.x1);
    }
    if (yh >= 0) fused_psi<false>(Y, oy_at(yh, i), far * dy, ph.y0, ph.y1);
    if (zh >= 0) fused_psi<false>(Z, oz_at(zh, i), far * dz, ph.z0, ph.z1);
  };
  auto psi_e = [&](int i) {
    const unsigned far = i + kPsiAhead < i1 ? kPsiAhead : 0;
    if (xband) {
      const int c = band_cell<true>(X, i);
      if (c >= 0) fused_psi<true>(X, (unsigned)c * plane + jk, c + 2 < X.nb ? 2 * plane : 0, pe.x0, pe.x1);
    }
    if (ye >= 0) fused_psi<true>(Y, oy_at(ye, i), far * dy, pe.y0, pe.y1);
    if (ze >= 0) fused_psi<true>(Z, oz_at(ze, i), far * dz, pe.z0, pe.z1);
  };
  const bool bands_h = xband || yh >= 0 || zh >= 0, bands_e = xband || ye >= 0 || ze >= 0;


  __syncthreads();  // the barriers are initialised
  bool ok = mbar_wait(bar, 0);
  if (ok && last >= 1) ok = mbar_wait(bar + 1 % NS, 0);

  const int at = r * W + q0;
  const T* const pcol = sprof + q0;         // + c W
  const T* const prow = sprof + 4 * W + r;  // + c R1
  const unsigned char* const ct = sc + 2 * (r * kTileC + q0 + kb - kc);
  auto ids = [&](int n) -> unsigned {  // the group's classes, 16 bits each
    const unsigned char* c = ct + (n % NS) * kTileCBytes;
    if constexpr (V == 2) return *reinterpret_cast<const unsigned*>(c);
    return *reinterpret_cast<const unsigned short*>(c);
  };
  constexpr FusedMix kMix = EXACT ? kSets : kLookUp;
  FusedCoef<T> ch, ce;
  unsigned id = 0;
  bool first = true;
  Vec<T> ey, ez, hyp{}, hzp{};
  if (in) {
    ey = ldw<T>(se + at + ES);
    ez = ldw<T>(se + at + 2 * ES);
  }
  for (int i = ib, n = 0; i < i1; i++, n++, off += plane) {
    const bool act = own && i >= i0, yz = i < p.nx, more = i + 1 < i1;
    const T* E = se + (n % NS) * 3 * ES + at;
    const T* En = se + ((n + 1) % NS) * 3 * ES + at;
    const T* H = sh + (n % NS) * 3 * HS + at;
    T* const N = sx + (n % 2) * 3 * HS + at;
    Vec<T> ex, hx, hy, hz, eyn, ezn;
    bool mixed = false;
    FusedHere<T> t;
    t.i = i, t.j = j, t.k = k;
    t.prow = prow, t.pcol = pcol;
    if (in) {
      const unsigned idn = ids(n);
      mixed = V == 2 && (idn >> 16) != (idn & 0xffffu);
      if (idn != id || first) {
        id = idn;
        first = false;
        if (!mixed) {
          const T* row = p.tab + (id & 0xffffu) * (unsigned)p.row.stride;
          fused_coef<false>(p.row, row, yh, zh, ch);
          if (own) fused_coef<true>(p.row, row, ye, ze, ce);
        }
      }
      t.xc = xband ? band_cell<false>(X, i) : -1;
      t.ox = (unsigned)t.xc * plane + jk;
      t.oy = oy_at(yh, i);
      t.oz = oz_at(zh, i);
      t.store = act;
      if (bands_h) psi_h(i);
      ex = ldw<T>(E);
      eyn = ldw<T>(En + ES);
      ezn = ldw<T>(En + 2 * ES);
      if (!mixed) {
        fused_h<EXACT>(p, FusedCells<T, kSame, false>{&ch, p.tab, p.row, id, yh, zh}, t, ph, E, H, ex, ey, ez, eyn, ezn, hx, hy, hz);
      } else if constexpr (kMix == kLookUp) {
        fused_h<EXACT>(p, FusedCells<T, kLookUp, false>{nullptr, p.tab, p.row, id, yh, zh}, t, ph, E, H, ex, ey, ez, eyn, ezn, hx, hy, hz);
      } else {
        FusedCoef<T> m[V];
#pragma unroll
        for (int q = 0; q < V; q++) fused_coef<false>(p.row, p.tab + (id >> 16 * q & 0xffffu) * (unsigned)p.row.stride, yh, zh, m[q]);
        fused_h<EXACT>(p, FusedCells<T, kSets, false>{m, p.tab, p.row, id, yh, zh}, t, ph, E, H, ex, ey, ez, eyn, ezn, hx, hy, hz);
      }
      stv(N, hx);
      stv(N + HS, hy);
      stv(N + 2 * HS, hz);
      if (act) {
        stv(p.fo[0] + off, hx);
        stv(p.fo[1] + off, hy);
        stv(p.fo[2] + off, hz);
      }

    }
    if (act && bands_e) psi_e(i);
    if (tid >= NT - 32 && ok && n + 2 <= last) ok = mbar_wait(bar + (n + 2) % NS, ((n + 2) / NS) & 1);
    __syncthreads();
    if (tid == 0 && n + NS <= last) issue(n + NS);
    if (act) {
      t.xc = xband ? band_cell<true>(X, i) : -1;
      t.ox = (unsigned)t.xc * plane + jk;
      t.oy = oy_at(ye, i);
      t.oz = oz_at(ze, i);
      if (!mixed) {
        fused_e<EXACT>(p, FusedCells<T, kSame, true>{&ce, p.tab, p.row, id, ye, ze}, t, pe, yz, N, hx, hy, hz, hyp, hzp, ex, ey, ez);
      } else if constexpr (kMix == kLookUp) {
        fused_e<EXACT>(p, FusedCells<T, kLookUp, true>{nullptr, p.tab, p.row, id, ye, ze}, t, pe, yz, N, hx, hy, hz, hyp, hzp, ex, ey, ez);
      } else {
        FusedCoef<T> m[V];
#pragma unroll
        for (int q = 0; q < V; q++) fused_coef<true>(p.row, p.tab + (id >> 16 * q & 0xffffu) * (unsigned)p.row.stride, ye, ze, m[q]);
        fused_e<EXACT>(p, FusedCells<T, kSets, true>{m, p.tab, p.row, id, ye, ze}, t, pe, yz, N, hx, hy, hz, hyp, hzp, ex, ey, ez);
      }
      if (src_here) {
        const int ts = *p.ts;
#pragma unroll
        for (int q = 0; q < V; q++) {
          inject_sources(p.src, 0, i, j, k + q, ts, ex.v[q]);
          if (yz) {
            inject_sources(p.src, 1, i, j, k + q, ts, ey.v[q]);
            inject_sources(p.src, 2, i, j, k + q, ts, ez.v[q]);
          }
        }
      }
      stv(p.fo[3] + off, ex);
      stv(p.fo[4] + off, ey);
      stv(p.fo[5] + off, ez);

    }
    ey = eyn;
    ez = ezn;
    hyp = hy;
    hzp = hz;
  }
  if (!ok) {
    atomicExch(p.fault, 4);  // the handle's status code: a device wait ran out
    for (int m = max(0, last - NS + 1); m <= last; m++) mbar_wait(bar + m % NS, (m / NS) & 1);  // copies in flight
  }
}

// ---------------------------------------------------------------------------
// Ey and Ez at i = nx with the reference's reads one plane past Hz and Hy
// (fdtd_kernels.ts:159-204): Ex(i=0) after its bulk update stands in for
// Hz(nx), the start of the Hz array for Hy(nx).  One thread per (j, k), after
// the step's main launch: new H from the copy written, old E from the other.
// ---------------------------------------------------------------------------
template <typename T, bool EXACT>
__device__ __forceinline__ void fused_wall_thread(const FusedParams<T>& p, int ts, int t) {
  using A = Ar<T, EXACT>;
  const int ny = p.ny, nz = p.nz, P = p.pitch, i = p.nx;
  const int j = t / (nz + 1), k = t % (nz + 1);
  if (j > ny) return;
  const T* const* fi = p.fi;
  T* const* fo = p.fo;
  const unsigned jk = (unsigned)(j * P + k), off = (unsigned)i * p.plane + jk;
  const T* row = p.tab + p.cls[off] * (unsigned)p.row.stride;
  const bool jy = j >= 1 && j < ny, kz = k >= 1 && k < nz;
  constexpr int V = FusedShape<T>::V;
  const FusedAxis<T>&Y = p.axis[1], &Z = p.axis[2];
  const int kq = k % V;  // place in its group
  const int yc = band_cell<true>(Y, j), zg = band_cell<true>(Z, k - kq), zc = zg >= 0 && in_band(Z.prof[1][0][k]) ? zg + kq : -1;
  FusedCoef<T> n;
  fused_coef<true>(p.row, row, yc, zg, n);
  const T hx = (j < ny && k < nz) ? fo[0][off] : T(0);
  if (j < ny) {  // Ey
    // Ex(0, j, k) after its bulk update
    FusedCoef<T> n0;
    fused_coef<true>(p.row, p.tab + p.cls[jk] * (unsigned)p.row.stride, yc, zg, n0);
    T hz_i = fi[3][jk];
    if (jy && kz)
      hz_i = A::lin3(n0.x.c0, hz_i, n0.x.c1, A::dif(fo[2][jk], fo[2][jk - P]), n0.z0.v[kq], A::dif(fo[1][jk], fo[1][jk - 1]));
    const T dhz = A::dif(hz_i, fo[2][off - p.plane]);
    const T dhx = kz ? A::dif(hx, fo[0][off - 1]) : T(0);
    T e = fi[4][off];
    if (kz) e = A::lin3(n.y.c0, e, n.z1.v[kq], dhx, n.y.c2, dhz);
    if (zc >= 0) {
      T& psi = Z.pe[1][(unsigned)((i * (ny + 1) + j) * Z.nb + zc)];
      fused_cpml<EXACT>(psi, Z.prof[1][0][k], Z.prof[1][1][k], row[kRowCpsi + 8], dhx, e);
    }
    inject_sources(p.src, 1, i, j, k, ts, e);
    fo[4][off] = e;
  }
  if (k < nz) {  // Ez
    const int oa = j * nz + k, len = nz + 1, pl = ny * len;
    const int i2 = oa / pl, j2 = (oa - i2 * pl) / len, k2 = oa % len;
    const T hy_i = fo[2][(unsigned)i2 * p.plane + (unsigned)(j2 * P + k2)];
    const T dhy = A::dif(hy_i, fo[1][off - p.plane]);
    const T dhx = jy ? A::dif(hx, fo[0][off - P]) : T(0);
    T e = fi[5][off];
    if (jy) e = A::lin3(n.z.c0, e, n.z.c1, dhy, n.z.c2, dhx);
    if (yc >= 0) {
      T& psi = Y.pe[0][(unsigned)((i * Y.nb + yc) * P + k)];
      fused_cpml<EXACT>(psi, Y.prof[1][0][j], Y.prof[1][1][j], row[kRowCpsi + 11], dhx, e);
    }
    inject_sources(p.src, 2, i, j, k, ts, e);
    fo[5][off] = e;
  }
}

// Tile of block b.  Tiles in the y bands come first, then the rest of those in
// the z bands, then the others.
// The tiles with Psi take about twice the time of the others: one that started
// last would leave the device waiting for it.
template <typename T>
__device__ __forceinline__ void fused_place(const FusedParams<T>& p, int b, int& bx, int& by, int& bz) {
  const int nj = p.slow_j[0] + p.slow_j[1], nk = p.slow_k[0] + p.slow_k[1], mj = p.tj - nj, mk = p.tk - nk;
  const int n1 = nj * p.tk * p.tx, n2 = mj * nk * p.tx;
  if (b < n1) {
    bx = b % p.tk;
    b /= p.tk;
    const int y = b % nj;
    by = y < p.slow_j[0] ? y : y + mj;
    bz = b / nj;
  } else {
    const bool z = b < n1 + n2;
    b -= z ? n1 : n1 + n2;
    const int w = z ? nk : mk, x = b % w;
    bx = !z ? p.slow_k[0] + x : x < p.slow_k[0] ? x : x + mk;
    b /= w;
    by = p.slow_j[0] + b % mj;
    bz = b / mj;
  }
  if (p.axis[0].nb > 0) bz = bz == 0 ? p.tx - 1 : bz - 1;  // the chunk of the x band at the high end is not the last
}

// ---------------------------------------------------------------------------
// Single-problem launches.  Each copy has a step counter: a launch finds its
// step in the counter of the copy it reads and block 0 leaves the next one in
// the other copy's, so no launch writes the counter its own blocks read.
//
// The epilogue of a step is a launch of its own, queued after the NEXT step's:
// it reads the copy that the next step only reads, and may start when the last
// block of that step has (programmatic launch), so its blocks fill the slots
// that the step's last blocks leave idle; it ends only when that step has.  As
// blocks of the step's own kernel it costs the step registers, which spill; on
// a second stream beside the step it measured no faster than after it.
// ---------------------------------------------------------------------------
template <typename T, bool EXACT>
__global__ void __launch_bounds__(FusedShape<T>::kThreads, FusedShape<T>::kBlocks)
    k_fused(const __grid_constant__ FusedParams<T> p) {
  extern __shared__ __align__(128) unsigned char fused_smem[];
  int bx, by, bz;
  fused_place(p, blockIdx.x, bx, by, bz);
  fused_tile<T, EXACT>(p, bx, by, bz, fused_smem);
}

// Epilogue of the step that wrote this copy: `late`, under the next step's
// parameters and beside it; else under its own, after it.
template <typename T>
__global__ void __launch_bounds__(256)
    k_fused_epilogue(const __grid_constant__ FusedParams<T> p, const __grid_constant__ FarField ff,
                     const __grid_constant__ Probes pr, int late) {
  if (!late) launch_wait();
  launch_next();
  // `late`: this launch starts when every block of the running step has passed its
  // launch_next, which stands after its launch_wait.  So the launch before that step
  // had ended, and it had waited, at its own end at the latest, for the step whose
  // copy is read here: that copy was written and flushed before any block of this
  // launch was there to read it, and its next writer is queued behind this launch.
  // No block has read the copy before it was written, but a multiprocessor's cache
  // may hold lines of an earlier epilogue's: the fence drops them.
  if (late) __threadfence();
  const T* f[6];
#pragma unroll
  for (int c = 0; c < 6; c++) f[c] = late ? p.fi[c] : p.fo[c];
  epilogue_thread(Fields<const T>{f[0], f[1], f[2], f[3], f[4], f[5]}, PaddedGrid{p.pitch, p.ny + 1}, ff, pr,
                  (late ? *p.ts : *p.ts_next) - 1, (long long)blockIdx.x * blockDim.x + threadIdx.x);
  if (late) launch_wait();
}

template <typename T, bool EXACT>
__global__ void __launch_bounds__(256) k_fused_wall(const __grid_constant__ FusedParams<T> p) {
  fused_wall_thread<T, EXACT>(p, *p.ts, blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------
// Cell classes.  A cell's key is, per component, its self coefficient and for
// each curl coefficient its CPsi inside a band or the coefficient times the
// cell size outside (both are the coefficient before the kappa division times
// the cell size), plus what the update leaves alone.  Keys are hashed into an
// open-addressing table; then every cell writes its values where its class's
// row lacks them, and in a last pass compares what the step would look up with
// its own coefficients bit for bit.  Any difference (a key that does not
// determine the values, or two keys with one hash) fails the build, and the
// problem keeps the half-step path.
// ---------------------------------------------------------------------------
constexpr int kClassSlots = 1 << 18;
constexpr int kMaxClasses = 65536;   // 16-bit ids

struct ClassTable {
  unsigned long long* key;  // [kClassSlots], 0 = free
  unsigned* id;             // dense class of the slot
  int* count;               // [0] classes, [1] failed, [2] next id
};

struct ClassLayout {
  ClassRow row;
  int z0[2][2], zw[2][2];   // [H, E][n, p face]: slab start and width (0: none)
};

// Component extents, curl axes and Psi slots of component c (0..5 = Hx Hy Hz Ex Ey Ez).
__device__ constexpr int kCurlAxis[6][2] = {{2, 1}, {0, 2}, {1, 0}, {1, 2}, {2, 0}, {0, 1}};
__device__ constexpr int kCurlSlot[6][2] = {{0, 0}, {0, 1}, {1, 1}, {3, 2}, {3, 2}, {3, 2}};

template <typename T>
struct CellComp {
  bool exists, held;  // along x and y: the component has this (i, j); the bulk update leaves it alone
  bool used, psi;     // its coefficients / its CPsi are used at this k (see fused_hold)
  T c0, c[2], p[2];   // p: CPsi where the cell lies in a band of that axis
  int ci[2];          // band position (n face, then p face), -1 outside
};

// What component c has at (i, j, k), or past its last k at that last k: the
// class of a group at the wall is then that of the cells before it.
template <typename T, class C>
__device__ __forceinline__ CellComp<T> cell_comp(const StepParams<T, C>& s, int c, int i, int j, int k) {
  const int nx = s.g.nx, ny = s.g.ny, nz = s.g.nz;
  const bool el = c >= 3;
  const int ni = (c == 1 || c == 2 || c == 3) ? nx : nx + 1, nj = (c == 0 || c == 2 || c == 4) ? ny : ny + 1,
            nk = (c == 0 || c == 1 || c == 5) ? nz : nz + 1;
  CellComp<T> v{};
  v.ci[0] = v.ci[1] = -1;
  v.exists = i < ni && j < nj;
  if (!v.exists) return v;
  v.psi = k < nk;
  v.used = v.psi && !((c == 3 || c == 4) && (k == 0 || k == nz));
  k = min(k, nk - 1);
  const int idx = (i * nj + j) * nk + k, pos[3] = {i, j, k};
  T u[2];
  s.coef.get(c, idx, s.coef.invk((el ? 0 : 3) + kCurlAxis[c][0], pos[kCurlAxis[c][0]]),
             s.coef.invk((el ? 0 : 3) + kCurlAxis[c][1], pos[kCurlAxis[c][1]]), v.c0, v.c[0], v.c[1], u[0], u[1]);
  for (int w = 0; w < 2; w++) {
    const int a = kCurlAxis[c][w], slot = kCurlSlot[c][w];
    for (int side = 0; side < 2; side++) {
      const Face<T>& F = s.face[2 * a + side];
      const int ci = band_ci(F, pos[a], el);
      if (ci < 0) continue;
      const int pi = a == 0 ? (ci * nj + j) * nk + k : a == 1 ? (i * F.nc + ci) * nk + k : (i * nj + j) * F.nc + ci;
      v.p[w] = s.coef.cpsi(F, slot, pi, u[w], s.dcell[a]);
      v.ci[w] = (side ? s.face[2 * a].nc : 0) + ci;
    }
  }
  const bool jy = j >= 1 && j < ny;
  v.held = (c == 3 && !jy) || (c == 4 && i < 1) || (c == 5 && !(i >= 1 && jy));
  return v;
}

__device__ __forceinline__ unsigned long long value_bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ unsigned long long value_bits(double x) { return (unsigned long long)__double_as_longlong(x); }

template <typename T, class C>
__device__ __forceinline__ unsigned long long class_hash(const StepParams<T, C>& s, int i, int j, int k) {
  unsigned long long h = 0x9e3779b97f4a7c15ULL;
  auto mix = [&](unsigned long long w) {
    h = (h ^ w) * 0xff51afd7ed558ccdULL;
    h ^= h >> 32;
  };
  for (int c = 0; c < 6; c++) {
    const CellComp<T> v = cell_comp(s, c, i, j, k);
    mix(v.exists ? v.held ? 2 : 1 : 0);
    if (!v.exists) continue;
    mix(value_bits(v.c0));
    for (int w = 0; w < 2; w++) mix(value_bits(v.ci[w] >= 0 ? v.p[w] : mul(v.c[w], s.dcell[kCurlAxis[c][w]])));
  }
  return h ? h : 1;
}

// Where the step looks up curl coefficient w of component c at k: along z for
// every cell of a slab.
template <typename T>
__device__ __forceinline__ int curl_offset(const ClassLayout& L, int c, int w, const CellComp<T>& v, int k) {
  const int a = kCurlAxis[c][w], o = L.row.o[a] + kCurlSlot[c][w] * L.row.n[a], el = c >= 3;
  if (a == 2) {
    for (int side = 0; side < 2; side++) {
      const int d = k - L.z0[el][side];
      if (d >= 0 && d < L.zw[el][side]) return o + (side ? L.zw[el][0] : 0) + d;
    }
  } else if (v.ci[w] >= 0) {
    return o + v.ci[w];
  }
  return 4 * c + 1 + w;
}

struct CellAt {
  int i, j, k;
};
__device__ __forceinline__ CellAt cell_at(unsigned t, int pitch, int rows) {
  const unsigned r = t / (unsigned)pitch;
  return {(int)(r / (unsigned)rows), (int)(r % (unsigned)rows), (int)(t % (unsigned)pitch)};
}

__device__ __forceinline__ unsigned class_slot(const ClassTable& tb, unsigned long long h) {
  unsigned q = (unsigned)h & (kClassSlots - 1);
  while (tb.key[q] != h) q = (q + 1) & (kClassSlots - 1);  // ends: k_class_find left h in the table
  return q;
}

template <typename T, class C>
__global__ void __launch_bounds__(256) k_class_find(const __grid_constant__ StepParams<T, C> s, int pitch, unsigned n,
                                                    ClassTable tb) {
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    if (*(volatile int*)(tb.count + 1)) return;
    const CellAt x = cell_at(t, pitch, s.g.ny + 1);
    const unsigned long long h = class_hash(s, x.i, x.j, x.k);
    unsigned q = (unsigned)h & (kClassSlots - 1);
    for (int probe = 0;; probe++) {
      const unsigned long long have = tb.key[q];
      if (have == h) break;
      if (have == 0) {
        const unsigned long long old = atomicCAS(tb.key + q, 0ULL, h);
        if (old == 0) {
          const int id = atomicAdd(tb.count, 1);
          tb.id[q] = (unsigned)id;
          if (id >= kMaxClasses) tb.count[1] = 1;
          break;
        }
        if (old == h) break;
      }
      if (probe >= kClassSlots) {
        tb.count[1] = 1;
        break;
      }
      q = (q + 1) & (kClassSlots - 1);
    }
  }
}

// fill: the cells' ids, and the values their rows lack; otherwise the check.
template <typename T, class C>
__global__ void __launch_bounds__(256) k_class_rows(const __grid_constant__ StepParams<T, C> s, int pitch, unsigned n,
                                                    ClassTable tb, const __grid_constant__ ClassLayout L, T* tab,
                                                    unsigned short* cls, int fill) {
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const CellAt x = cell_at(t, pitch, s.g.ny + 1);
    const unsigned id = fill ? tb.id[class_slot(tb, class_hash(s, x.i, x.j, x.k))] : cls[t];
    if (fill) cls[t] = (unsigned short)id;
    T* row = tab + (size_t)id * L.row.stride;
    auto put = [&](int o, T v) {
      if (value_bits(row[o]) == value_bits(v)) return;
      if (fill)
        row[o] = v;
      else
        tb.count[1] = 1;
    };
    for (int c = 0; c < 6; c++) {
      const CellComp<T> v = cell_comp(s, c, x.i, x.j, x.k);
      const bool up = v.exists && !v.held;
      // a component that does not exist at this (i, j) is zero and stays so
      if (v.used || !v.exists) put(4 * c, up ? v.c0 : v.exists ? T(1) : T(0));
      for (int w = 0; w < 2; w++) {
        if (v.used || !v.exists) put(curl_offset(L, c, w, v, x.k), up ? v.c[w] : T(0));
        if (v.psi && v.ci[w] >= 0) put(kRowCpsi + 2 * c + w, v.p[w]);
      }
    }
  }
}

// Dense array (ni, nj, nk) <-> padded array with strides si, sj.
template <typename T>
__global__ void __launch_bounds__(256) k_repack(T* pad, long long si, long long sj, T* dense, int ni, int nj, int nk,
                                                int to_pad) {
  const long long n = (long long)ni * nj * nk;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(t % nk);
    const long long r = t / nk;
    T* q = pad + (r / nj) * si + (r % nj) * sj + k;
    if (to_pad)
      *q = dense[t];
    else
      dense[t] = *q;
  }
}

// ---------------------------------------------------------------------------
// Launchers (fdtd_fused.cu).
// ---------------------------------------------------------------------------
template <typename T, bool EXACT>
cudaError_t fused_step(const FusedParams<T>& p, bool early, cudaStream_t st);
template <typename T, bool EXACT>
cudaError_t fused_wall(const FusedParams<T>& p, cudaStream_t st);
template <typename T>
cudaError_t fused_epilogue(const FusedParams<T>& p, const FarField& ff, const Probes& pr, unsigned blocks,
                           bool late, bool early, cudaStream_t st);
template <typename T, class C>
cudaError_t fused_class_find(const StepParams<T, C>& s, int pitch, unsigned n, const ClassTable& tb, cudaStream_t st);
template <typename T, class C>
cudaError_t fused_class_rows(const StepParams<T, C>& s, int pitch, unsigned n, const ClassTable& tb,
                             const ClassLayout& layout, T* tab, unsigned short* cls, cudaStream_t st);
template <typename T>
cudaError_t fused_repack(T* pad, long long si, long long sj, T* dense, int ni, int nj, int nk, int to_pad,
                         cudaStream_t st);

}  // namespace fdtd
