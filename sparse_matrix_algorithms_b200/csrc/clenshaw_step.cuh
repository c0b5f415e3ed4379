// The fused Clenshaw step of CSR matrices and of the matrix-free models (1D Laplacian, 3D
// Anderson, XXZ chain), included by csr_clenshaw_f{64,32}.cu and model_clenshaw_f{64,32}.cu.
//
//   out[i, :] = ck*Q[i, :] + alpha * sum_j A[i,j] B1[j, :] + beta*B1[i, :] - B2[i, :]
//
// A thread owns V consecutive columns of one row (V*sizeof(T) = 32 bytes where the widths,
// strides and addresses allow it: one 256-bit access per neighbour row); a CTA of 128 threads
// owns the whole rows that fit.  Blocks wider than 64 vectors are cut into panels, the panel
// being the slow grid dimension, so that the neighbour rows of a panel are still in L2 when
// their last reader comes.
//
// What bounds it.  The n x b streams (Q, B1, B2, out) come from HBM when they exceed the L2,
// the neighbour rows from L2 (15 TB/s measured), and between a row's pointer, its column
// indices and its gathers lie two dependent latencies that only resident warps can hide.  So
// registers go to occupancy, not to operands in flight: at most U = 4 neighbour rows are held
// at a time, the epilogue's rows are prefetched into L2 at the start and loaded only after the
// gathers, and 40 registers keep 12 CTAs on an SM.  Measured on the 3D Anderson lattice
// (n = 262144, 7 entries a row), step after step on one B200, in a burst of some steps and in whole
// filters, which run under the power cap (SM clock 1.45-1.6 GHz):
//   FP32 b = 64   66 -> 43 us (6.6 TB/s of algorithmic bytes) and 50,  b = 768   640 -> 522 and 580,
//   FP64 b = 64  121 -> 85 us (6.6 TB/s) and 100.
// Against the kernel before it: 16-byte halves at a 32-byte stride doubled the L1 wavefronts
// (73 % of the LSU data pipe), and 63 registers left 45 % of the warps (DRAM 4.0 TB/s).
//
// Steps alternate the direction in which they walk the rows (rev): what the last CTAs of a
// step touched is what the first CTAs of the next read from L2 (FP64 b = 64: 97 -> 93 us).
//
// Steps are launched as programmatic dependents of the previous step (when the context allows
// it): a CTA reads what no step writes -- its row pointers -- and starts the prefetch of its
// row of Q, then waits for the previous grid before it touches B1 or B2 or writes anything.
//
// A model's CTA first writes the columns of its rows to shared memory, one thread per entry (the
// work of a whole row in each of its threads -- divisions, a sorting network, 64-80 registers --
// made the Anderson step 2.4 times slower than the CSR one: 96 us at n = 110592, b = 64 FP64);
// from there on it is a CSR matrix with one value on the diagonal and one off it.  XXZ rows of few
// threads are walked bit by bit instead, by each of those.
//
// Every configuration accumulates with FMA in ascending column order -- the order of the
// reference's CSC product on a symmetric matrix -- so all write bit-identical results
// (the XXZ model in its bond order).
#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "sma_internal.h"
#include "vec.cuh"

namespace sma {
namespace rows {

constexpr int kThreads = 128;
constexpr int kPanel = 64;  // vectors of a row in one panel

// What one launch needs; leading dimensions in bytes.
template <typename T>
struct Step {
  const int *rowptr, *colind;
  const T *val;
  sma_stencil model;  // the models' data, and the kind of operator they make up
  int kind;
  uint32_t entries;  // room for a model row's columns in shared memory
  const T *Q, *B1, *B2;
  T *out;
  const T *cseg;      // per-column coefficients (PC), else null
  const int *colseg;  // PC: the coefficient of column c is cseg[colseg[c]], or cseg[c] when null
  const T *topseg;    // PC: the highest coefficients, like cseg
  T *dots;            // DOTS: per CTA the sums of out B1 over its rows, `plane` later of B1 B1
  uint64_t plane;
  uint32_t dotcols;   // the columns that have them
  uint64_t ldq, ldb, ldo;
  T ck, top, alpha, beta;
  uint32_t n, b;      // rows, columns
  uint32_t lanes;     // vectors of a row in one panel
  uint32_t rows;      // rows of a CTA (rows * lanes <= kThreads)
  uint32_t divlanes;  // ceil(2^16 / lanes): i / lanes = i * divlanes >> 16 for i < 192
  int rev;
  bool tune;          // host: the step may be one of the autotuner's trials
};

template <typename T>
__device__ __forceinline__ const T *at(const T *p, uint64_t bytes) {
  return reinterpret_cast<const T *>(reinterpret_cast<const char *>(p) + bytes);
}

// Byte offset of a gathered row: 32 x 32 -> 64 bit product unless the leading dimension itself
// needs 64 bits (W).
template <bool W>
__device__ __forceinline__ uint64_t row_bytes(uint32_t row, uint64_t ld) {
  if constexpr (W) return (uint64_t)row * ld;
  return (uint64_t)row * (uint32_t)ld;
}

// Where a row's entries come from.
template <typename T>
struct CsrRow {
  const int *cols;
  const T *vals;
  __device__ __forceinline__ int col(int j) const { return __ldg(cols + j); }
  __device__ __forceinline__ T val(int j) const { return __ldg(vals + j); }
};
template <typename T>
struct ModelRow {  // entry `dpos` is the diagonal
  const int *cols;
  int dpos;
  T diag, off;
  __device__ __forceinline__ int col(int j) const { return cols[j]; }
  __device__ __forceinline__ T val(int j) const { return j == dpos ? diag : off; }
};

// What the gathered rows are multiplied with before they enter the product: nothing, or in the
// first step of a recurrence the highest coefficient (rounded like the block c_K Q it replaces).
struct Unscaled {
  template <typename T>
  __device__ __forceinline__ T operator()(T x, int) const { return x; }
};
template <typename T, int V>
struct Scaled {
  const T (&c)[V];
  __device__ __forceinline__ T operator()(T x, int i) const { return mul_rn(c[i], x); }
};

// The V columns of a thread, from the one that its pointers are at: next to each other, in one
// access; or (STRIDED) a row's threads apart, V accesses of one element, those past the row left out.
template <typename T, int V, bool STRIDED>
struct Columns {
  uint32_t step;  // STRIDED: between two columns
  int count;      // STRIDED: those that there are
  static constexpr bool kStrided = STRIDED;
  template <bool KEEP = true>
  __device__ __forceinline__ void load(const T *p, T (&f)[V]) const {
    if constexpr (STRIDED) load_if(true, p, f);
    else ldv<T, V, KEEP>(p, f);
  }
  __device__ __forceinline__ void load_if(bool ok, const T *p, T (&f)[V]) const {
    if constexpr (STRIDED) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        T x[1];
        ldv_if<T, 1>(ok && i < count, p + (uint64_t)i * step, x);
        f[i] = x[0];
      }
    } else {
      ldv_if<T, V>(ok, p, f);
    }
  }
  __device__ __forceinline__ void store(T *p, const T (&f)[V]) const {
    if constexpr (STRIDED) {
#pragma unroll
      for (int i = 0; i < V; ++i)
        if (i < count) p[(uint64_t)i * step] = f[i];
    } else {
      stv<T, V>(p, f);
    }
  }
};

// R consecutive entries from j: all R gathers are issued before the first FMA; FMAs in
// ascending entry order.
template <typename T, int V, int R, bool W, typename Row, typename C, typename F>
__device__ __forceinline__ void chunk(const Row &row, int j, const T *B1c, uint64_t ldb, T (&acc)[V],
                                      const C &cols, F f) {
  int c[R];
  T x[R][V], v[R];
#pragma unroll
  for (int u = 0; u < R; ++u) c[u] = row.col(j + u);
#pragma unroll
  for (int u = 0; u < R; ++u) cols.load(at(B1c, row_bytes<W>((uint32_t)c[u], ldb)), x[u]);
#pragma unroll
  for (int u = 0; u < R; ++u) v[u] = row.val(j + u);
#pragma unroll
  for (int u = 0; u < R; ++u)
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = fma(v[u], f(x[u][i], i), acc[i]);
}

// acc += the row's entries [j, end): chunks of U, then the r < U remaining entries as ONE chunk
// of exactly r (a switch over r).
template <typename T, int V, int U, bool W, typename Row, typename C, typename F>
__device__ __forceinline__ void row_product(const Row &row, int j, int end, const T *B1c,
                                            uint64_t ldb, T (&acc)[V], const C &cols, F f) {
  for (; j + U <= end; j += U) chunk<T, V, U, W>(row, j, B1c, ldb, acc, cols, f);
  switch (end - j) {
    case 7: if constexpr (U > 7) chunk<T, V, 7, W>(row, j, B1c, ldb, acc, cols, f); break;
    case 6: if constexpr (U > 6) chunk<T, V, 6, W>(row, j, B1c, ldb, acc, cols, f); break;
    case 5: if constexpr (U > 5) chunk<T, V, 5, W>(row, j, B1c, ldb, acc, cols, f); break;
    case 4: if constexpr (U > 4) chunk<T, V, 4, W>(row, j, B1c, ldb, acc, cols, f); break;
    case 3: chunk<T, V, 3, W>(row, j, B1c, ldb, acc, cols, f); break;
    case 2: chunk<T, V, 2, W>(row, j, B1c, ldb, acc, cols, f); break;
    case 1: chunk<T, V, 1, W>(row, j, B1c, ldb, acc, cols, f); break;
    default: break;
  }
}

// The same for rows of unequal lengths: chunks of U whose accesses past the row's end are
// predicated off (the entry arrays are readable that far, kRowPad).  The rows of a warp then walk
// one code path; with the exact chunks above each remainder is a path of its own, and the warp
// waits for the gathers of all of them in turn (XXZ L = 16, b = 32: 5.3 -> 4.0 us a step FP64,
// 4.1 -> 3.1 FP32; L = 18 13.2 -> 12.3).  An absent entry adds 0 * 0.
template <typename T, int V, int U, bool W, typename Row, typename C, typename F>
__device__ __forceinline__ void ragged_product(const Row &row, int j, int end, const T *B1c,
                                               uint64_t ldb, T (&acc)[V], const C &cols, F f) {
  for (; j < end; j += U) {
    int c[U];
    T x[U][V], v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = row.col(j + u);
#pragma unroll
    for (int u = 0; u < U; ++u)
      cols.load_if(j + u < end, at(B1c, row_bytes<W>((uint32_t)c[u], ldb)), x[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      v[u] = row.val(j + u);
      if (j + u >= end) v[u] = T(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = fma(v[u], f(x[u][i], i), acc[i]);
  }
}

// ------------------------------------------------------------------ the models' rows
// Entry u of model row `row`: its place among the row's entries in accumulation order and its
// column, or place -1 when the row has no such entry.
struct Entry {
  int place, col;
};

// tridiag(-1, 2, -1): u = 0, 1, 2 are the columns row - 1, row, row + 1, evaluated as the
// reference's lap1d_matblock! (polfed.jl:1209-1219) -x[i-1] + 2 x[i] - x[i+1].
__device__ __forceinline__ Entry lap1d_entry(uint32_t row, uint32_t n, int u) {
  const int64_t col = (int64_t)row + u - 1;
  if (col < 0 || col >= n) return {-1, 0};
  return {row == 0 ? u - 1 : u, (int)col};
}

// 3D Anderson model on an L^3 periodic lattice, row i = x + L (y + L z): u = 0 is the diagonal,
// 1..6 the neighbours x+-1, y+-1, z+-1 (distinct for L >= 3).  An entry's place is the number of
// smaller columns: the order of the stored matrix's CSR row.
__device__ __forceinline__ Entry anderson_entry(uint32_t row, uint32_t L, int u) {
  const uint32_t l2 = L * L, z = row / l2, rem = row - z * l2, y = rem / L, x = rem - y * L;
  const int r = (int)row, l = (int)L, ll = (int)l2;
  const int c[7] = {r,
                    x + 1 == L ? r - (l - 1) : r + 1,      x == 0 ? r + (l - 1) : r - 1,
                    y + 1 == L ? r - (l - 1) * l : r + l,  y == 0 ? r + (l - 1) * l : r - l,
                    z + 1 == L ? r - (l - 1) * ll : r + ll, z == 0 ? r + (l - 1) * ll : r - ll};
  int mine = c[0], place = 0;
#pragma unroll
  for (int k = 1; k < 7; ++k) mine = k == u ? c[k] : mine;
#pragma unroll
  for (int k = 0; k < 7; ++k) place += c[k] < mine;
  return {place, mine};
}

// Random-field XXZ chain of length L in the Sz = 0 sector.  Row r is the basis state s =
// states[r] (bit i = site i up); its index is its combinatorial rank sum_j C(p_j, j) over its set
// bits p_1 < p_2 < ... .  u = 0 is the diagonal; u = i + 1 flips the antiparallel bond (i, i + 1),
// which moves one set bit by one position and the rank by +-C(i, k), k the number of set bits
// below i; u = L flips the periodic bond (L-1, 0) and ranks the flipped state.  Places in bond
// order.
__device__ __forceinline__ Entry xxz_entry(uint32_t row, const sma_stencil &m, int u) {
  if (u == 0) return {0, (int)row};
  const unsigned s = __ldg(m.states + row);
  const int i = u - 1;
  const unsigned flips = s ^ (s >> 1);  // bit i: bond (i, i + 1) is antiparallel, i < L - 1
  const unsigned below = (1u << i) - 1u;
  const int place = 1 + __popc(flips & below);
  if (u < m.L) {
    if (!((flips >> i) & 1u)) return {-1, 0};
    const int d = __ldg(m.binom + i * 17 + __popc(s & below));
    return {place, (s >> i) & 1u ? (int)row + d : (int)row - d};
  }
  if (!(((s >> (m.L - 1)) ^ s) & 1u)) return {-1, 0};
  unsigned t = s ^ (1u | (1u << (m.L - 1)));
  int col = 0;
  for (int j = 1; t; ++j) {
    col += __ldg(m.binom + (__ffs(t) - 1) * 17 + j);
    t &= t - 1;
  }
  return {place, col};
}

// The columns of the CTA's rows [row0, row0 + rows) into cols (a.entries each), their number into
// cnt and the place of the diagonal into dpos: one thread per entry.
template <typename T>
__device__ __forceinline__ void model_rows(const Step<T> &a, uint32_t row0, int *cols, int *cnt,
                                           int *dpos) {
  const sma_stencil &m = a.model;
  if (threadIdx.x < a.rows) cnt[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < a.rows * a.entries; e += kThreads) {
    const uint32_t r = e / a.entries, row = row0 + r;
    const int u = (int)(e - r * a.entries);
    if (row >= a.n) continue;
    const Entry x = a.kind == OP_LAP1D      ? lap1d_entry(row, a.n, u)
                    : a.kind == OP_ANDERSON ? anderson_entry(row, (uint32_t)m.L, u)
                                            : xxz_entry(row, m, u);
    if (x.place < 0) continue;
    cols[r * a.entries + x.place] = x.col;
    if (x.col == (int)row) dpos[r] = x.place;
    atomicAdd(cnt + r, 1);
  }
  __syncthreads();
}

// An XXZ row walked bit by bit by each thread that takes columns of it, for rows of few threads: in
// shared memory the L + 1 places of such a row are filled by about as many threads as then read them.
struct Walk {
  unsigned state, todo;  // bit i of todo: bond (i, i + 1) still to come, the periodic one is bit L - 1
  uint32_t periodic;     // its column
};

__device__ __forceinline__ Walk xxz_walk(const sma_stencil &m, uint32_t row) {
  const unsigned s = __ldg(m.states + row);
  const Entry p = xxz_entry(row, m, m.L);
  const unsigned bonds = (s ^ (s >> 1)) & ((1u << (m.L - 1)) - 1u);
  return {s, bonds | (p.place < 0 ? 0u : 1u << (m.L - 1)), (uint32_t)p.col};
}

// acc += the walked row: the diagonal and the bonds in ascending order (the places of xxz_entry), U at
// a time, the last of them predicated like ragged rows.
template <typename T, int V, int U, bool W, typename F>
__device__ __forceinline__ void walk_product(const sma_stencil &m, Walk w, uint32_t row, T diag, T off,
                                             const T *B1c, uint64_t ldb, T (&acc)[V], F f) {
  const unsigned last = 1u << (m.L - 1);
  bool first = true;
  do {
    T x[U][V], v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      uint32_t col = row;
      bool there = true;
      v[u] = off;
      if (u == 0 && first) {
        v[u] = diag;
      } else {
        there = w.todo != 0;
        const unsigned bit = w.todo & -w.todo;
        w.todo ^= bit;
        if (bit == last) {
          col = w.periodic;
        } else if (there) {
          const int d = __ldg(m.binom + (__ffs(bit) - 1) * 17 + __popc(w.state & (bit - 1u)));
          col = w.state & bit ? row + d : row - d;
        }
        if (!there) v[u] = T(0);
      }
      ldv_if<T, V>(there, at(B1c, row_bytes<W>(col, ldb)), x[u]);
    }
    first = false;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = fma(v[u], f(x[u][i], i), acc[i]);
  } while (w.todo);
}

// The coefficients of the thread's V columns: c in all, or from cseg.
template <typename T, int V, bool PC, typename C>
__device__ __forceinline__ void coefficients(const Step<T> &a, T c, const T *cseg, uint32_t c0, const C &cols,
                                             T (&ck)[V]) {
  if constexpr (!PC) {
#pragma unroll
    for (int i = 0; i < V; ++i) ck[i] = c;
  } else if (a.colseg == nullptr) {  // one polynomial per column: its coefficients side by side
    cols.load(cseg + c0, ck);
  } else {  // segments are runs of columns: equal ends, one coefficient
    const uint32_t step = C::kStrided ? cols.step : 1;
    const int count = C::kStrided ? cols.count : V;
    const int s0 = __ldg(a.colseg + c0), s1 = __ldg(a.colseg + c0 + (count - 1) * step);
    ck[0] = __ldg(cseg + s0);
#pragma unroll
    for (int i = 1; i < V; ++i)
      ck[i] = s0 == s1 || i >= count ? ck[0] : __ldg(cseg + __ldg(a.colseg + c0 + i * step));
  }
}

// Where in a recurrence a step stands.  B1 = c_K Q, the block that it starts from, is never
// written: the first step gathers it from Q, and the second, whose B2 it is, has Q's row anyway.
// DOTS: an inner step that also sums out B1 and B1 B1 down the columns of its CTA's rows, of which
// it holds both factors.
enum Form { INNER, FIRST, SECOND, DOTS };

// Where the rows' entries come from: a stored matrix, a model's columns in shared memory, or walked.
enum Rows { STORED, SHARED, WALKED };

// HQ, HS, HB: whether the terms with Q, B1's own row and B2 are there.  CTAS: CTAs an SM holds.
// FLAT: a CTA does not take whole rows, its threads go on in the next row where the CTA before ended.
template <typename T, int V, int U, int CTAS, bool HQ, bool HS, bool HB, bool PC, bool W, int MODEL,
          bool RAGGED, Form P, bool FLAT, bool STRIDED>
__global__ void __launch_bounds__(kThreads, CTAS) step_kernel(const Step<T> a) {
  extern __shared__ int model_smem[];  // a.rows x a.entries columns, then counts and places
  const uint32_t bx = a.rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
  const uint32_t by = a.rev ? gridDim.y - 1 - blockIdx.y : blockIdx.y;
  static_assert(!FLAT || !(MODEL != STORED || P == DOTS), "these need whole rows");
  static_assert(!STRIDED || !(MODEL == WALKED || P == DOTS), "not with these");
  uint32_t row0 = bx * a.rows, i = threadIdx.x;
  if constexpr (FLAT) {
    row0 = bx * kThreads / a.lanes;
    i += bx * kThreads - row0 * a.lanes;
  }
  const uint32_t r = i * a.divlanes >> 16;
  uint32_t row = row0 + r;
  uint32_t c0 = (by * a.lanes + i - r * a.lanes) * V;
  if constexpr (STRIDED) c0 = by * a.lanes * V + i - r * a.lanes;
  const bool in = (FLAT || r < a.rows) && row < a.n && c0 < a.b;
  Columns<T, V, STRIDED> cols{};
  if constexpr (STRIDED) cols = {a.lanes, in ? (int)min((uint32_t)V, (a.b - c0 + a.lanes - 1) / a.lanes) : 0};
  int start = 0, end = 0;
  if (in) {
    if constexpr (MODEL == STORED) {
      start = __ldg(a.rowptr + row);
      end = __ldg(a.rowptr + row + 1);
    }
    if constexpr (HQ && !STRIDED) prefetch_l2(at(a.Q + c0, row * a.ldq));
  }
  int *cnt = model_smem + a.rows * a.entries, *dpos = cnt + a.rows;
  if constexpr (MODEL == SHARED) model_rows(a, bx * a.rows, model_smem, cnt, dpos);
  Walk walk{};
  if constexpr (MODEL == WALKED)
    if (in) walk = xxz_walk(a.model, row);
  pdl_wait_then_trigger();
  if constexpr (P != DOTS) {
    if (!in) return;
  }
  T dot[P == DOTS ? 2 * V : 1] = {};
  if (P != DOTS || in) {
    if constexpr (MODEL == SHARED) row = after_wait(row);  // B1's places come from shared memory
    else c0 = after_wait(c0);
    const uint64_t own = row * a.ldb;
    if constexpr (HB && P != SECOND && !STRIDED) prefetch_l2(at(a.B2 + c0, own));
    T acc[V], top[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = T(0);
    if constexpr (P == FIRST) coefficients<T, V, PC>(a, a.top, a.topseg, c0, cols, top);
    auto product = [&](const auto &row, int j, int end, auto f) {
      if constexpr (RAGGED) ragged_product<T, V, U, W>(row, j, end, a.B1 + c0, a.ldb, acc, cols, f);
      else row_product<T, V, U, W>(row, j, end, a.B1 + c0, a.ldb, acc, cols, f);
    };
    auto gather = [&](const auto &row, int j, int end) {
      if constexpr (P == FIRST) product(row, j, end, Scaled<T, V>{top});
      else product(row, j, end, Unscaled{});
    };
    if constexpr (MODEL == WALKED) {
      const T diag = (T)__ldg(a.model.diag + row), off = (T)a.model.hop;
      if constexpr (P == FIRST)
        walk_product<T, V, U, W>(a.model, walk, row, diag, off, a.B1 + c0, a.ldb, acc, Scaled<T, V>{top});
      else
        walk_product<T, V, U, W>(a.model, walk, row, diag, off, a.B1 + c0, a.ldb, acc, Unscaled{});
    } else if constexpr (MODEL == SHARED) {
      const T diag = a.kind == OP_LAP1D ? T(2) : (T)__ldg(a.model.diag + row);
      gather(ModelRow<T>{model_smem + r * a.entries, dpos[r], diag, (T)a.model.hop}, 0, cnt[r]);
    } else {
      gather(CsrRow<T>{a.colind, a.val}, start, end);
    }
    T q[V], s[V], t[V], ck[V], o[V];
    if constexpr (HQ) cols.template load<false>(at(a.Q + c0, row * a.ldq), q);
    if constexpr (HB && P != SECOND) cols.template load<false>(at(a.B2 + c0, own), t);
    if constexpr (HS && P != FIRST) cols.load(at(a.B1 + c0, own), s);
    if constexpr (HQ) coefficients<T, V, PC>(a, a.ck, a.cseg, c0, cols, ck);
    if constexpr (P == SECOND) coefficients<T, V, PC>(a, a.top, a.topseg, c0, cols, top);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if constexpr (P == FIRST) s[i] = mul_rn(top[i], q[i]);
      if constexpr (P == SECOND) t[i] = mul_rn(top[i], q[i]);
    }
#pragma unroll
    for (int i = 0; i < V; ++i)
      o[i] = clenshaw_combine<HQ, HS, HB>(acc[i], q[i], s[i], t[i], ck[i], a.alpha, a.beta);
    cols.store(const_cast<T *>(at(a.out + c0, row * a.ldo)), o);
    if constexpr (P == DOTS) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        dot[i] = o[i] * s[i];
        dot[V + i] = s[i] * s[i];
      }
    }
  }
  // A tree over the CTA's rows, whose order depends on their number alone; shuffles where whole rows
  // share a warp at power-of-two distances (XXZ L = 20, 256 moments of 16 vectors: 4.38 ms against
  // 4.73 with the tree in shared memory throughout, 5.43 with a pass of its own).
  if constexpr (P == DOTS) {
    if ((a.lanes & (a.lanes - 1)) == 0 && a.lanes <= 16) {
      __shared__ T red[4][2 * V][16];
      for (uint32_t o = 16; o >= a.lanes; o /= 2)
#pragma unroll
        for (int k = 0; k < 2 * V; ++k) dot[k] += __shfl_down_sync(~0u, dot[k], o);
      const uint32_t l = threadIdx.x % 32, w = threadIdx.x / 32;
      if (w && l < a.lanes)
#pragma unroll
        for (int k = 0; k < 2 * V; ++k) red[w][k][l] = dot[k];
      __syncthreads();
      if (r == 0)
#pragma unroll
        for (int k = 0; k < 2 * V; ++k) dot[k] += red[1][k][l] + (red[2][k][l] + red[3][k][l]);
    } else {
      __shared__ T red[2 * V][kThreads];
#pragma unroll
      for (int k = 0; k < 2 * V; ++k) red[k][threadIdx.x] = dot[k];
      for (uint32_t rows = a.rows; rows > 1;) {
        const uint32_t half = (rows + 1) / 2;
        __syncthreads();
        if (r + half < rows) {
#pragma unroll
          for (int k = 0; k < 2 * V; ++k)
            red[k][threadIdx.x] = dot[k] += red[k][threadIdx.x + half * a.lanes];
        }
        rows = half;
      }
    }
    if (r == 0) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        if (c0 + i >= a.dotcols) break;
        a.dots[(uint64_t)bx * a.dotcols + c0 + i] = dot[i];
        a.dots[a.plane + (uint64_t)bx * a.dotcols + c0 + i] = dot[V + i];
      }
    }
  }
}

}  // namespace rows
}  // namespace sma

#include "csr_bulk.cuh"

namespace sma {
namespace rows {

// ------------------------------------------------------------------ launch
template <typename T, int V, int U, int CTAS, bool HQ, bool HS, bool HB, bool PC, bool W, int MODEL,
          bool RAGGED, Form P, bool FLAT = false, bool STRIDED = false>
void launch(const sma_op *op, cudaStream_t st, const Step<T> &a, dim3 grid) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  if (MODEL == SHARED) cfg.dynamicSmemBytes = (a.rows * (a.entries + 2) + kRowPad) * sizeof(int);  // 18 KB at most
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // the first step gathers the caller's Q, which the grid before may have read and written in
  // place: it starts after that grid has ended, with nothing of it in L1
  cfg.numAttrs = op->ctx->pdl && P != FIRST ? 1 : 0;
  SMA_CUDA(cudaLaunchKernelEx(&cfg, step_kernel<T, V, U, CTAS, HQ, HS, HB, PC, W, MODEL, RAGGED, P, FLAT, STRIDED>, a));
  SMA_CHECK_LAUNCH();
}

inline bool ragged(const sma_op *op) { return op->kind == OP_XXZ || op->ragged; }

// Vectors of a panel: the whole row up to kPanel; else a multiple of 4 (128 bytes), with as few
// panels as need be, or up to twice as many if more of a CTA's threads then have work (a CTA takes
// whole rows of a panel, so 48 lanes leave a quarter idle: 96 vectors in 3 panels instead of 2, us
// a step, Anderson L = 64 FP32 598 -> 582, XXZ L = 18 FP64 150 -> 141; 66 in 3 124 -> 117).  A
// row that fits one panel stays in one: in two, 43 vectors took 114 -> 122 us (Anderson L = 48).
inline uint32_t panel_lanes(uint32_t vecs) {
  if (vecs <= kPanel) return vecs;
  const uint32_t fewest = (vecs + kPanel - 1) / kPanel;
  uint32_t best = 0;
  double most = 0.0;
  for (uint32_t p = fewest; p <= 2 * fewest; ++p) {
    const uint32_t lanes = ((vecs + p - 1) / p + 3) / 4 * 4;
    const double work = (double)(kThreads / lanes * lanes) * vecs / ((vecs + lanes - 1) / lanes * lanes);
    if (work > 1.02 * most) {
      most = work;
      best = lanes;
    }
  }
  return best;
}

// XXZ rows are walked where few threads share one: at most 6, or 16 in a stream of a wave and more
// (us a step, places in shared memory and walked: L = 16, b = 1 FP64 17.8 and 4.4, b = 6 6.0 and 4.6;
// L = 20, b = 8 45.5 and 16.8, b = 32 67.9 and 57.2; L = 22, b = 64 530 and 517; on the other side
// L = 14, b = 32 3.3 and 4.7; L = 16, b = 32 6.2 and 6.9; L = 20, b = 128 224 and 238).
inline bool walked(const sma_op *op, uint32_t lanes, int64_t threads) {
  return op->kind == OP_XXZ && (lanes <= 6 || (lanes <= 16 && threads >= 8LL * kThreads * op->ctx->num_sms));
}

// Where not 0 or negative, `gathers` and `flat` take the place of the rules for them.
template <typename T, int V, bool HQ, bool HS, bool HB, bool PC, bool W, int MODEL, Form P, bool STRIDED = false>
void launch_width(const sma_op *op, cudaStream_t st, Step<T> a, int gathers = 0, int flat_wanted = -1) {
  const uint32_t vecs = (a.b + V - 1) / V;
  a.lanes = panel_lanes(vecs);
  // FP64 rows of 4 and 5 such threads take one more, three columns each: b = 15 and 17 at n = 50000,
  // 41.0 -> 38.3 and 43.5 -> 42.3 us (three steps, five entries a row), b = 13 33.5 either way
  if (STRIDED && sizeof(T) == 8 && (vecs == 4 || vecs == 5)) ++a.lanes;
  a.rows = kThreads / a.lanes;
  a.divlanes = (65536 + a.lanes - 1) / a.lanes;
  if constexpr (MODEL == SHARED && !STRIDED)
    if (walked(op, a.lanes, (int64_t)a.n * vecs)) return launch_width<T, V, HQ, HS, HB, PC, W, WALKED, P>(op, st, a);
  // Waves of 8-CTA residency decide what a step's time is.  Six and more: a stream, which wants
  // every warp it can get.  Below, more and more a latency, which wants more gathers in flight at
  // less occupancy -- unless a row has no more than four.  Us a step, step after step:
  //   Anderson L = 20, b = 64 FP64 (0.85 waves)  exact U = 8 4.0, U = 4 5.6
  //   Anderson L = 64, b = 64 FP32 (14)          exact U = 8 43.8, U = 4 42.5
  //   1D Laplacian n = 20000, b = 32 FP32 (0.5)  exact U = 8 3.2, U = 4 2.9
  //   XXZ L = 16, b = 32 FP64 (0.7)              ragged U = 8 4.5, U = 6 5.7, U = 4 5.5
  //   XXZ L = 18, b = 32 FP64 (2.6)              ragged U = 8 13.4, U = 6 13.1, U = 4 13.6
  //   XXZ L = 20, b = 64 FP32 (9.8)              ragged U = 6 51.0, U = 4 48.0
  const int64_t wave = 8LL * kThreads * op->ctx->num_sms, threads = (int64_t)a.n * vecs;
  const bool uneven = ragged(op);
  if (gathers == 0)
    gathers = threads >= 6 * wave || op->nnz <= 4 * op->n ? 4 : uneven && threads >= 2 * wave ? 6 : 8;
  // Whole rows leave threads idle where lanes do not divide 128.  Going on in the next row instead
  // takes a division per CTA and lets warps straddle rows: the better way for streams, unless whole
  // warps are idle or a few threads of long rows (us a step, whole rows and flat, Anderson L = 48:
  // 13 lanes 34.1 and 32.6, 22 55.8 and 52.0, 43 117 and 107, 50 143 and 128; 48 120 and 121, 60
  // 152 and 155).
  constexpr bool kFlat = !(MODEL != STORED || P == DOTS || P == FIRST || STRIDED);
  const uint32_t used = a.rows * a.lanes;
  const bool flat = kFlat && gathers != 8 && used < kThreads && (uint64_t)a.n * a.lanes < (uint64_t)1 << 32 &&
                    (flat_wanted < 0 ? used % 32 != 0 && (a.lanes <= 40 || kThreads - used >= 16) : flat_wanted > 0);
  const uint32_t gx = flat ? (uint32_t)(((uint64_t)a.n * a.lanes + kThreads - 1) / kThreads)
                           : (a.n + a.rows - 1) / a.rows;
  constexpr uint32_t kGridY = 65535;
  const uint32_t ny = (vecs + a.lanes - 1) / a.lanes;
  const uint32_t span = kGridY * a.lanes * V, width = a.b;
  for (uint32_t p = 0; p < ny; p += kGridY) {  // more than one pass only beyond 65535 panels
    if (p) {
      a.B1 += span;
      a.out += span;
      if (HQ) a.Q += span;
      if (HB) a.B2 += span;
      if (PC) { if (a.colseg) a.colseg += span; else { a.cseg += span; if (P != INNER) a.topseg += span; } }
    }
    a.b = width - p * a.lanes * V;
    const dim3 grid(gx, std::min(kGridY, ny - p));
    if constexpr (STRIDED) {  // four addresses a gather
      if (uneven) launch<T, V, 4, 8, HQ, HS, HB, PC, W, MODEL, true, P, false, true>(op, st, a, grid);
      else launch<T, V, 4, 8, HQ, HS, HB, PC, W, MODEL, false, P, false, true>(op, st, a, grid);
      continue;
    }
    // A walked row holds its state beside the gathers: two at a time of 16-byte FP64 and of 32-byte
    // vectors, whose four spill (L = 22, b = 8 FP64 63.5 us against 87), four of the others.
    if constexpr (MODEL == WALKED) {
      constexpr bool kTwo = V * sizeof(T) == 32 || (sizeof(T) == 8 && V == 2);
      constexpr int kCtas = !kTwo || P == FIRST || P == DOTS ? 8 : 12;
      launch<T, V, kTwo ? 2 : 4, kCtas, HQ, HS, HB, PC, W, MODEL, true, P>(op, st, a, grid);
    } else if constexpr (P == FIRST) {  // the coefficients take registers too, and it is one step
      if (uneven) launch<T, V, 6, 8, HQ, HS, HB, PC, W, MODEL, true, P>(op, st, a, grid);
      else launch<T, V, 4, 8, HQ, HS, HB, PC, W, MODEL, false, P>(op, st, a, grid);
    } else if (gathers == 8) {
      if (uneven) launch<T, V, 8, 6, HQ, HS, HB, PC, W, MODEL, true, P>(op, st, a, grid);
      else launch<T, V, 8, 8, HQ, HS, HB, PC, W, MODEL, false, P>(op, st, a, grid);
    } else if (gathers == 6 && uneven) {
      if (flat) launch<T, V, 6, 8, HQ, HS, HB, PC, W, MODEL, true, P, kFlat>(op, st, a, grid);
      else launch<T, V, 6, 8, HQ, HS, HB, PC, W, MODEL, true, P>(op, st, a, grid);
    } else if (uneven) {
      if (flat) launch<T, V, 4, 12, HQ, HS, HB, PC, W, MODEL, true, P, kFlat>(op, st, a, grid);
      else launch<T, V, 4, 12, HQ, HS, HB, PC, W, MODEL, true, P>(op, st, a, grid);
    } else {
      if (flat) launch<T, V, 4, 12, HQ, HS, HB, PC, W, MODEL, false, P, kFlat>(op, st, a, grid);
      else launch<T, V, 4, 12, HQ, HS, HB, PC, W, MODEL, false, P>(op, st, a, grid);
    }
  }
}

// ------------------------------------------------------------------ the autotuner
// With SMA_AUTOTUNE=1 the first launches of each shape of an operator with n >= 20000 run every
// configuration in turn, four times, on the real steps, bracketed by events, and the fastest is kept:
// for matrices that the rules, which were measured on lattices, chains and rings of up to 100 entries
// a row, may not fit.  SMA_AUTOTUNE_VERBOSE=1 does the same and prints the table, as a check of the
// rules: what it found is kept only with SMA_AUTOTUNE=1.  With neither the rules alone choose.
struct Config {
  bool bulk;
  int V, gathers, flat;
};

template <typename T, bool HQ, bool HS, bool HB, bool PC>
void launch_config(const sma_op *op, cudaStream_t st, const Step<T> &a, const Config &c) {
  auto with = [&](auto width) {
    constexpr int V = decltype(width)::value;
    if constexpr (!PC)
      if (c.bulk) return launch_bulk<T, V, HQ, HS, HB>(op, st, a);
    launch_width<T, V, HQ, HS, HB, PC, false, false, INNER>(op, st, a, c.gathers, c.flat);
  };
  if constexpr (sizeof(T) == 4)
    if (c.V == 8) return with(std::integral_constant<int, 8>{});
  if (c.V == 4) return with(std::integral_constant<int, 4>{});
  if (c.V == 2) return with(std::integral_constant<int, 2>{});
  with(std::integral_constant<int, 1>{});
}

// Whole rows and flat ones, with every number of gathers that there is, at the widest vectors and at
// half of them; the BULK family where it fits.
template <typename T, bool HQ, bool HS, bool HB, bool PC>
std::vector<Config> configs(const sma_op *op, const Step<T> &a, int widest) {
  std::vector<Config> all;
  for (int v = widest; v >= 1 && 2 * v >= widest; v /= 2) {
    const uint32_t lanes = panel_lanes(a.b / v);
    for (int gathers : {8, 6, 4}) {
      if (gathers == 6 && !ragged(op)) continue;
      all.push_back({false, v, gathers, 0});
      if (gathers != 8 && kThreads % lanes) all.push_back({false, v, gathers, 1});
    }
  }
  if constexpr (!PC) {
    bool fits = widest == 4 ? bulk_fits<T, 4, HQ, HS, HB>(op, a) : widest == 2 ? bulk_fits<T, 2, HQ, HS, HB>(op, a)
                                                                              : false;
    if constexpr (sizeof(T) == 4) fits = widest == 8 ? bulk_fits<T, 8, HQ, HS, HB>(op, a) : fits;
    if (fits) all.push_back({true, widest, 0, 0});
  }
  return all;
}

// v: the rule's vector width.
template <typename T, bool HQ, bool HS, bool HB, bool PC>
bool tuned_step(const sma_op *op, cudaStream_t st, const Step<T> &a, int widest, int v) {
  const sma_ctx *ctx = op->ctx;
  if (!(ctx->tune || ctx->tune_verbose) || !a.tune || op->n < 20000) return false;
  cudaStreamCaptureStatus cap;
  SMA_CUDA(cudaStreamIsCapturing(st, &cap));
  const std::vector<Config> cfg = configs<T, HQ, HS, HB, PC>(op, a, widest);
  CsrTune &t = const_cast<sma_op *>(op)->tuned[{(int64_t)sizeof(T) * 16 + widest,
                                                cfg.back().bulk * 16 + HQ * 8 + HS * 4 + HB * 2 + PC, a.b}];
  if (t.done && !ctx->tune) return false;
  if (t.done) {
    launch_config<T, HQ, HS, HB, PC>(op, st, a, cfg[t.fastest]);
    return true;
  }
  if (cap != cudaStreamCaptureStatusNone) return false;
  if (cfg.back().bulk && !op->bulk_err) {
    SMA_CUDA(cudaMalloc((void **)&const_cast<sma_op *>(op)->bulk_err, sizeof(int)));
    SMA_CUDA(cudaMemset(op->bulk_err, 0, sizeof(int)));
  }
  cudaEvent_t e[2];
  const size_t i = t.events.size() / 2;
  for (cudaEvent_t &x : e) {
    SMA_CUDA(cudaEventCreate(&x));
    t.events.push_back(x);
  }
  SMA_CUDA(cudaEventRecord(e[0], st));
  launch_config<T, HQ, HS, HB, PC>(op, st, a, cfg[i % cfg.size()]);
  SMA_CUDA(cudaEventRecord(e[1], st));
  if (i + 1 < 4 * cfg.size()) return true;
  SMA_CUDA(cudaEventSynchronize(e[1]));
  std::vector<float> best(cfg.size(), INFINITY);
  for (size_t k = 0; k <= i; ++k) {
    float ms = 0.f;
    SMA_CUDA(cudaEventElapsedTime(&ms, t.events[2 * k], t.events[2 * k + 1]));
    best[k % cfg.size()] = std::min(best[k % cfg.size()], ms);
  }
  t.release();
  t.fastest = (int)(std::min_element(best.begin(), best.end()) - best.begin());
  t.done = true;
  if (!ctx->tune_verbose) return true;
  fprintf(stderr, "sma autotune: %s n=%lld b=%lld variant=%d%d%d%d, the rule has V%d ->", sizeof(T) == 8 ? "fp64" : "fp32",
          (long long)op->n, (long long)a.b, (int)HQ, (int)HS, (int)HB, (int)PC, v);
  for (size_t k = 0; k < cfg.size(); ++k)
    fprintf(stderr, " %s%s/V%d/U%d=%.1fus", (int)k == t.fastest ? "*" : "",
            cfg[k].bulk ? "bulk" : cfg[k].flat ? "flat" : "rows", cfg[k].V, cfg[k].gathers, 1e3 * best[k]);
  fprintf(stderr, "\n");
  return true;
}

inline bool aligned(const void *p, int bytes) { return ((uintptr_t)p % bytes) == 0; }

template <typename T, typename Fits>
int widest_vector(Fits fits) {
  int v = 32 / (int)sizeof(T);
  while (v > 1 && !fits(v)) v /= 2;
  return v;
}

// The vector width: the widest that widths, strides and addresses allow, but half of it below 40000
// threads, and less while the step would not give every SM half a CTA (us a step:
// Anderson L = 16, b = 32 FP64, 32768 threads 2.6, 65536 2.4; L = 20, b = 64 FP32, 64000 threads
// 2.9, 128000 3.2; XXZ L = 14, b = 32 FP64, 27456 threads 3.1, 54912 2.8).
inline int vector_width(const sma_op *op, int64_t b, int widest) {
  for (int v = widest; v > 1; v /= 2)
    if (op->n * (b / v) >= (v == widest ? 40000 : 64LL * op->ctx->num_sms)) return v;
  return 1;
}

// Where widths, strides or addresses allow accesses of one element only (odd widths in the
// allocation-free entry, below the degree that a padded copy pays for, and where that does not fit), a
// thread takes four columns of a row all the same, a row's threads apart: the row's pointers, columns
// and values serve four, and four times the gathers are in flight.  Us of three steps, one column a
// thread and four: 1D Laplacian n = 400000, b = 31 FP64 410 and 216, FP32 351 and 160; b = 3 48 and
// 34; Anderson L = 80, b = 15 324 and 254.  Not below 48000 threads (Anderson L = 20, b = 17, 40000:
// 22.5 and 24.6; b = 25, 56000: 25.4 and 24.8), for ragged rows not below 8 threads a row (XXZ L = 18,
// b = 15 48 and 57; b = 31 72 and 64), for a model's rows of one thread only in large operators
// (Anderson L = 37, b = 3 32.1 and 33.6; L = 50 45.3 and 43.6).
inline bool strided(const sma_op *op, int64_t b, int widest) {
  const int64_t vecs = (b + 3) / 4;
  return widest == 1 && op->kind != OP_XXZ && b >= 3 && op->n * vecs >= 48000 && (!ragged(op) || vecs >= 8) &&
         (vecs > 1 || op->kind == OP_CSR || op->n >= 100000);
}

template <typename T, bool HQ, bool HS, bool HB, bool PC, int MODEL, Form P = INNER>
void step(const sma_op *op, cudaStream_t st, int64_t b, Step<T> a) {
  if (op->n == 0 || b == 0) return;
  require(b < (int64_t)1 << 31, SMA_ERR_ARG, "block too wide");
  if constexpr (MODEL != STORED) {
    a.model = op->stencil;
    a.kind = op->kind;
    if (op->kind == OP_LAP1D) a.model.hop = -1.0;
    a.entries = op->kind == OP_LAP1D ? 3 : op->kind == OP_ANDERSON ? 7 : (uint32_t)op->stencil.L + 1;
  } else {
    if constexpr (sizeof(T) == 8) a.val = op->val64;
    else a.val = op->val32;
    a.rowptr = op->rowptr;
    a.colind = op->colind;
  }
  a.n = (uint32_t)op->n;
  a.b = (uint32_t)b;
  auto fits = [&](int v) {
    const int bytes = v * (int)sizeof(T);
    return b % v == 0 && a.ldb % bytes == 0 && a.ldo % bytes == 0 && aligned(a.B1, bytes) &&
           aligned(a.out, bytes) && (!HQ || (a.ldq % bytes == 0 && aligned(a.Q, bytes))) &&
           (!HB || P == SECOND || aligned(a.B2, bytes)) &&
           (!PC || a.colseg || (aligned(a.cseg, bytes) && (P == INNER || aligned(a.topseg, bytes))));
  };
  if (a.ldb >> 32) return launch_width<T, 1, HQ, HS, HB, PC, true, MODEL, P>(op, st, a);
  const int widest = widest_vector<T>(fits), v = vector_width(op, b, widest);
  if constexpr (P != DOTS)
    if (strided(op, b, widest)) return launch_width<T, 4, HQ, HS, HB, PC, false, MODEL, P, true>(op, st, a);
  if constexpr (MODEL == STORED && P == INNER)
    if (tuned_step<T, HQ, HS, HB, PC>(op, st, a, widest, v)) return;
  if constexpr (sizeof(T) == 4)
    if (v == 8) return launch_width<T, 8, HQ, HS, HB, PC, false, MODEL, P>(op, st, a);
  if (v == 4) return launch_width<T, 4, HQ, HS, HB, PC, false, MODEL, P>(op, st, a);
  if (v == 2) return launch_width<T, 2, HQ, HS, HB, PC, false, MODEL, P>(op, st, a);
  launch_width<T, 1, HQ, HS, HB, PC, false, MODEL, P>(op, st, a);
}

}  // namespace rows

template <typename T>
rows::Step<T> clenshaw_arguments(const T *Q, int64_t ldq, const T *B1, const T *B2, int64_t ldb, T *out,
                                 int64_t ldo, double alpha, double beta, bool rev, bool tune = true) {
  rows::Step<T> a{};
  a.Q = Q;
  a.B1 = B1;
  a.B2 = B2;
  a.out = out;
  a.ldq = (uint64_t)ldq * sizeof(T);
  a.ldb = (uint64_t)ldb * sizeof(T);
  a.ldo = (uint64_t)ldo * sizeof(T);
  a.alpha = (T)alpha;
  a.beta = (T)beta;
  a.rev = rev;
  a.tune = tune;
  return a;
}

template <typename T, int MODEL>
void clenshaw_step(const sma_op *op, cudaStream_t st, int64_t b, const T *Q, int64_t ldq,
                   const T *B1, const T *B2, int64_t ldb, T *out, int64_t ldo, double ck,
                   double alpha, double beta, bool has_self, bool rev, bool tune = false) {
  rows::Step<T> a = clenshaw_arguments<T>(Q, ldq, B1, B2, ldb, out, ldo, alpha, beta, rev, tune);
  a.ck = (T)ck;
  if (Q && has_self && B2) return rows::step<T, true, true, true, false, MODEL>(op, st, b, a);
  if (Q && has_self && !B2) return rows::step<T, true, true, false, false, MODEL>(op, st, b, a);
  if (!Q && !has_self && !B2) return rows::step<T, false, false, false, false, MODEL>(op, st, b, a);
  throw Error(SMA_ERR_INTERNAL, "unsupported Clenshaw step variant");
}

// The first step of a recurrence (B1 null: it is c_top Q) and the second (B2 is c_top Q).
template <typename T, int MODEL>
void clenshaw_start(const sma_op *op, cudaStream_t st, int64_t b, const T *Q, int64_t ldq, const T *B1,
                    int64_t ldb, T *out, int64_t ldo, double top, double ck, double alpha, double beta,
                    bool rev) {
  rows::Step<T> a = clenshaw_arguments<T>(Q, ldq, B1 ? B1 : Q, nullptr, B1 ? ldb : ldq, out, ldo, alpha,
                                          beta, rev);
  a.ck = (T)ck;
  a.top = (T)top;
  if (B1) rows::step<T, true, true, true, false, MODEL, rows::SECOND>(op, st, b, a);
  else rows::step<T, true, true, false, false, MODEL, rows::FIRST>(op, st, b, a);
}

// The segmented step: column c takes the coefficient cseg[colseg[c]], colseg nondecreasing, or
// cseg[c] when colseg is null; Q, B1 and B2 are all read.
template <typename T, int MODEL>
void clenshaw_step_seg(const sma_op *op, cudaStream_t st, int64_t b, const T *Q, int64_t ldq, const T *B1,
                       const T *B2, int64_t ldb, T *out, int64_t ldo, const T *cseg, const int *colseg,
                       double alpha, double beta, bool rev) {
  rows::Step<T> a = clenshaw_arguments<T>(Q, ldq, B1, B2, ldb, out, ldo, alpha, beta, rev);
  a.cseg = cseg;
  a.colseg = colseg;
  rows::step<T, true, true, true, true, MODEL>(op, st, b, a);
}

// Its first step (B1 null) and second, topseg the highest coefficients.
template <typename T, int MODEL>
void clenshaw_start_seg(const sma_op *op, cudaStream_t st, int64_t b, const T *Q, int64_t ldq, const T *B1,
                        int64_t ldb, T *out, int64_t ldo, const T *topseg, const T *cseg, const int *colseg,
                        double alpha, double beta, bool rev) {
  rows::Step<T> a = clenshaw_arguments<T>(Q, ldq, B1 ? B1 : Q, nullptr, B1 ? ldb : ldq, out, ldo, alpha,
                                          beta, rev);
  a.topseg = topseg;
  a.cseg = cseg;
  a.colseg = colseg;
  if (B1) rows::step<T, true, true, true, true, MODEL, rows::SECOND>(op, st, b, a);
  else rows::step<T, true, true, false, true, MODEL, rows::FIRST>(op, st, b, a);
}

// out = ck Q + alpha A B1 + beta B1, with the sums of a DOTS step (n x b blocks, ld = b).
template <int MODEL>
void clenshaw_dots(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, const double *B1,
                   double *out, double ck, double alpha, double beta, bool rev, int64_t cols,
                   double *dots, int64_t plane) {
  rows::Step<double> a = clenshaw_arguments<double>(Q, b, B1, nullptr, b, out, b, alpha, beta, rev);
  a.ck = ck;
  a.dots = dots;
  a.plane = (uint64_t)plane;
  a.dotcols = (uint32_t)cols;
  rows::step<double, true, true, false, false, MODEL, rows::DOTS>(op, st, b, a);
}

}  // namespace sma
