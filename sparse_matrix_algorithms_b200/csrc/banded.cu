// Many Clenshaw steps in one launch, for operators whose rows hold a full narrow band: entry
// (i, j) for every |i - j| <= W, W = 1 or 2, and no other (1D Laplacians and chains).
//
// One step of such a matrix reaches W rows far, so a CTA that holds rows [r - h, r + R + h) of B1,
// B2 and Q takes h / W steps on them before it needs anything from its neighbours; it writes back
// the R rows in the middle, and what it recomputes of the neighbours' rows is 2 h of R + 2 h.  A
// step by itself is a latency of 2.7 us and more (launch, two dependent reads, drain), or four
// passes over blocks that no cache holds; here neither is paid more than once in 8 to 32 steps.
//
// A thread owns S consecutive rows of one column: their elements of B1, B2 and Q and their matrix
// entries stay in registers, rows of the neighbour threads come through shared memory (the first
// and last W rows of every strip, double buffered: one barrier a step).  What is left is FP32 or
// FP64 arithmetic, 2 W + 7 operations an element.  Measured on one B200, us a step with the step
// kernel and here, tridiagonal:
//   n = 20000   FP32 b = 32 2.75 and 0.57, b = 160 6.6 and 2.2; FP64 b = 64 5.7 and 1.4
//   n = 1000    FP64 b = 8 2.26 and 0.36
//   n = 10^6    FP32 b = 64 149 and 42; FP64 b = 64 305 and 59
// and pentadiagonal n = 20000 FP64 b = 64 6.8 and 3.4: it was the faster of the two at every size.
//
// Accumulation order, rounding and epilogue are the step kernel's (clenshaw_step.cuh): the same
// bits.  Rows outside the matrix are zero rows with zero entries.
#include <algorithm>
#include <cmath>

#include "sma_internal.h"
#include "vec.cuh"

namespace sma {
namespace banded {

constexpr int kMaxThreads = 256;
constexpr int kMaxSteps = 32;
constexpr int kColumns = 8;  // columns of a CTA: 32-byte pieces of FP32 rows, 64 of FP64

template <typename T>
struct Args {
  const int *rowptr;
  const T *val;  // null: tridiag(-1, 2, -1)
  const T *Q, *B1, *B2;  // B1 null: B1 = top Q, B2 = 0
  T *out, *prev;         // the newest block, and the one before it (null: not wanted)
  int64_t ldq, ldb, ldo, n;
  int b, columns, rows, halo, steps;  // rows: written by a CTA
  bool last;  // the last of the steps is the recurrence's
  T alpha, beta, alpha_last, beta_last;
  T top, coef[kMaxSteps];
  const T *topcol, *coefcol;  // PC: the coefficients of step i are coefcol[-i b ...]
};

template <typename T, int W, int S, bool PC>
__global__ void __launch_bounds__(kMaxThreads) kernel(const __grid_constant__ Args<T> a) {
  __shared__ T edge[2][2 * W][kMaxThreads];  // per strip its first W rows, then its last W
  const int tid = threadIdx.x, strip = tid / a.columns, lane = tid - strip * a.columns;
  const bool below = tid >= a.columns, above = tid + a.columns < (int)blockDim.x;
  const int64_t out0 = (int64_t)blockIdx.x * a.rows, r0 = out0 - a.halo + (int64_t)strip * S;
  T v[S][2 * W + 1];
  if (r0 >= W && r0 + S <= a.n - W) {
    const T *p = a.val ? a.val + __ldg(a.rowptr + r0) : nullptr;
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int j = 0; j < 2 * W + 1; ++j)
        v[s][j] = p ? __ldg(p + s * (2 * W + 1) + j) : j == W ? T(2) : T(-1);
  } else {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const int64_t row = r0 + s;
      const bool in = row >= 0 && row < a.n;
      const int64_t first = in && a.val ? __ldg(a.rowptr + row) - max(row - W, (int64_t)0) : 0;
#pragma unroll
      for (int j = 0; j < 2 * W + 1; ++j) {
        const int64_t col = row + j - W;
        const bool there = in && col >= 0 && col < a.n;
        v[s][j] = !there ? T(0) : a.val ? __ldg(a.val + first + col) : j == W ? T(2) : T(-1);
      }
    }
  }
  pdl_wait_then_trigger();
  // every address in the blocks has c in it: none of their loads, which the compiler may take for
  // loads of constants, can move above the wait for the launch that wrote them
  const int64_t c = after_wait((int64_t)blockIdx.y * a.columns + lane);
  // most threads own rows that are all there, with all entries: nothing of theirs is predicated
  const bool whole = r0 >= 0 && r0 + S <= a.n && c < a.b;
  auto read = [&](const T *block, int64_t ld, T (&to)[S]) {
    const T *p = block + r0 * ld + c;
    if (whole) {
#pragma unroll
      for (int s = 0; s < S; ++s, p += ld) to[s] = __ldcg(p);
    } else {
#pragma unroll
      for (int s = 0; s < S; ++s, p += ld) {
        const bool in = r0 + s >= 0 && r0 + s < a.n && c < a.b;
        to[s] = in ? __ldcg(p) : T(0);
      }
    }
  };
  T q[S], x[S], y[S];
  read(a.Q, a.ldq, q);
  if (a.B1) {
    read(a.B1, a.ldb, x);
    read(a.B2, a.ldb, y);
  } else {
    T top = a.top;
    if constexpr (PC) top = c < a.b ? __ldcg(a.topcol + c) : T(0);
#pragma unroll
    for (int s = 0; s < S; ++s) {
      x[s] = mul_rn(top, q[s]);
      y[s] = T(0);
    }
  }
  auto coefficient = [&](int i) {
    if constexpr (!PC) return a.coef[i];
    else return c < a.b ? __ldcg(a.coefcol - (int64_t)i * a.b + c) : T(0);
  };
  T next = coefficient(0);
  // b2 <- ck q + alpha A b1 + beta b1 - b2
  auto step = [&](int i, const T (&b1)[S], T (&b2)[S]) {
    const T ck = next;
    if (i + 1 < a.steps) next = coefficient(i + 1);
    const bool fin = a.last && i == a.steps - 1;
    const T alpha = fin ? a.alpha_last : a.alpha, beta = fin ? a.beta_last : a.beta;
    T(&e)[2 * W][kMaxThreads] = edge[i & 1];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      e[k][tid] = b1[k];
      e[W + k][tid] = b1[S - W + k];
    }
    __syncthreads();
    T up[W], down[W];
#pragma unroll
    for (int k = 0; k < W; ++k) {
      up[k] = below ? e[W + k][tid - a.columns] : T(0);
      down[k] = above ? e[k][tid + a.columns] : T(0);
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
      T acc = T(0);
#pragma unroll
      for (int j = 0; j < 2 * W + 1; ++j) {
        const int t = s + j - W;
        acc = fma(v[s][j], t < 0 ? up[W + t] : t >= S ? down[t - S] : b1[t], acc);
      }
      b2[s] = clenshaw_combine<true, true, true>(acc, q[s], b1[s], b2[s], ck, alpha, beta);
    }
  };
  for (int i = 0; i < a.steps; i += 2) {
    step(i, x, y);
    if (i + 1 < a.steps) step(i + 1, y, x);
  }
  if (a.steps & 1) {  // the newest is y
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const T t = x[s];
      x[s] = y[s];
      y[s] = t;
    }
  }
  auto write = [&](T *block, int64_t ld, const T (&from)[S]) {
    T *p = block + r0 * ld + c;
    if (whole && r0 >= out0 && r0 + S <= out0 + a.rows) {
#pragma unroll
      for (int s = 0; s < S; ++s, p += ld) *p = from[s];
    } else {
#pragma unroll
      for (int s = 0; s < S; ++s, p += ld)
        if (c < a.b && r0 + s >= out0 && r0 + s < out0 + a.rows && r0 + s < a.n) *p = from[s];
    }
  };
  write(a.out, a.ldo, x);
  if (a.prev) write(a.prev, a.ldo, y);
}

// How a filter is cut: CTAs of `strips` strips over `rows` rows and `columns` columns, `steps`
// steps a launch.
struct Plan {
  int columns, strips, rows, steps;
};

// The cheapest by a model of the time of a step, in cycles: the SM with the most CTAs works its
// strips off (2 W + 10 operations an element at 128 FP32 or 64 FP64 lanes), a barrier and the
// latency of a step come on top, and a launch with its reads and writes is shared by its steps.
Plan plan(int64_t n, int64_t b, int64_t K, int band, int strip_rows, int elem_bytes, int num_sms) {
  Plan best{};
  const int64_t groups = (b + kColumns - 1) / kColumns;
  const int columns = (int)((b + groups - 1) / groups);
  const int lanes = elem_bytes == 8 ? 64 : 128;
  double cost = INFINITY;
  for (int steps = 8; steps <= kMaxSteps; steps *= 2) {
    const int t = (int)std::min<int64_t>(steps, K);
    for (int strips = 1; strips * columns <= kMaxThreads; ++strips) {
      const int rows = strips * strip_rows - 2 * t * band;
      if (rows <= 0) continue;
      const int64_t ctas = (n + rows - 1) / rows * groups, waves = (ctas + num_sms - 1) / num_sms;
      const double strip = (double)strip_rows * columns * (2 * band + 10) / lanes;
      const double c = waves * strips * strip * (1.0 + 2.0 / t) + 120.0 + 6000.0 / t;
      if (c < cost) {
        cost = c;
        best = {columns, strips, rows, t};
      }
    }
  }
  return best;
}

}  // namespace banded

namespace {

// S: a row takes three elements and 2 W + 1 entries in registers.  Eight rows; FP64 with five
// entries takes half (n = 10^5, b = 160: 4 rows 39.6 us a step, 8 rows 45.4; with three entries 23.4
// and 15.5), FP32 gains nothing for sure from twice (n = 10^6, b = 8 5.5 and 4.3, b = 32 19.8 and 21.9).
constexpr int strip_rows(int elem_bytes, int band) { return elem_bytes == 8 && band > 1 ? 4 : 8; }

template <typename T, int W, bool PC>
void launch(const sma_op *op, cudaStream_t st, const banded::Args<T> &a, const banded::Plan &p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((a.n + p.rows - 1) / p.rows), (unsigned)((a.b + p.columns - 1) / p.columns));
  cfg.blockDim = dim3((unsigned)(p.strips * p.columns));
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = op->ctx->pdl ? 1 : 0;
  SMA_CUDA(cudaLaunchKernelEx(&cfg, banded::kernel<T, W, strip_rows(sizeof(T), W), PC>, a));
  SMA_CHECK_LAUNCH();
}

}  // namespace

// W of an operator of this form, else 0.
int banded_width(int64_t n, const std::vector<int> &rowptr, const std::vector<int> &cols) {
  const int64_t w = n > 0 ? rowptr[1] - rowptr[0] - 1 : 0;
  if (w < 1 || w > 2 || n <= 2 * w) return 0;
  for (int64_t i = 0; i < n; ++i) {
    const int64_t lo = std::max<int64_t>(0, i - w), hi = std::min<int64_t>(n - 1, i + w);
    if (rowptr[i + 1] - rowptr[i] != hi - lo + 1) return 0;
    for (int64_t j = lo; j <= hi; ++j)
      if (cols[rowptr[i] + (j - lo)] != j) return 0;
  }
  return (int)w;
}

// Not in place: the last launch would write rows of Q that other CTAs still read.
template <typename T>
bool banded_fits(const sma_op *op, int64_t K, const T *Q, int64_t ldq, const T *Y, int64_t ldy, int64_t b) {
  const uintptr_t q = (uintptr_t)Q, y = (uintptr_t)Y;
  const uintptr_t q_end = q + ((op->n - 1) * ldq + b) * sizeof(T), y_end = y + ((op->n - 1) * ldy + b) * sizeof(T);
  return op->band > 0 && K >= 2 && b <= 65535LL * banded::kColumns && (q_end <= y || y_end <= q);
}

template <typename T>
FilterCount banded_filter(const sma_op *op, cudaStream_t st, const std::vector<double> *coeffs,
                          const T *table, int64_t K, double smin, double smax, const T *Q, int64_t ldq,
                          T *Y, int64_t ldy, int64_t b, T *const buf[4]) {
  const double c = 0.5 * (smin + smax), invd = 2.0 / (smax - smin);
  banded::Args<T> a{};
  a.n = op->n;
  a.b = (int)b;
  if (op->kind == OP_CSR) {
    a.rowptr = op->rowptr;
    if constexpr (sizeof(T) == 8) a.val = op->val64;
    else a.val = op->val32;
  }
  a.Q = Q;
  a.ldq = ldq;
  a.ldb = b;
  a.alpha = (T)(2.0 * invd);
  a.beta = (T)(-2.0 * c * invd);
  a.alpha_last = (T)invd;
  a.beta_last = (T)(-(c * invd));
  if (table) a.topcol = table + K * b;
  else a.top = (T)(*coeffs)[K];
  const banded::Plan p = banded::plan(op->n, b, K, op->band, strip_rows(sizeof(T), op->band), sizeof(T),
                                      op->ctx->num_sms);
  a.columns = p.columns;
  a.rows = p.rows;
  a.halo = p.steps * op->band;
  FilterCount fc;
  const double blk = (double)op->n * (double)b * sizeof(T), mat = clenshaw_step_bytes(op, 0, sizeof(T));
  int at = 0;
  for (int64_t k = K - 1; k >= 0; k -= a.steps, at ^= 2) {
    a.steps = (int)std::min<int64_t>(p.steps, k + 1);
    a.last = k + 1 == a.steps;
    a.out = a.last ? Y : buf[at];
    a.prev = a.last ? nullptr : buf[at + 1];
    a.ldo = a.last ? ldy : b;
    if (table) a.coefcol = table + k * b;
    else
      for (int i = 0; i < a.steps; ++i) a.coef[i] = (T)(*coeffs)[k - i];
    if (op->band == 1) {
      if (table) launch<T, 1, true>(op, st, a, p);
      else launch<T, 1, false>(op, st, a, p);
    } else {
      if (table) launch<T, 2, true>(op, st, a, p);
      else launch<T, 2, false>(op, st, a, p);
    }
    fc.steps += a.steps;
    fc.bytes += mat + (1 + (a.B1 ? 2 : 0) + (a.last ? 1 : 2)) * blk;
    a.B1 = buf[at];
    a.B2 = buf[at + 1];
  }
  return fc;
}

template bool banded_fits<double>(const sma_op *, int64_t, const double *, int64_t, const double *, int64_t, int64_t);
template bool banded_fits<float>(const sma_op *, int64_t, const float *, int64_t, const float *, int64_t, int64_t);
template FilterCount banded_filter<double>(const sma_op *, cudaStream_t, const std::vector<double> *,
                                           const double *, int64_t, double, double, const double *, int64_t,
                                           double *, int64_t, int64_t, double *const[4]);
template FilterCount banded_filter<float>(const sma_op *, cudaStream_t, const std::vector<double> *,
                                          const float *, int64_t, double, double, const float *, int64_t,
                                          float *, int64_t, int64_t, float *const[4]);

}  // namespace sma
