// Block Clenshaw filter Y = p(A_hat) Q (apply_poly_block!,
// chebyshev_subspace_iteration.jl:554-635, polfed.jl:464-545).
//
//   B_{K+1} = B_{K+2} = 0
//   B_k = c_k Q + 2 A_hat B_{k+1} - B_{k+2}       (k = K..1)
//   Y   = c_0 Q + A_hat B_1 - B_2,    A_hat = (A - cI)/d
//
// evaluated as the reference does: B_k = c_k Q + alpha*A B_{k+1} + beta*B_{k+1} - B_{k+2}
// with invd = 2/(smax-smin), alpha = 2*invd, beta = -2*c*invd
// (chebyshev_subspace_iteration.jl:562-565).
//
// The reference zero-fills B1 and B2 and runs K+1 sparse products.  The first step
// multiplies zeros and gives B1 = c_K Q (bit-identical: every dropped term is an exact
// zero), which the next two steps form from Q themselves.  Each step is ONE fused kernel
// launch (clenshaw_step.cuh) for device operators, for full narrow bands many steps are one
// (banded.cu); caller-supplied operators get the product from their callback followed by the
// axpy kernel, and a scaled block to start from.
#include "sma_internal.h"

namespace sma {

template <typename T>
void ClenshawWork<T>::ensure(const sma_op *op, int64_t n_, int64_t b, cudaStream_t st) {
  if (n_ == n && b <= bcap && b1.p) return;
  drop_graph();  // the graph holds the old buffers' addresses
  n = n_;
  bcap = b;
  b1.alloc(n * b, st);
  b2.alloc(n * b, st);
  tmp.alloc(n * b, st);
  q.release();
  y.release();
  b3.release();
  if (op->kind == OP_MATBLOCK || op->kind == OP_CSR_HALF) ax.alloc(n * b, st);
}

template <typename T>
bool ClenshawWork<T>::fits_with(DevBuf<T> &extra, const sma_op *op, int64_t n_, int64_t w,
                                cudaStream_t st) {
  try {
    ensure(op, n_, w, st);
    if (!extra.p) extra.alloc(n * bcap, st);
    return true;
  } catch (const Error &e) {
    if (e.code != SMA_ERR_NOMEM) throw;
    cudaGetLastError();  // the failed allocation is not an error of a later launch
    b1.release();
    b2.release();
    tmp.release();
    q.release();
    b3.release();
    bcap = 0;
    return false;
  }
}

template <typename T>
void ClenshawWork<T>::drop_graph() {
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  exec = nullptr;
  graph = nullptr;
  g_op = nullptr;
  g_b = -1;
  g_calls = 0;
}

// The fused step runs on the widest vectors that divide the width.  An odd width leaves 8- or
// 4-byte accesses, so the recurrence's own blocks (and a staged copy of Q) take the width of
// least cost: columns times the time of a column relative to 32-byte vectors, measured as 1.18
// with 16 bytes (FP32 n = 262144, b = 64: 49 against 42.5 us) and 1.6 with 8 (FP64 n = 27000,
// b = 37: 10.3 us against 6.6 at b = 40); 4-byte accesses are put at 2.5.
int64_t recurrence_width(int64_t b, int elem_bytes) {
  const double cost[4] = {1.0, 1.18, 1.6, 2.5};  // 32, 16, 8 and 4 bytes
  int64_t best = b;
  double least = 0.0;
  for (int k = 0, bytes = 32; bytes >= elem_bytes; bytes /= 2, ++k) {
    const int64_t v = bytes / elem_bytes, w = (b + v - 1) / v * v;
    if (k == 0 || (double)w * cost[k] < least) {
      least = (double)w * cost[k];
      best = w;
    }
  }
  return best;
}

// The same where a copy of Q is its price: not where a thread takes one column anyway (vector_width in
// clenshaw_step.cuh: fewer than half a CTA an SM with two; n = 3000, b = 3, K = 4 27.2 us with the
// copy, 26.1 without).
int64_t staged_width(const sma_op *op, int64_t b, int elem_bytes) {
  return op->n * b < 128LL * op->ctx->num_sms ? b : recurrence_width(b, elem_bytes);
}

double clenshaw_step_bytes(const sma_op *op, int64_t b, int elem_bytes) {
  // nnz*(value + column index) + row pointers + Q, B1, B2 reads and one write
  double mat = 0.0;
  if (op->kind == OP_CSR || op->kind == OP_CSR_HALF)  // half storage: its stored entries
    mat = (double)op->nnz * (elem_bytes + 4) + 4.0 * (op->n + 1);
  return mat + 4.0 * (double)op->n * (double)b * elem_bytes;
}

void check_bulk_error(const sma_op *op, cudaStream_t st) {
  if (!op->bulk_err) return;
  int h = 0;
  SMA_CUDA(cudaMemcpyAsync(&h, op->bulk_err, sizeof(int), cudaMemcpyDeviceToHost, st));
  SMA_CUDA(cudaStreamSynchronize(st));
  if (h != 0) {
    SMA_CUDA(cudaMemsetAsync(op->bulk_err, 0, sizeof(int), st));
    SMA_CUDA(cudaStreamSynchronize(st));
    throw Error(SMA_ERR_TIMEOUT, h == 1 ? "a bulk-copy CSR step gave up waiting for its copies"
                                        : "a bulk-copy CSR step met a CTA larger than its shared memory");
  }
}

void op_apply(const sma_op *op, cudaStream_t st, const double *X, int64_t ldx, double *Y,
              int64_t ldy, int64_t b) {
  if (b == 0 || op->n == 0) return;
  if (op->kind == OP_MATBLOCK) {
    require(ldx == ldy, SMA_ERR_ARG, "matrix-free operator callbacks need equal leading dimensions");
    const int rc = op->fn(op->user, X, Y, op->n, b, ldx, (void *)st);
    if (rc != 0) throw Error(SMA_ERR_CALLBACK, "matblock callback returned " + std::to_string(rc));
    SMA_CUDA(cudaGetLastError());
    return;
  }
  if (op->kind == OP_CSR_HALF) return half_product<double>(op, st, X, ldx, Y, ldy, b);
  launch_clenshaw_step<double>(op, st, b, nullptr, 0, X, nullptr, ldx, Y, ldy, 0.0, 1.0, 0.0, false);
  check_bulk_error(op, st);
}

template <typename T>
static void matblock_apply(const sma_op *op, cudaStream_t st, const T *X, T *AX, int64_t ld,
                           int64_t b) {
  if (op->kind == OP_CSR_HALF) return half_product<T>(op, st, X, ld, AX, ld, b);
  if constexpr (sizeof(T) == 8) {
    const int rc = op->fn(op->user, (const double *)X, (double *)AX, op->n, b, ld, (void *)st);
    if (rc != 0) throw Error(SMA_ERR_CALLBACK, "matblock callback returned " + std::to_string(rc));
  } else {
    throw Error(SMA_ERR_ARG, "caller-supplied operators take FP64 blocks only");
  }
}

// Whether a filter's first two steps form the block c_K Q themselves (record_filter).
static bool folds(const sma_op *op, int64_t K) {
  return op->kind != OP_MATBLOCK && op->kind != OP_CSR_HALF && K >= 2;
}

// Steps and algorithmic bytes of a filter of b columns, whatever width its blocks are padded to: Q,
// B1, B2 read and one block written a step, without B1 and B2 in the first and B2 in the second of a
// folded one, else a scaled block to start from, and no B2 in the first step.
template <typename T>
static FilterCount count_filter(const sma_op *op, int64_t K, int64_t b) {
  FilterCount fc;
  fc.steps = K;
  fc.bytes = (double)K * clenshaw_step_bytes(op, 0, sizeof(T)) +
             (double)(4 * K + (folds(op, K) ? -3 : 1)) * (double)op->n * (double)b * sizeof(T);
  return fc;
}

// The launches of one filter (K >= 1) on recurrence blocks of width w >= b (w = b for operators
// without a fused step; Q is read over w columns but by the last step).
template <typename T>
static void record_filter(const sma_op *op, cudaStream_t st,
                          const std::vector<double> &coeffs, double smin, double smax,
                          const T *Q, int64_t ldq, T *Y, int64_t ldy, int64_t b, int64_t w,
                          ClenshawWork<T> &work) {
  const int64_t n = op->n;
  const int64_t K = (int64_t)coeffs.size() - 1;
  const double c = 0.5 * (smin + smax);
  const double invd = 2.0 / (smax - smin);
  const double alpha = 2.0 * invd;
  const double beta = -2.0 * c * invd;
  const bool fused = op->kind != OP_MATBLOCK && op->kind != OP_CSR_HALF;
  T *B1 = work.b1.p, *B2 = work.b2.p, *TMP = work.tmp.p;
  const int64_t ld = w;
  auto rotate = [&]() {  // B1, B2, TMP = TMP, B1, B2
    T *t = B2;
    B2 = B1;
    B1 = TMP;
    TMP = t;
  };
  // Step K+1 of the reference is B1 = c_K Q (its product multiplies zeros).  With a fused step the
  // next two form it from Q, which they read anyhow: two passes over a block and a launch less
  // (Anderson L = 64: FP32 b = 768, K = 16 10.0 -> 9.56 ms; per-column b = 496, K = 24, whose zero
  // blocks and first product are gone too, 10.57 -> 10.02 ms).  A first step
  // that is also the last could write to the Q that it gathers (Y = Q): it takes the block.
  const bool fold = folds(op, K);
  int64_t ci = K - 1;
  if (fold) {
    launch_clenshaw_start<T>(op, st, w, Q, ldq, nullptr, ld, TMP, ld, coeffs[K], coeffs[ci], alpha, beta,
                             ci & 1);
    B1 = TMP;
    TMP = work.b1.p;
    --ci;
    if (ci >= 1) {
      launch_clenshaw_start<T>(op, st, w, Q, ldq, B1, ld, TMP, ld, coeffs[K], coeffs[ci], alpha, beta, ci & 1);
      rotate();
      --ci;
    }
  } else {
    launch_scale_block<T>(st, n, w, Q, ldq, B1, ld, coeffs[K]);
  }
  bool b2_zero = !fold;
  for (; ci >= 1; --ci) {
    if (fused) {
      launch_clenshaw_step<T>(op, st, w, Q, ldq, B1, B2, ld, TMP, ld, coeffs[ci], alpha, beta, true, ci & 1);
    } else {
      matblock_apply<T>(op, st, B1, work.ax.p, ld, b);
      launch_clenshaw_axpy<T>(st, n, b, Q, ldq, work.ax.p, ld, B1, b2_zero ? nullptr : B2, ld,
                              TMP, ld, coeffs[ci], alpha, beta);
    }
    rotate();
    b2_zero = false;
  }
  // final step: Y = c_0 Q + invd*A B1 - c*invd*B1 - B2
  if (fold && K == 2) {
    launch_clenshaw_start<T>(op, st, b, Q, ldq, B1, ld, Y, ldy, coeffs[K], coeffs[0], invd, -(c * invd));
    b2_zero = true;  // not read
  } else if (fused) {
    launch_clenshaw_step<T>(op, st, b, Q, ldq, B1, b2_zero ? nullptr : B2, ld, Y, ldy, coeffs[0],
                            invd, -(c * invd), true, false);
  } else {
    matblock_apply<T>(op, st, B1, work.ax.p, ld, b);
    launch_clenshaw_axpy<T>(st, n, b, Q, ldq, work.ax.p, ld, B1, b2_zero ? nullptr : B2, ld, Y,
                            ldy, coeffs[0], invd, -(c * invd));
  }
}

// Filters of degree below this run eagerly (launch overhead is then not the question).
constexpr int64_t kGraphMinDegree = 32;
constexpr int64_t kPadMinDegree = 4;

template <typename T>
static FilterCount apply_poly_block_impl(const sma_op *op, cudaStream_t st,
                                         const std::vector<double> &coeffs, double smin,
                                         double smax, const T *Q, int64_t ldq, T *Y, int64_t ldy,
                                         int64_t b, ClenshawWork<T> &work) {
  FilterCount fc;
  const int64_t n = op->n;
  const int64_t K = (int64_t)coeffs.size() - 1;
  require(K >= 0, SMA_ERR_ARG, "empty coefficient vector");
  if (n == 0 || b == 0) return fc;
  if (K == 0) {  // no loop: Y = c_0 Q
    launch_scale_block<T>(st, n, b, Q, ldq, Y, ldy, coeffs[0]);
    fc.bytes += 2.0 * (double)n * (double)b * sizeof(T);
    return fc;
  }
  const bool fused = op->kind != OP_MATBLOCK && op->kind != OP_CSR_HALF;
  const bool persistent = op->kind == OP_CSR && op->ctx->persistent && K >= kGraphMinDegree;
  int64_t w = b;
  bool stage = false;  // run on a copy of Q: half a step's time, for a gain with every step
  if (!persistent && banded_fits(op, K, Q, ldq, Y, ldy, b) && work.fits_with(work.b3, op, n, b, st)) {
    T *const buf[4] = {work.b1.p, work.b2.p, work.tmp.p, work.b3.p};
    return banded_filter<T>(op, st, &coeffs, nullptr, K, smin, smax, Q, ldq, Y, ldy, b, buf);
  }
  if (fused && !persistent && K >= kPadMinDegree) {
    w = staged_width(op, b, sizeof(T));
    int64_t vec = 32;  // the access that w allows
    while ((w * (int64_t)sizeof(T)) % vec) vec /= 2;
    stage = w != b || (ldq * (int64_t)sizeof(T)) % vec || (uintptr_t)Q % vec;
    if (stage && !work.fits(op, n, w, st)) {
      w = b;
      stage = false;
    }
  }
  work.ensure(op, n, w, st);
  if (persistent) {
    if (work.coef.count < (size_t)(K + 1)) work.coef.alloc(K + 1, st);
    if (!work.barrier.p) work.barrier.alloc(3, st);
    return persistent_filter<T>(op, st, coeffs, smin, smax, Q, ldq, Y, ldy, b, work.b1.p,
                                work.b2.p, work.tmp.p, work.coef.p, work.barrier.p);
  }
  fc = count_filter<T>(op, K, b);
  auto eager = [&]() {
    if (stage) {  // zero columns stay zero through the recurrence
      if (!work.q.p) work.q.alloc(n * work.bcap, st);
      launch_pad_block<T, T>(st, n, b, Q, ldq, w, work.q.p, w);
      record_filter<T>(op, st, coeffs, smin, smax, work.q.p, w, Y, ldy, b, w, work);
    } else {
      record_filter<T>(op, st, coeffs, smin, smax, Q, ldq, Y, ldy, b, w, work);
    }
    return fc;
  };
  if (!fused || K < kGraphMinDegree || !op->ctx->filter_graphs) return eager();
  // repeated filter -> CUDA graph on the staging blocks
  const bool same = work.g_op == op && work.g_b == b && work.g_smin == smin &&
                    work.g_smax == smax && work.g_coeffs == coeffs;
  if (!same) {
    work.drop_graph();
    work.g_op = op;
    work.g_b = b;
    work.g_smin = smin;
    work.g_smax = smax;
    work.g_coeffs = coeffs;
  }
  work.g_calls += 1;
  if (work.g_calls == 1) return eager();  // a graph pays from its second use
  try {
    if (!work.q.p) work.q.alloc(n * work.bcap, st);
    if (!work.y.p) work.y.alloc(n * work.bcap, st);
  } catch (const Error &e) {  // no memory for the staging blocks: step by step
    if (e.code != SMA_ERR_NOMEM) throw;
    cudaGetLastError();  // the failed allocation is not an error of a later launch
    return eager();
  }
  launch_pad_block<T, T>(st, n, b, Q, ldq, w, work.q.p, w);
  if (!work.exec) {
    const int64_t l0 = g_kernel_launches.load();
    SMA_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    try {
      record_filter<T>(op, st, coeffs, smin, smax, work.q.p, w, work.y.p, w, w, w, work);
    } catch (...) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(st, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    SMA_CUDA(cudaStreamEndCapture(st, &work.graph));
    SMA_CUDA(cudaGraphInstantiate(&work.exec, work.graph, 0));
    work.g_launches = g_kernel_launches.load() - l0;
    g_kernel_launches.fetch_sub(work.g_launches);  // counted when the graph runs
  }
  SMA_CUDA(cudaGraphLaunch(work.exec, st));
  g_kernel_launches.fetch_add(work.g_launches);
  work.replays += 1;
  launch_copy_block<T, T>(st, n, b, work.y.p, w, Y, ldy);
  return fc;
}

template <typename T>
FilterCount apply_poly_block(const sma_op *op, cudaStream_t st, const std::vector<double> &coeffs,
                             double smin, double smax, const T *Q, int64_t ldq, T *Y, int64_t ldy,
                             int64_t b, ClenshawWork<T> &work) {
  const FilterCount fc = apply_poly_block_impl<T>(op, st, coeffs, smin, smax, Q, ldq, Y, ldy, b, work);
  check_bulk_error(op, st);
  return fc;
}

template struct ClenshawWork<double>;
template struct ClenshawWork<float>;
template FilterCount apply_poly_block<double>(const sma_op *, cudaStream_t,
                                              const std::vector<double> &, double, double,
                                              const double *, int64_t, double *, int64_t, int64_t,
                                              ClenshawWork<double> &);
template FilterCount apply_poly_block<float>(const sma_op *, cudaStream_t,
                                             const std::vector<double> &, double, double,
                                             const float *, int64_t, float *, int64_t, int64_t,
                                             ClenshawWork<float> &);

}  // namespace sma
