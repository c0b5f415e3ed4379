// FP64 Clenshaw steps of CSR matrices (clenshaw_step.cuh).
#include "clenshaw_step.cuh"

namespace sma {

template <>
void csr_clenshaw_step<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                               const double *B1, const double *B2, int64_t ldb, double *out,
                               int64_t ldo, double ck, double alpha, double beta, bool has_self,
                               bool rev, bool tune) {
  clenshaw_step<double, false>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev, tune);
}

template <>
void csr_clenshaw_start<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                                const double *B1, int64_t ldb, double *out, int64_t ldo, double top,
                                double ck, double alpha, double beta, bool rev) {
  clenshaw_start<double, false>(op, st, b, Q, ldq, B1, ldb, out, ldo, top, ck, alpha, beta, rev);
}

template <>
void csr_clenshaw_step_seg<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                           const double *B1, const double *B2, int64_t ldb, double *out, int64_t ldo,
                           const double *cseg, const int *colseg, double alpha, double beta, bool rev) {
  clenshaw_step_seg<double, false>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, cseg, colseg, alpha, beta, rev);
}

template <>
void csr_clenshaw_start_seg<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                            const double *B1, int64_t ldb, double *out, int64_t ldo, const double *topseg,
                            const double *cseg, const int *colseg, double alpha, double beta, bool rev) {
  clenshaw_start_seg<double, false>(op, st, b, Q, ldq, B1, ldb, out, ldo, topseg, cseg, colseg, alpha, beta, rev);
}

void csr_clenshaw_dots(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, const double *B1,
                       double *out, double ck, double alpha, double beta, bool rev, int64_t cols,
                       double *dots, int64_t plane) {
  clenshaw_dots<false>(op, st, b, Q, B1, out, ck, alpha, beta, rev, cols, dots, plane);
}

// The CTAs of a DOTS step, 0 where a pass of its own is as good: a CTA's sums are 2 / rows of a
// block, written once and read once, against the two blocks of the pass.
int64_t clenshaw_dot_chunks(const sma_op *op, int64_t b) {
  if (op->kind == OP_MATBLOCK || op->kind == OP_CSR_HALF) return 0;
  const int v = rows::vector_width(op, b, rows::widest_vector<double>([&](int w) { return b % w == 0; }));
  const int64_t rows = rows::kThreads / (b / v);
  return b / v <= 16 ? (op->n + rows - 1) / rows : 0;
}

}  // namespace sma
