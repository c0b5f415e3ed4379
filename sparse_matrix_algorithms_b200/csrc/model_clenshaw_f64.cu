// FP64 Clenshaw steps of the matrix-free models (clenshaw_step.cuh).
#include "clenshaw_step.cuh"

namespace sma {

template <>
void model_clenshaw_step<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q,
                                 int64_t ldq, const double *B1, const double *B2, int64_t ldb,
                                 double *out, int64_t ldo, double ck, double alpha, double beta,
                                 bool has_self, bool rev) {
  clenshaw_step<double, true>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev);
}

template <>
void model_clenshaw_start<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q,
                                  int64_t ldq, const double *B1, int64_t ldb, double *out, int64_t ldo,
                                  double top, double ck, double alpha, double beta, bool rev) {
  clenshaw_start<double, true>(op, st, b, Q, ldq, B1, ldb, out, ldo, top, ck, alpha, beta, rev);
}

template <>
void model_clenshaw_step_seg<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                           const double *B1, const double *B2, int64_t ldb, double *out, int64_t ldo,
                           const double *cseg, const int *colseg, double alpha, double beta, bool rev) {
  clenshaw_step_seg<double, true>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, cseg, colseg, alpha, beta, rev);
}

template <>
void model_clenshaw_start_seg<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                            const double *B1, int64_t ldb, double *out, int64_t ldo, const double *topseg,
                            const double *cseg, const int *colseg, double alpha, double beta, bool rev) {
  clenshaw_start_seg<double, true>(op, st, b, Q, ldq, B1, ldb, out, ldo, topseg, cseg, colseg, alpha, beta, rev);
}

void model_clenshaw_dots(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, const double *B1,
                         double *out, double ck, double alpha, double beta, bool rev, int64_t cols,
                         double *dots, int64_t plane) {
  clenshaw_dots<true>(op, st, b, Q, B1, out, ck, alpha, beta, rev, cols, dots, plane);
}

}  // namespace sma
