// FP32 Clenshaw steps of CSR matrices (clenshaw_step.cuh).
#include "clenshaw_step.cuh"

namespace sma {

template <>
void csr_clenshaw_step<float>(const sma_op *op, cudaStream_t st, int64_t b, const float *Q, int64_t ldq,
                               const float *B1, const float *B2, int64_t ldb, float *out,
                               int64_t ldo, double ck, double alpha, double beta, bool has_self,
                               bool rev, bool tune) {
  clenshaw_step<float, false>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev, tune);
}

template <>
void csr_clenshaw_start<float>(const sma_op *op, cudaStream_t st, int64_t b, const float *Q, int64_t ldq,
                                const float *B1, int64_t ldb, float *out, int64_t ldo, double top,
                                double ck, double alpha, double beta, bool rev) {
  clenshaw_start<float, false>(op, st, b, Q, ldq, B1, ldb, out, ldo, top, ck, alpha, beta, rev);
}

template <>
void csr_clenshaw_step_seg<float>(const sma_op *op, cudaStream_t st, int64_t b, const float *Q, int64_t ldq,
                           const float *B1, const float *B2, int64_t ldb, float *out, int64_t ldo,
                           const float *cseg, const int *colseg, double alpha, double beta, bool rev) {
  clenshaw_step_seg<float, false>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, cseg, colseg, alpha, beta, rev);
}

template <>
void csr_clenshaw_start_seg<float>(const sma_op *op, cudaStream_t st, int64_t b, const float *Q, int64_t ldq,
                            const float *B1, int64_t ldb, float *out, int64_t ldo, const float *topseg,
                            const float *cseg, const int *colseg, double alpha, double beta, bool rev) {
  clenshaw_start_seg<float, false>(op, st, b, Q, ldq, B1, ldb, out, ldo, topseg, cseg, colseg, alpha, beta, rev);
}

}  // namespace sma
