// FP32 Clenshaw steps of CSR matrices (clenshaw_step.cuh).
#include "clenshaw_step.cuh"

namespace sma {

template <>
void csr_clenshaw_step<float>(const sma_op *op, cudaStream_t st, int64_t b, const float *Q, int64_t ldq,
                               const float *B1, const float *B2, int64_t ldb, float *out,
                               int64_t ldo, double ck, double alpha, double beta, bool has_self,
                               bool rev) {
  clenshaw_step<float, false>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev);
}

// The segmented step: column c takes the coefficient cseg[colseg[c]], colseg nondecreasing, or
// cseg[c] when colseg is null; Q, B1 and B2 are all read.
template <>
void csr_clenshaw_step_seg<float>(const sma_op *op, cudaStream_t st, int64_t b, const float *Q, int64_t ldq,
                           const float *B1, const float *B2, int64_t ldb, float *out, int64_t ldo,
                           const float *cseg, const int *colseg, double alpha, double beta, bool rev) {
  rows::Step<float> a{};
  a.Q = Q;
  a.B1 = B1;
  a.B2 = B2;
  a.out = out;
  a.cseg = cseg;
  a.colseg = colseg;
  a.ldq = (uint64_t)ldq * sizeof(float);
  a.ldb = (uint64_t)ldb * sizeof(float);
  a.ldo = (uint64_t)ldo * sizeof(float);
  a.alpha = (float)alpha;
  a.beta = (float)beta;
  a.rev = rev;
  rows::step<float, true, true, true, true, false>(op, st, b, a);
}

}  // namespace sma
