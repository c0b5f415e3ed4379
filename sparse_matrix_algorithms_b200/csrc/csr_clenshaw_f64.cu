// FP64 Clenshaw steps of CSR matrices (clenshaw_step.cuh).
#include "clenshaw_step.cuh"

namespace sma {

template <>
void csr_clenshaw_step<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                               const double *B1, const double *B2, int64_t ldb, double *out,
                               int64_t ldo, double ck, double alpha, double beta, bool has_self,
                               bool rev) {
  clenshaw_step<double, false>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev);
}

// The segmented step: column c takes the coefficient cseg[colseg[c]], colseg nondecreasing, or
// cseg[c] when colseg is null; Q, B1 and B2 are all read.
template <>
void csr_clenshaw_step_seg<double>(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, int64_t ldq,
                           const double *B1, const double *B2, int64_t ldb, double *out, int64_t ldo,
                           const double *cseg, const int *colseg, double alpha, double beta, bool rev) {
  rows::Step<double> a{};
  a.Q = Q;
  a.B1 = B1;
  a.B2 = B2;
  a.out = out;
  a.cseg = cseg;
  a.colseg = colseg;
  a.ldq = (uint64_t)ldq * sizeof(double);
  a.ldb = (uint64_t)ldb * sizeof(double);
  a.ldo = (uint64_t)ldo * sizeof(double);
  a.alpha = (double)alpha;
  a.beta = (double)beta;
  a.rev = rev;
  rows::step<double, true, true, true, true, false>(op, st, b, a);
}

}  // namespace sma
