// CUDA kernels of libsma (sm_100a).
//
// The hot one, the fused block Clenshaw step
//
//     out[i,:] = ck*Q[i,:] + alpha*sum_j A[i,j]*B1[j,:] + beta*B1[i,:] - B2[i,:],
//
// replaces the reference's `mul!(AX,A,B1)` followed by a separate 4-array axpy sweep
// (chebyshev_subspace_iteration.jl:573-582, polfed.jl:483-492); AX never reaches memory.
// It lives in clenshaw_step.cuh; this file holds its dispatcher and the small kernels around
// the solvers.
#include "ordered_sum.cuh"
#include "sma_internal.h"
#include "vec.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>

namespace sma {

std::atomic<int64_t> g_kernel_launches{0};

namespace {

// ------------------------------------------------------------------ elementwise block ops
// Element t of an n x b block is (t / b, t % b).  I: the index type; 32-bit divisions, where the
// block allows them, are a quarter of the 64-bit ones that made these kernels slower than memory.
template <typename T, typename I>
__global__ void scale_block_kernel(I total, I b, const T *__restrict__ Q, int64_t ldq,
                                   T *__restrict__ out, int64_t ldo, T ck) {
  const I stride = (I)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const I i = (I)t / b, j = (I)t - i * b;
    out[(int64_t)i * ldo + j] = mul_rn(ck, Q[(int64_t)i * ldq + j]);
  }
}

template <typename T, typename I>
__global__ void clenshaw_axpy_kernel(I total, I b, const T *__restrict__ Q, int64_t ldq,
                                     const T *__restrict__ AX, int64_t ldax,
                                     const T *__restrict__ B1, const T *__restrict__ B2,
                                     int64_t ldb, T *__restrict__ out, int64_t ldo, T ck, T alpha,
                                     T beta) {
  const I stride = (I)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const I r = (I)t / b;
    const int64_t i = r, j = (I)t - r * b;
    const T q = Q[i * ldq + j], a = AX[i * ldax + j], s = B1[i * ldb + j];
    out[i * ldo + j] = B2 ? clenshaw_combine<true, true, true>(a, q, s, B2[i * ldb + j], ck, alpha, beta)
                          : clenshaw_combine<true, true, false>(a, q, s, T(0), ck, alpha, beta);
  }
}

// dst (n x w) <- src (n x b), w >= b, the columns past b zero
template <typename TS, typename TD, typename I>
__global__ void copy_block_kernel(I total, I w, I b, const TS *__restrict__ src, int64_t lds,
                                  TD *__restrict__ dst, int64_t ldd) {
  const I stride = (I)gridDim.x * blockDim.x;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += stride) {
    const I i = (I)t / w, j = (I)t - i * w;
    dst[(int64_t)i * ldd + j] = j < b ? (TD)src[(int64_t)i * lds + j] : TD(0);
  }
}

inline int grid_for(int64_t total) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 148LL * 32));
}

// ------------------------------------------------------------------ random start blocks
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}

// Element (i, j) of an n x m standard-normal block: flat index k = i + j*n (Julia's
// column-major randn fill order), uniforms 2k and 2k+1 of the SplitMix64 counter
// stream seed ^ 0x5DEECE66D, Box-Muller z = sqrt(-2 ln(1-u0)) cos(2 pi u1).
__global__ void randn_kernel(int64_t n, int64_t m, uint64_t seed, double *__restrict__ out,
                             int64_t ld) {
  const uint64_t s = seed ^ 0x5DEECE66DULL;
  const uint64_t golden = 0x9E3779B97F4A7C15ULL;
  const int64_t total = n * m;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / m, j = t % m;
    const uint64_t k = (uint64_t)i + (uint64_t)j * (uint64_t)n;
    const uint64_t x0 = mix64(s + (2 * k + 1) * golden);
    const uint64_t x1 = mix64(s + (2 * k + 2) * golden);
    const double u0 = (double)(x0 >> 11) * (1.0 / 9007199254740992.0);
    const double u1 = (double)(x1 >> 11) * (1.0 / 9007199254740992.0);
    out[i * ld + j] = sqrt(-2.0 * log1p(-u0)) * cos(2.0 * 3.141592653589793 * u1);
  }
}

// ------------------------------------------------------------------ column reductions
// mode 0: sum X Y down every column; mode 1: sum (Y - lam X)^2.  The order of the sums is part of
// the result (a mixed-precision solve scales residuals with these norms before it rounds them to
// FP32): a chunk of rows in eight interleaved groups, the groups one after the other, then the chunks.
// Stage 1: the 2^lc threads of a row group sit on consecutive columns, so that narrow blocks use
// every lane; a CTA takes 32 >> lc chunks of up to 32 columns.
__global__ void __launch_bounds__(256)
colred_stage1(int mode, int lc, int64_t n, int64_t k, const double *__restrict__ X, int64_t ldx,
              const double *__restrict__ Y, int64_t ldy, const double *__restrict__ lam,
              double *__restrict__ partial, int64_t chunks, int64_t rows_per_chunk) {
  __shared__ double sh[256];
  const int tid = threadIdx.x, cl = tid & ((1 << lc) - 1), rl = tid >> lc;
  const int64_t col = ((int64_t)blockIdx.y << lc) + cl;
  const int64_t chunk = (int64_t)blockIdx.x * (32 >> lc) + rl / 8;
  const int64_t r0 = chunk * rows_per_chunk, r1 = min(n, r0 + rows_per_chunk);
  double s = 0.0;
  if (col < k && chunk < chunks) {
    const double l = mode == 1 ? lam[col] : 0.0;
#pragma unroll 4
    for (int64_t i = r0 + rl % 8; i < r1; i += 8) {
      const double x = X[i * ldx + col];
      const double y = Y[i * ldy + col];
      if (mode == 0) {
        s = fma(x, y, s);
      } else {
        const double d = fma(-l, x, y);
        s = fma(d, d, s);
      }
    }
  }
  sh[tid] = s;
  __syncthreads();
  if (rl % 8 == 0 && col < k && chunk < chunks) {
    double t = 0.0;
#pragma unroll
    for (int r = 0; r < 8; ++r) t += sh[tid + (r << lc)];
    partial[chunk * k + col] = t;
  }
}

constexpr int kSumLanes = 4;
__global__ void __launch_bounds__(256)
colred_stage2(int mode, int64_t chunks, int64_t k, const double *__restrict__ partial, double *__restrict__ out) {
  __shared__ OrderedSum<kSumLanes, 16> sum;
  const int64_t col = (int64_t)blockIdx.x * kSumLanes + threadIdx.x % kSumLanes;
  const double t = sum(col < k ? partial + col : nullptr, k, chunks);
  if (threadIdx.x < kSumLanes && col < k) out[col] = mode == 1 ? sqrt(t) : t;
}

// The sums of a KPM step, sum X Y and, `plane` further on, sum Y Y from one read of both blocks, whose
// order is free.  Stage 1: a CTA sums one chunk of rows of up to 32 columns; 256 >> lc rows are in
// flight per pass.
__global__ void __launch_bounds__(256)
dots_stage1(int lc, int64_t n, int64_t k, const double *__restrict__ X, int64_t ldx,
            const double *__restrict__ Y, int64_t ldy, double *__restrict__ partial,
            int64_t rows_per_chunk, int64_t plane) {
  __shared__ double sh[2][256];
  const int tid = threadIdx.x, cl = tid & ((1 << lc) - 1), rl = tid >> lc, R = 256 >> lc;
  const int64_t col = ((int64_t)blockIdx.y << lc) + cl;
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_chunk;
  const int64_t r1 = min(n, r0 + rows_per_chunk);
  double s = 0.0, s2 = 0.0;
  if (col < k) {
#pragma unroll 4
    for (int64_t i = r0 + rl; i < r1; i += R) {
      const double x = X[i * ldx + col];
      const double y = Y[i * ldy + col];
      s = fma(x, y, s);
      s2 = fma(y, y, s2);
    }
  }
  sh[0][tid] = s;
  sh[1][tid] = s2;
  for (int h = 128; h >= 1 << lc; h >>= 1) {
    __syncthreads();
    if (tid < h) {
      sh[0][tid] += sh[0][tid + h];
      sh[1][tid] += sh[1][tid + h];
    }
  }
  if (rl == 0 && col < k) {
    partial[(int64_t)blockIdx.x * k + col] = sh[0][tid];
    partial[plane + (int64_t)blockIdx.x * k + col] = sh[1][tid];
  }
}

// Stage 2: out[g k + col] = the sum over the chunks of group g (groups of chunks x k partials one
// after the other), eight row groups of a CTA sharing the chunks: a serial sum of the 1184
// partials of a KPM reduction took 80 of its 90 us.
__global__ void __launch_bounds__(256)
dots_stage2(int64_t chunks, int64_t k, int64_t total, const double *__restrict__ partial,
            double *__restrict__ out) {
  __shared__ double sh[8][33];
  const int cl = threadIdx.x % 32, rl = threadIdx.x / 32;
  const int64_t e = (int64_t)blockIdx.x * 32 + cl;
  double t = 0.0;
  if (e < total) {
    const double *p = partial + (e / k) * chunks * k + e % k;
#pragma unroll 4
    for (int64_t c = rl; c < chunks; c += 8) t += p[c * k];
  }
  sh[rl][cl] = t;
  __syncthreads();
  if (rl == 0 && e < total) {
    t = 0.0;
#pragma unroll
    for (int r = 0; r < 8; ++r) t += sh[r][cl];
    out[e] = t;
  }
}

// ------------------------------------------------------------------ layout helpers
// out (row-major C x R, ldo) = in^T where in is row-major R x C (ldi)
__global__ void transpose_kernel(int64_t R, int64_t C, const double *__restrict__ in, int64_t ldi,
                                 double *__restrict__ out, int64_t ldo) {
  __shared__ double tile[32][33];
  const int64_t r0 = (int64_t)blockIdx.y * 32, c0 = (int64_t)blockIdx.x * 32;
  for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
    const int64_t r = r0 + dy, c = c0 + threadIdx.x;
    if (r < R && c < C) tile[dy][threadIdx.x] = in[r * ldi + c];
  }
  __syncthreads();
  for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
    const int64_t c = c0 + dy, r = r0 + threadIdx.x;
    if (r < R && c < C) out[c * ldo + r] = tile[threadIdx.x][dy];
  }
}

__global__ void symmetrize_kernel(int64_t k, const double *__restrict__ G, int64_t ldg,
                                  double *__restrict__ H, int64_t ldh) {
  const int64_t total = k * k;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % k, j = t / k;
    H[i + j * ldh] = 0.5 * (G[i + j * ldg] + G[j + i * ldg]);
  }
}

__global__ void place_blocks_kernel(double *__restrict__ T, int64_t ldt, int64_t o, int64_t r,
                                    const double *__restrict__ Aj, int64_t lda,
                                    const double *__restrict__ Bj, int64_t ldbj, int64_t r2) {
  // column-major T; Aj r x r, Bj r2 x r (column-major); a null block is skipped
  const int64_t totalA = Aj ? r * r : 0, totalB = Bj ? r2 * r : 0;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < totalA + totalB;
       t += (int64_t)gridDim.x * blockDim.x) {
    if (t < totalA) {
      const int64_t i = t % r, j = t / r;
      T[(o + i) + (o + j) * ldt] = Aj[i + j * lda];
    } else {
      const int64_t u = t - totalA;
      const int64_t i = u % r2, j = u / r2;
      const double v = Bj[i + j * ldbj];
      T[(o + r + i) + (o + j) * ldt] = v;
      T[(o + j) + (o + r + i) * ldt] = v;
    }
  }
}

__global__ void gather_cols_cm_kernel(int64_t M, int64_t k, const double *__restrict__ src,
                                      int64_t lds, const int64_t *__restrict__ idx,
                                      double *__restrict__ dst, int64_t ldd) {
  const int64_t total = M * k;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % M, j = t / M;
    dst[i + j * ldd] = src[i + idx[j] * lds];
  }
}

__global__ void gather_cols_rm_kernel(int64_t n, int64_t k, const double *__restrict__ src,
                                      int64_t lds, const int64_t *__restrict__ idx,
                                      double *__restrict__ dst, int64_t ldd) {
  const int64_t total = n * k;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / k, j = t % k;
    dst[i * ldd + j] = src[i * lds + idx[j]];
  }
}

__global__ void add_diag_kernel(int64_t k, double *G, int64_t ld, double shift) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k;
       i += (int64_t)gridDim.x * blockDim.x)
    G[i + i * ld] += shift;
}

__global__ void zero_lower_kernel(int64_t k, double *G, int64_t ld) {
  const int64_t total = k * k;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % k, j = t / k;
    if (i > j) G[i + j * ld] = 0.0;
  }
}

__global__ void identity_kernel(int64_t k, double *G, int64_t ld) {
  const int64_t total = k * k;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t % k, j = t / k;
    G[i + j * ld] = i == j ? 1.0 : 0.0;
  }
}

// ------------------------------------------------------------------ CSR checks
__global__ void gershgorin_kernel(int64_t n, const int *__restrict__ rowptr,
                                  const int *__restrict__ colind, const double *__restrict__ val,
                                  double *__restrict__ pmin, double *__restrict__ pmax) {
  __shared__ double smin[256], smax[256];
  double lo = INFINITY, hi = -INFINITY;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double d = 0.0, r = 0.0;
    for (int j = rowptr[i]; j < rowptr[i + 1]; ++j) {
      if (colind[j] == i) d = val[j];
      else r += fabs(val[j]);
    }
    lo = fmin(lo, d - r);
    hi = fmax(hi, d + r);
  }
  smin[threadIdx.x] = lo;
  smax[threadIdx.x] = hi;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      smin[threadIdx.x] = fmin(smin[threadIdx.x], smin[threadIdx.x + s]);
      smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + s]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    pmin[blockIdx.x] = smin[0];
    pmax[blockIdx.x] = smax[0];
  }
}

// flags bit 0: columns not strictly increasing in a row; bit 1: A != A^T
__global__ void check_csr_kernel(int64_t n, const int *__restrict__ rowptr,
                                 const int *__restrict__ colind, const double *__restrict__ val,
                                 int *__restrict__ flags) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int s = rowptr[i], e = rowptr[i + 1];
    for (int t = s; t < e; ++t) {
      const int j = colind[t];
      if (t + 1 < e && colind[t + 1] <= j) atomicOr(flags, 1);
      if (j < 0 || j >= n) { atomicOr(flags, 1); continue; }
      const double v = val[t];
      // find (j, i) in row j by binary search
      int lo = rowptr[j], hi = rowptr[j + 1] - 1;
      bool found = false;
      double w = 0.0;
      while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const int c = colind[mid];
        if (c == i) { found = true; w = val[mid]; break; }
        if (c < i) lo = mid + 1; else hi = mid - 1;
      }
      if (found ? !(w == v) : (v != 0.0)) atomicOr(flags, 2);
    }
  }
}

}  // namespace

// ------------------------------------------------------------------ public launchers
template <typename T>
void launch_clenshaw_step(const sma_op *op, cudaStream_t st, int64_t b, const T *Q, int64_t ldq,
                          const T *B1, const T *B2, int64_t ldb, T *out, int64_t ldo, double ck,
                          double alpha, double beta, bool has_self, bool rev, bool tune) {
  if (op->n == 0 || b == 0) return;
  if (op->kind == OP_CSR) {
    csr_clenshaw_step<T>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev, tune);
  } else if (op->kind == OP_LAP1D || op->kind == OP_ANDERSON || op->kind == OP_XXZ) {
    model_clenshaw_step<T>(op, st, b, Q, ldq, B1, B2, ldb, out, ldo, ck, alpha, beta, has_self, rev);
  } else {
    throw Error(SMA_ERR_INTERNAL, "fused Clenshaw step needs a device operator");
  }
}

template <typename T>
void launch_clenshaw_start(const sma_op *op, cudaStream_t st, int64_t b, const T *Q, int64_t ldq,
                           const T *B1, int64_t ldb, T *out, int64_t ldo, double top, double ck,
                           double alpha, double beta, bool rev) {
  if (op->n == 0 || b == 0) return;
  if (op->kind == OP_CSR) {
    csr_clenshaw_start<T>(op, st, b, Q, ldq, B1, ldb, out, ldo, top, ck, alpha, beta, rev);
  } else if (op->kind == OP_LAP1D || op->kind == OP_ANDERSON || op->kind == OP_XXZ) {
    model_clenshaw_start<T>(op, st, b, Q, ldq, B1, ldb, out, ldo, top, ck, alpha, beta, rev);
  } else {
    throw Error(SMA_ERR_INTERNAL, "fused Clenshaw step needs a device operator");
  }
}

void launch_clenshaw_dots(const sma_op *op, cudaStream_t st, int64_t b, const double *Q, const double *B1,
                          double *out, double ck, double alpha, double beta, bool rev, int64_t cols,
                          double *dots, int64_t plane) {
  if (op->n == 0 || b == 0) return;
  if (op->kind == OP_CSR)
    csr_clenshaw_dots(op, st, b, Q, B1, out, ck, alpha, beta, rev, cols, dots, plane);
  else
    model_clenshaw_dots(op, st, b, Q, B1, out, ck, alpha, beta, rev, cols, dots, plane);
}

template <typename T>
void launch_scale_block(cudaStream_t st, int64_t n, int64_t b, const T *Q, int64_t ldq, T *out,
                        int64_t ldo, double ck) {
  const int64_t total = n * b;
  if (total == 0) return;
  if (total >> 32)
    scale_block_kernel<T, uint64_t><<<grid_for(total), 256, 0, st>>>(total, b, Q, ldq, out, ldo, (T)ck);
  else
    scale_block_kernel<T, uint32_t><<<grid_for(total), 256, 0, st>>>((uint32_t)total, (uint32_t)b, Q,
                                                                     ldq, out, ldo, (T)ck);
  SMA_CHECK_LAUNCH();
}

template <typename T>
void launch_clenshaw_axpy(cudaStream_t st, int64_t n, int64_t b, const T *Q, int64_t ldq,
                          const T *AX, int64_t ldax, const T *B1, const T *B2, int64_t ldb,
                          T *out, int64_t ldo, double ck, double alpha, double beta) {
  const int64_t total = n * b;
  if (total == 0) return;
  if (total >> 32)
    clenshaw_axpy_kernel<T, uint64_t><<<grid_for(total), 256, 0, st>>>(
        total, b, Q, ldq, AX, ldax, B1, B2, ldb, out, ldo, (T)ck, (T)alpha, (T)beta);
  else
    clenshaw_axpy_kernel<T, uint32_t><<<grid_for(total), 256, 0, st>>>(
        (uint32_t)total, (uint32_t)b, Q, ldq, AX, ldax, B1, B2, ldb, out, ldo, (T)ck, (T)alpha, (T)beta);
  SMA_CHECK_LAUNCH();
}

template <typename TS, typename TD>
void launch_pad_block(cudaStream_t st, int64_t n, int64_t b, const TS *src, int64_t lds, int64_t w,
                      TD *dst, int64_t ldd) {
  const int64_t total = n * w;
  if (total == 0) return;
  if (total >> 32)
    copy_block_kernel<TS, TD, uint64_t><<<grid_for(total), 256, 0, st>>>(total, w, b, src, lds, dst, ldd);
  else
    copy_block_kernel<TS, TD, uint32_t><<<grid_for(total), 256, 0, st>>>(
        (uint32_t)total, (uint32_t)w, (uint32_t)b, src, lds, dst, ldd);
  SMA_CHECK_LAUNCH();
}

template <typename TS, typename TD>
void launch_copy_block(cudaStream_t st, int64_t n, int64_t b, const TS *src, int64_t lds, TD *dst,
                       int64_t ldd) {
  launch_pad_block<TS, TD>(st, n, b, src, lds, b, dst, ldd);
}

template void launch_pad_block<double, double>(cudaStream_t, int64_t, int64_t, const double *,
                                               int64_t, int64_t, double *, int64_t);
template void launch_pad_block<float, float>(cudaStream_t, int64_t, int64_t, const float *, int64_t,
                                             int64_t, float *, int64_t);
template void launch_clenshaw_step<double>(const sma_op *, cudaStream_t, int64_t, const double *,
                                           int64_t, const double *, const double *, int64_t,
                                           double *, int64_t, double, double, double, bool, bool, bool);
template void launch_clenshaw_step<float>(const sma_op *, cudaStream_t, int64_t, const float *,
                                          int64_t, const float *, const float *, int64_t, float *,
                                          int64_t, double, double, double, bool, bool, bool);
template void launch_clenshaw_start<double>(const sma_op *, cudaStream_t, int64_t, const double *,
                                            int64_t, const double *, int64_t, double *, int64_t, double,
                                            double, double, double, bool);
template void launch_clenshaw_start<float>(const sma_op *, cudaStream_t, int64_t, const float *,
                                           int64_t, const float *, int64_t, float *, int64_t, double,
                                           double, double, double, bool);
template void launch_scale_block<double>(cudaStream_t, int64_t, int64_t, const double *, int64_t,
                                         double *, int64_t, double);
template void launch_scale_block<float>(cudaStream_t, int64_t, int64_t, const float *, int64_t,
                                        float *, int64_t, double);
template void launch_clenshaw_axpy<double>(cudaStream_t, int64_t, int64_t, const double *, int64_t,
                                           const double *, int64_t, const double *, const double *,
                                           int64_t, double *, int64_t, double, double, double);
template void launch_clenshaw_axpy<float>(cudaStream_t, int64_t, int64_t, const float *, int64_t,
                                          const float *, int64_t, const float *, const float *,
                                          int64_t, float *, int64_t, double, double, double);
template void launch_copy_block<double, double>(cudaStream_t, int64_t, int64_t, const double *,
                                                int64_t, double *, int64_t);
template void launch_copy_block<double, float>(cudaStream_t, int64_t, int64_t, const double *,
                                               int64_t, float *, int64_t);
template void launch_copy_block<float, double>(cudaStream_t, int64_t, int64_t, const float *,
                                               int64_t, double *, int64_t);
template void launch_copy_block<float, float>(cudaStream_t, int64_t, int64_t, const float *,
                                              int64_t, float *, int64_t);

void launch_randn(cudaStream_t st, int64_t n, int64_t m, uint64_t seed, double *out, int64_t ld) {
  if (n * m == 0) return;
  randn_kernel<<<grid_for(n * m), 256, 0, st>>>(n, m, seed, out, ld);
  SMA_CHECK_LAUNCH();
}

// 2^lc columns of a CTA: up to 32
static int column_lanes(int64_t k) {
  int lc = 0;
  while (lc < 5 && (1 << lc) < k) ++lc;
  return lc;
}

void column_dots(cudaStream_t st, int64_t n, int64_t k, const double *X, int64_t ldx, const double *Y,
                 int64_t ldy, double *partial) {
  const int lc = column_lanes(k);
  const int64_t chunks = column_dot_chunks(n, k);
  const dim3 grid((unsigned)chunks, (unsigned)((k + (1 << lc) - 1) >> lc));
  dots_stage1<<<grid, 256, 0, st>>>(lc, n, k, X, ldx, Y, ldy, partial, (n + chunks - 1) / chunks, chunks * k);
  SMA_CHECK_LAUNCH();
}

// Chunks of rows: four CTAs an SM over the whole grid, each thread summing at least eight rows.
int64_t column_dot_chunks(int64_t n, int64_t k) {
  const int64_t ctiles = (k + 31) / 32;
  const int64_t rows = k >= 32 ? 64 : 8 * (256 / std::max<int64_t>(k, 1));
  return std::max<int64_t>(1, std::min<int64_t>((n + rows - 1) / rows, (148 * 4 + ctiles - 1) / ctiles));
}

void column_dot_totals(cudaStream_t st, int64_t chunks, int64_t k, int64_t groups, const double *partial,
                       double *out) {
  const int64_t total = groups * k;
  dots_stage2<<<(unsigned)((total + 31) / 32), 256, 0, st>>>(chunks, k, total, partial, out);
  SMA_CHECK_LAUNCH();
}

void column_reduce(cudaStream_t st, int mode, int64_t n, int64_t k, const double *X, int64_t ldx,
                   const double *Y, int64_t ldy, const double *lam, double *out,
                   DevBuf<double> &scratch) {
  if (k == 0) return;
  const int64_t tiles = (k + 31) / 32;
  int64_t chunks = std::max<int64_t>(1, std::min<int64_t>((n + 63) / 64, (148 * 8 + tiles - 1) / tiles));
  const int64_t rows = (n + chunks - 1) / chunks;
  chunks = rows ? (n + rows - 1) / rows : 1;
  if (scratch.count < (size_t)(chunks * k)) scratch.alloc(chunks * k, st);
  const int lc = column_lanes(k), each = 32 >> lc;
  const dim3 grid((unsigned)((chunks + each - 1) / each), (unsigned)((k + (1 << lc) - 1) >> lc));
  colred_stage1<<<grid, 256, 0, st>>>(mode, lc, n, k, X, ldx, Y, ldy, lam, scratch.p, chunks, rows);
  SMA_CHECK_LAUNCH();
  colred_stage2<<<(unsigned)((k + kSumLanes - 1) / kSumLanes), 256, 0, st>>>(mode, chunks, k, scratch.p, out);
  SMA_CHECK_LAUNCH();
}

static void transpose(cudaStream_t st, int64_t R, int64_t C, const double *in, int64_t ldi,
                      double *out, int64_t ldo) {
  if (R * C == 0) return;
  dim3 grid((unsigned)((C + 31) / 32), (unsigned)((R + 31) / 32));
  transpose_kernel<<<grid, dim3(32, 8), 0, st>>>(R, C, in, ldi, out, ldo);
  SMA_CHECK_LAUNCH();
}

void launch_rowmajor_to_colmajor(cudaStream_t st, int64_t n, int64_t k, const double *src,
                                 int64_t lds, double *dst) {
  transpose(st, n, k, src, lds, dst, n);
}

void launch_colmajor_to_rowmajor(cudaStream_t st, int64_t n, int64_t k, const double *src,
                                 double *dst, int64_t ldd) {
  // column-major n x k (ld n) is row-major k x n (ld n)
  transpose(st, k, n, src, n, dst, ldd);
}

void launch_symmetrize(cudaStream_t st, int64_t k, const double *G, int64_t ldg, double *H,
                       int64_t ldh) {
  if (k == 0) return;
  symmetrize_kernel<<<grid_for(k * k), 256, 0, st>>>(k, G, ldg, H, ldh);
  SMA_CHECK_LAUNCH();
}

void launch_place_blocks(cudaStream_t st, double *T, int64_t ldt, int64_t o, int64_t r,
                         const double *Aj, int64_t lda, const double *Bj, int64_t ldbj,
                         int64_t r2) {
  const int64_t total = (Aj ? r * r : 0) + (Bj ? r2 * r : 0);
  if (total == 0) return;
  place_blocks_kernel<<<grid_for(total), 256, 0, st>>>(T, ldt, o, r, Aj, lda, Bj, ldbj, r2);
  SMA_CHECK_LAUNCH();
}

void launch_gather_columns_cm(cudaStream_t st, int64_t M, int64_t k, const double *src,
                              int64_t lds, const int64_t *idx, double *dst, int64_t ldd) {
  if (M * k == 0) return;
  gather_cols_cm_kernel<<<grid_for(M * k), 256, 0, st>>>(M, k, src, lds, idx, dst, ldd);
  SMA_CHECK_LAUNCH();
}

void launch_gather_columns_rm(cudaStream_t st, int64_t n, int64_t k, const double *src,
                              int64_t lds, const int64_t *idx, double *dst, int64_t ldd) {
  if (n * k == 0) return;
  gather_cols_rm_kernel<<<grid_for(n * k), 256, 0, st>>>(n, k, src, lds, idx, dst, ldd);
  SMA_CHECK_LAUNCH();
}

void launch_add_diagonal(cudaStream_t st, int64_t k, double *G, int64_t ld, double shift) {
  if (k == 0) return;
  add_diag_kernel<<<grid_for(k), 256, 0, st>>>(k, G, ld, shift);
  SMA_CHECK_LAUNCH();
}

void launch_zero_lower(cudaStream_t st, int64_t k, double *G, int64_t ld) {
  if (k == 0) return;
  zero_lower_kernel<<<grid_for(k * k), 256, 0, st>>>(k, G, ld);
  SMA_CHECK_LAUNCH();
}

void launch_identity(cudaStream_t st, int64_t k, double *G, int64_t ld) {
  if (k == 0) return;
  identity_kernel<<<grid_for(k * k), 256, 0, st>>>(k, G, ld);
  SMA_CHECK_LAUNCH();
}

void gershgorin_device(const sma_op *op, double *smin, double *smax) {
  cudaStream_t st = op->ctx->stream;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((op->n + 255) / 256, 1024));
  DevBuf<double> part(2 * grid, st);
  gershgorin_kernel<<<grid, 256, 0, st>>>(op->n, op->rowptr, op->colind, op->val64, part.p,
                                          part.p + grid);
  SMA_CHECK_LAUNCH();
  std::vector<double> h(2 * grid);
  SMA_CUDA(cudaMemcpyAsync(h.data(), part.p, 2 * grid * sizeof(double), cudaMemcpyDeviceToHost, st));
  SMA_CUDA(cudaStreamSynchronize(st));
  double lo = INFINITY, hi = -INFINITY;
  for (int i = 0; i < grid; ++i) {
    lo = std::min(lo, h[i]);
    hi = std::max(hi, h[grid + i]);
  }
  *smin = lo;
  *smax = hi;
}

int check_csr_device(const sma_op *op) {
  cudaStream_t st = op->ctx->stream;
  DevBuf<int> flag(1, st);
  SMA_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(int), st));
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((op->n + 255) / 256, 4096));
  check_csr_kernel<<<grid, 256, 0, st>>>(op->n, op->rowptr, op->colind, op->val64, flag.p);
  SMA_CHECK_LAUNCH();
  int h = 0;
  SMA_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  SMA_CUDA(cudaStreamSynchronize(st));
  if (h & 1) return 1;
  if (h & 2) return 2;
  return 0;
}

}  // namespace sma
