// FP64 tensor-core products for the dense part of the solvers (DMMA: mma.sync f64 on the
// B200's FP64 tensor pipe).  Two shapes cover every tall-skinny product of the block
// orthogonalization, reorthogonalization and Rayleigh-Ritz lift (n >> m, k, p):
//
//   gram    C (m x k, column-major, ldc) = alpha X^T Y + beta C
//           X: n x m, Y: n x k, row-major (ldx, ldy) -- the reduction runs over n;
//   update  Y (n x p, row-major, ldy)    = alpha X B + beta Y
//           X: n x m row-major (ldx); B: m x p given as a column-major C (B = C, ldc) or as
//           the transpose of one (B = C^T, C p x m column-major, ldc).
//
// Both run mma.sync.aligned.m8n8k4.row.col.f64 on operand tiles that cp.async brings to shared
// memory, three chunks of 16 in flight and one barrier a chunk: a warp owns a 32 x 32 piece of the
// CTA's 64 x 64 output tile (smaller ones for narrow products), keeps its accumulators in
// registers and reads the next four indices' fragments while it multiplies.  The gram splits n
// over the grid; every CTA writes its partial tile to a workspace and a second kernel sums the
// partials one after the other, so results are deterministic (the same bits every run, and with
// every tile).  The update owns whole rows of Y: with beta = 0 it
// may write in place over X when p <= 64 (X <- X B, the triangular solve of CholQR written as a
// product with R^-1), since a CTA reads all of its rows of X before it writes them.
//
// What bounds it: the FP64 tensor pipe, 37.1 TFLOP/s measured from registers.  Four warps a CTA
// and three CTAs an SM keep it busier than eight and two (35.7 against 34.7 TFLOP/s at p = 512),
// and the copies' addresses are pointers that advance: recomputed for every chunk they cost as
// much as the barriers (31.3 TFLOP/s).
//
// DMMA fragment layout of m8n8k4 (PTX ISA, "Matrix Fragments for mma.m8n8k4 with .f64"):
// lane = 4 g + t (g = groupID 0..7, t = thread in group 0..3);
//   A (8 x 4, row):  a0 = A[g][t];   B (4 x 8, col): b0 = B[t][g];
//   C/D (8 x 8):     c0 = C[g][2t], c1 = C[g][2t + 1].
#include <algorithm>

#include "ordered_sum.cuh"
#include "sma_internal.h"
#include "vec.cuh"

namespace sma {
namespace dmma {

constexpr int kThreads = 128;  // four warps
constexpr int kDepth = 16;     // summation indices of a chunk

__device__ __forceinline__ void mma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// BYTES (8 or 16) from global to shared memory, zeros where !ok (the source is then not read).
template <int BYTES>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem, bool ok) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  const int n = ok ? BYTES : 0;
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// A CTA tile of WM x WN warps, each MT x NT fragments of 8 x 8; chunks in flight and CTAs an SM.
template <int WM_, int WN_, int MT_, int NT_, int STAGES_ = 3, int CTAS_ = 3>
struct Tile {
  using Self = Tile;
  static constexpr int WM = WM_, WN = WN_, MT = MT_, NT = NT_, kStages = STAGES_, kCtas = CTAS_;
  static constexpr int M = WM * MT * 8, N = WN * NT * 8;
  static_assert(WM * WN * 32 == kThreads, "four warps");
  static_assert(M % 16 == 0 && N % 16 == 0, "whole passes of 16-byte copies");
};

// acc += A B over one chunk: a(k, i) and b(k, j) give this lane's element of fragment i (j) at
// summation index k; the fragments of k + 4 are read before those of k are multiplied.
template <typename T, typename A, typename B>
__device__ __forceinline__ void multiply(double (&acc)[T::MT][T::NT][2], const A &a, const B &b) {
  double fa[2][T::MT], fb[2][T::NT];
#pragma unroll
  for (int i = 0; i < T::MT; ++i) fa[0][i] = a(0, i);
#pragma unroll
  for (int j = 0; j < T::NT; ++j) fb[0][j] = b(0, j);
#pragma unroll
  for (int k = 0; k < kDepth; k += 4) {
    const int cur = (k / 4) & 1;
    if (k + 4 < kDepth) {
#pragma unroll
      for (int i = 0; i < T::MT; ++i) fa[cur ^ 1][i] = a(k + 4, i);
#pragma unroll
      for (int j = 0; j < T::NT; ++j) fb[cur ^ 1][j] = b(k + 4, j);
    }
#pragma unroll
    for (int i = 0; i < T::MT; ++i)
#pragma unroll
      for (int j = 0; j < T::NT; ++j) mma_8x8x4(acc[i][j], fa[cur][i], fb[cur][j]);
  }
}

template <typename T>
__device__ __forceinline__ void clear(double (&acc)[T::MT][T::NT][2]) {
#pragma unroll
  for (int i = 0; i < T::MT; ++i)
#pragma unroll
    for (int j = 0; j < T::NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
}

// The chunks 0..nk-1 through the stages: load(stage, chunk) issues copies, use(stage) computes.
template <int kStages, typename Load, typename Use>
__device__ __forceinline__ void pipeline(int nk, const Load &load, const Use &use) {
#pragma unroll
  for (int c = 0; c < kStages - 1; ++c) {
    if (c < nk) load(c, c);
    cp_async_commit();
  }
  int stage = 0;
  for (int c = 0; c < nk; ++c) {
    cp_async_wait<kStages - 2>();  // chunk c has landed (this thread's part of it)
    __syncthreads();               // everybody's; and chunk c - 1 is consumed: its stage is free
    const int next = c + kStages - 1;
    if (next < nk) load(stage == 0 ? kStages - 1 : stage - 1, next);
    cp_async_commit();
    use(stage);
    stage = stage + 1 == kStages ? 0 : stage + 1;
  }
}

// ------------------------------------------------------------------ update
constexpr int kPad = kDepth + 4;  // shared rows of 20 doubles: conflict-free fragment reads

template <typename T>
struct UpdateSmem {
  double a[T::kStages][T::M][kPad];
  double b[T::kStages][T::N][kPad];  // stored [column][k]
};

// B(i, j): TB = false -> C[i + j ldc] (column-major m x p); TB = true -> C[j + i ldc] (the
// transpose of a column-major p x m).  vecx, vecc, vecy: 16-byte accesses of X, C (TB = false), Y.
template <bool TB, typename T>
__global__ void __launch_bounds__(kThreads, T::kCtas)
update_kernel(int64_t n, int m, int p, const double *X, int64_t ldx,  // Y may alias X
              const double *__restrict__ C, int64_t ldc, double *Y, int64_t ldy, double alpha,
              double beta, int coltiles, bool vecx, bool vecc, bool vecy) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  UpdateSmem<T> &sm = *reinterpret_cast<UpdateSmem<T> *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = warp % T::WM * T::MT * 8, wc = warp / T::WM * T::NT * 8;
  // column tiles next to each other: they read the same rows of X
  const int64_t row0 = (int64_t)(blockIdx.x / coltiles) * T::M;
  const int col0 = blockIdx.x % coltiles * T::N;
  double acc[T::MT][T::NT][2];
  clear<T>(acc);
  // This thread's 16-byte copies of a whole chunk: rows r of X (columns of C), two indices from c
  // on; the pointers advance with the chunks.
  constexpr int kPerRow = kDepth / 2, PA = T::M * kPerRow / kThreads, PB = T::N * kPerRow / kThreads;
  static_assert(T::M * kPerRow % kThreads == 0 && T::N * kPerRow % kThreads == 0, "whole passes");
  const int r = tid / kPerRow, c = tid % kPerRow * 2;
  constexpr int kStep = kThreads / kPerRow;  // rows between two copies of a thread
  const double *px[PA], *pc[PB];
#pragma unroll
  for (int i = 0; i < PA; ++i)
    px[i] = row0 + r + i * kStep < n ? X + (row0 + r + i * kStep) * ldx + c : nullptr;
#pragma unroll
  for (int i = 0; i < PB; ++i)
    pc[i] = !TB && col0 + r + i * kStep < p ? C + (int64_t)(col0 + r + i * kStep) * ldc + c : nullptr;
  auto load = [&](int stage, int chunk) {
    const int k0 = chunk * kDepth;
    const bool whole = k0 + kDepth <= m;
    if (vecx && whole) {
#pragma unroll
      for (int i = 0; i < PA; ++i) {
        cp_async<16>(&sm.a[stage][r + i * kStep][c], px[i] ? px[i] : X, px[i] != nullptr);
        if (px[i]) px[i] += kDepth;
      }
    } else {
      for (int e = tid; e < T::M * kDepth; e += kThreads) {
        const int rr = e / kDepth, cc = e % kDepth;
        const bool ok = row0 + rr < n && k0 + cc < m;
        cp_async<8>(&sm.a[stage][rr][cc], X + (ok ? (row0 + rr) * ldx + k0 + cc : 0), ok);
      }
    }
    if (!TB && vecc && whole) {
#pragma unroll
      for (int i = 0; i < PB; ++i) {
        cp_async<16>(&sm.b[stage][r + i * kStep][c], pc[i] ? pc[i] : C, pc[i] != nullptr);
        if (pc[i]) pc[i] += kDepth;
      }
    } else {
      for (int e = tid; e < T::N * kDepth; e += kThreads) {
        const int j = TB ? e % T::N : e / kDepth, kk = TB ? e / T::N : e % kDepth;
        const int gk = k0 + kk, gj = col0 + j;
        const bool ok = gk < m && gj < p;
        cp_async<8>(&sm.b[stage][j][kk], C + (!ok ? 0 : TB ? gj + (int64_t)gk * ldc : gk + (int64_t)gj * ldc), ok);
      }
    }
  };
  pipeline<T::kStages>((m + kDepth - 1) / kDepth, load, [&](int stage) {  // m = 0: Y = beta Y
    const double *a = &sm.a[stage][wr + g][t], *b = &sm.b[stage][wc + g][t];
    multiply<T>(acc, [&](int k, int i) { return a[i * 8 * kPad + k]; },
                [&](int k, int j) { return b[j * 8 * kPad + k]; });
  });
  // Y = alpha acc + beta Y (Y not read when beta == 0), the first product and the sum rounded once
#pragma unroll
  for (int i = 0; i < T::MT; ++i) {
    const int64_t yr = row0 + wr + i * 8 + g;
    if (yr >= n) continue;
#pragma unroll
    for (int j = 0; j < T::NT; ++j) {
      const int yc = col0 + wc + j * 8 + 2 * t;
      double *y = Y + yr * ldy + yc;
      auto result = [&](double sum, const double &old) {
        return beta == 0.0 ? alpha * sum : fma(alpha, sum, mul_rn(beta, old));
      };
      if (vecy && yc + 1 < p) {
        double2 *y2 = reinterpret_cast<double2 *>(y);
        const double2 o = beta == 0.0 ? make_double2(0.0, 0.0) : *y2;
        *y2 = make_double2(result(acc[i][j][0], o.x), result(acc[i][j][1], o.y));
      } else {
        if (yc < p) y[0] = result(acc[i][j][0], y[0]);
        if (yc + 1 < p) y[1] = result(acc[i][j][1], y[1]);
      }
    }
  }
}

// ------------------------------------------------------------------ gram
template <typename T>
struct GramSmem {
  double x[T::kStages][kDepth][T::M + 4];
  double y[T::kStages][kDepth][T::N + 4];
};

// Whether the tile at (m0, k0) lies below the diagonal.
template <typename T>
__host__ __device__ __forceinline__ bool below(int m0, int k0) { return m0 >= k0 + T::N; }

// Tile (blockIdx.x, blockIdx.y) of X^T Y over the rows of split blockIdx.z; its partial product
// column-major into the workspace.
template <typename T>
__global__ void __launch_bounds__(kThreads, T::kCtas)
gram_partial_kernel(int64_t n, int m, int k, const double *__restrict__ X, int64_t ldx,
                    const double *__restrict__ Y, int64_t ldy, int64_t rows_per_split,
                    double *__restrict__ part, bool vecx, bool vecy, bool upper) {
  const int m0 = blockIdx.x * T::M, k0 = blockIdx.y * T::N;
  if (upper && below<T>(m0, k0)) return;  // no barrier yet
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GramSmem<T> &sm = *reinterpret_cast<GramSmem<T> *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wm = warp % T::WM * T::MT * 8, wk = warp / T::WM * T::NT * 8;
  const int64_t r0 = (int64_t)blockIdx.z * rows_per_split;
  const int64_t r1 = min(n, r0 + rows_per_split);
  double acc[T::MT][T::NT][2];
  clear<T>(acc);
  const int64_t nrows = r1 > r0 ? r1 - r0 : 0;
  // This thread's 16-byte copies of a whole chunk: rows rx + i * .. of X (ry of Y) at columns cx
  // (cy); the pointers advance with the chunks.
  constexpr int WX = T::M / 2, WY = T::N / 2;  // copies of a row
  constexpr int SX = kThreads / WX, SY = kThreads / WY, PX = kDepth / SX, PY = kDepth / SY;
  const int rx = tid / WX, cx = tid % WX * 2, ry = tid / WY, cy = tid % WY * 2;
  const bool wholex = vecx && m0 + T::M <= m, wholey = vecy && k0 + T::N <= k;
  const double *px = X + (r0 + rx) * ldx + m0 + cx, *py = Y + (r0 + ry) * ldy + k0 + cy;
  const int64_t stepx = SX * ldx, stepy = SY * ldy;
  auto slow = [&](double *dst, int pitch, int W, const double *src, int64_t ld, int c0, int cols,
                  int64_t rb) {
    for (int e = tid; e < kDepth * W; e += kThreads) {
      const int rr = e / W, cc = e % W;
      const bool ok = rb + rr < r1 && c0 + cc < cols;
      cp_async<8>(dst + rr * pitch + cc, src + (ok ? (rb + rr) * ld + c0 + cc : 0), ok);
    }
  };
  auto load = [&](int stage, int chunk) {
    const int64_t rb = r0 + (int64_t)chunk * kDepth;
    const bool whole = rb + kDepth <= r1;
    if (wholex && whole) {
#pragma unroll
      for (int i = 0; i < PX; ++i) {
        cp_async<16>(&sm.x[stage][rx + i * SX][cx], px, true);
        px += stepx;
      }
    } else {
      slow(&sm.x[stage][0][0], T::M + 4, T::M, X, ldx, m0, m, rb);
    }
    if (wholey && whole) {
#pragma unroll
      for (int i = 0; i < PY; ++i) {
        cp_async<16>(&sm.y[stage][ry + i * SY][cy], py, true);
        py += stepy;
      }
    } else {
      slow(&sm.y[stage][0][0], T::N + 4, T::N, Y, ldy, k0, k, rb);
    }
  };
  pipeline<T::kStages>((int)((nrows + kDepth - 1) / kDepth), load, [&](int stage) {
    const double *a = &sm.x[stage][t][wm + g], *b = &sm.y[stage][t][wk + g];  // A = X^T
    multiply<T>(acc, [&](int kk, int i) { return a[kk * (T::M + 4) + i * 8]; },
                [&](int kk, int j) { return b[kk * (T::N + 4) + j * 8]; });
  });
  double *pt = part + (((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * (T::M * T::N);
#pragma unroll
  for (int i = 0; i < T::MT; ++i)
#pragma unroll
    for (int j = 0; j < T::NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        pt[wm + i * 8 + g + (wk + j * 8 + 2 * t + h) * T::M] = acc[i][j][h];
}

// Element e of C = alpha * sum_z part_z + beta C: its place in the partials of split 0, or -1 where
// those below the diagonal were never written.
template <typename T>
__device__ __forceinline__ int64_t partial_place(int64_t e, int m, int tiles_m, bool upper) {
  const int i = (int)(e % m), j = (int)(e / m), bx = i / T::M, by = j / T::N;
  if (upper && below<T>(bx * T::M, by * T::N)) return -1;
  return ((int64_t)by * tiles_m + bx) * (T::M * T::N) + i % T::M + j % T::N * T::M;
}
__device__ __forceinline__ void finish(double *C, int64_t ldc, int64_t e, int m, double s, double alpha,
                                       double beta) {
  double *c = C + e % m + e / m * ldc;
  *c = beta == 0.0 ? alpha * s : alpha * s + beta * *c;
}

// Both sum the splits one after the other, whatever the tiles were: with few splits a thread an
// element, with many a CTA LANES elements at a time.
template <typename T>
__global__ void __launch_bounds__(256)
gram_reduce_kernel(int m, int k, int tiles_m, int tiles_k, int splits, const double *__restrict__ part,
                   double *C, int64_t ldc, double alpha, double beta, bool upper) {
  const int64_t total = (int64_t)m * k, stride = (int64_t)tiles_k * tiles_m * (T::M * T::N);
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t at = partial_place<T>(e, m, tiles_m, upper);
    if (at < 0) continue;
    double s = 0.0;
#pragma unroll 8
    for (int z = 0; z < splits; ++z) s += part[at + z * stride];
    finish(C, ldc, e, m, s, alpha, beta);
  }
}

template <typename T, int LANES>
__global__ void __launch_bounds__(256)
gram_reduce_many_kernel(int m, int k, int tiles_m, int tiles_k, int splits, const double *__restrict__ part,
                        double *C, int64_t ldc, double alpha, double beta, bool upper) {
  __shared__ OrderedSum<LANES, 8> sum;
  const int64_t total = (int64_t)m * k, stride = (int64_t)tiles_k * tiles_m * (T::M * T::N);
  for (int64_t e0 = (int64_t)blockIdx.x * LANES; e0 < total; e0 += (int64_t)gridDim.x * LANES) {
    const int64_t e = e0 + threadIdx.x % LANES, at = e < total ? partial_place<T>(e, m, tiles_m, upper) : -1;
    const double s = sum(at < 0 ? nullptr : part + at, stride, splits);
    if (threadIdx.x < LANES && at >= 0) finish(C, ldc, e, m, s, alpha, beta);
  }
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15) == 0; }

template <bool TB, typename T>
void launch_update(cudaStream_t st, int64_t n, int64_t m, int64_t p, const double *X, int64_t ldx,
                   const double *C, int64_t ldc, double *Y, int64_t ldy, double alpha, double beta) {
  const int64_t coltiles = (p + T::N - 1) / T::N, grid = (n + T::M - 1) / T::M * coltiles;
  require(grid < (int64_t)1 << 31, SMA_ERR_ARG, "product too large");
  const size_t smem = sizeof(UpdateSmem<T>);
  SMA_CUDA(cudaFuncSetAttribute(update_kernel<TB, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  update_kernel<TB, T><<<(unsigned)grid, kThreads, smem, st>>>(
      n, (int)m, (int)p, X, ldx, C, ldc, Y, ldy, alpha, beta, (int)coltiles,
      aligned16(X) && ldx % 2 == 0, aligned16(C) && ldc % 2 == 0, aligned16(Y) && ldy % 2 == 0);
  SMA_CHECK_LAUNCH();
}

template <typename T>
void launch_gram(cudaStream_t st, int num_sms, int64_t n, int64_t m, int64_t k, const double *X,
                 int64_t ldx, const double *Y, int64_t ldy, double *C, int64_t ldc, double alpha,
                 double beta, DevBuf<double> &work, bool upper, int64_t splits) {
  const int tm = (int)((m + T::M - 1) / T::M), tk = (int)((k + T::N - 1) / T::N);
  const int64_t rows = (n + splits - 1) / splits;
  const size_t need = (size_t)splits * tm * tk * T::M * T::N;
  if (work.count < need) work.alloc(need, st);
  const bool vecx = aligned16(X) && ldx % 2 == 0, vecy = aligned16(Y) && ldy % 2 == 0;
  const size_t smem = sizeof(GramSmem<T>);
  SMA_CUDA(cudaFuncSetAttribute(gram_partial_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  gram_partial_kernel<T><<<dim3(tm, tk, (unsigned)splits), kThreads, smem, st>>>(
      n, (int)m, (int)k, X, ldx, Y, ldy, rows, work.p, vecx, vecy, upper);
  SMA_CHECK_LAUNCH();
  auto reduce = [&](auto kernel, int elements) {
    const int blocks = (int)std::min<int64_t>((m * k + elements - 1) / elements, 8LL * num_sms);
    kernel<<<blocks, 256, 0, st>>>((int)m, (int)k, tm, tk, (int)splits, work.p, C, ldc, alpha, beta, upper);
  };
  if (splits <= 32) reduce(gram_reduce_kernel<T>, 256);
  else if (m * k <= 4096) reduce(gram_reduce_many_kernel<T, 8>, 8);
  else reduce(gram_reduce_many_kernel<T, 32>, 32);
  SMA_CHECK_LAUNCH();
}

using Wide = Tile<2, 2, 4, 4>;         // 64 x 64
using Short = Tile<2, 2, 4, 4, 2, 4>;  // the same for a short summation: more CTAs to hide its ends
using Narrow = Tile<4, 1, 2, 4>;       // 64 x 32
using Small = Tile<2, 2, 2, 2, 3, 6>;  // 32 x 32
using Tiny = Tile<2, 2, 1, 1, 3, 8>;   // 16 x 16, gram only

// The time of a product's tiles in us, from what a chunk takes: `shared`, its share of a busy SM
// (the tensor pipe and what a size of tile loses beside it), and `alone`, the latency of a CTA that
// has the SM for itself.  Measured with one tile against another at 60 shapes, n = 3000 to 262144:
// large tiles win only where they are full and make many waves (262144 x 1024 x 64: update 1042 us
// with 64 x 64, 1101 with 32 x 32; 30000 x 1024 x 64: 198 and 142).  Of the gram, whose tiles below
// the diagonal leave gaps, whole calls in us with 64 x 64, 64 x 32, 32 x 32 and 16 x 16:
//   262144 x 1024 x 64   1060, 1143, 1148, 1744     262144 x 480 x 32   579, 305, 323, 432
//   262144 x 160 x 160    694,  727,  497,  685      20000 x 32 x 32     36,  30,  25,  24
//   262144 x 200 x 16     313,  209,  227,  141       3000 x 16 x 8      38,  33,  30,  25
struct Rate {
  double shared, alone;
  int ctas;
};
constexpr Rate kWide{0.585, 1.05, Wide::kCtas}, kShort{0.60, 1.05, Short::kCtas},
    kNarrow{0.305, 0.75, Narrow::kCtas}, kSmall{0.160, 0.52, Small::kCtas};

inline double tiles_time(const Rate &r, int64_t tiles, int64_t chunks, int sms) {
  auto wave = [&](int64_t each) { return (chunks + 2) * std::max(r.alone, each * r.shared); };
  const int64_t slots = (int64_t)r.ctas * sms, rest = tiles % slots;
  return (tiles / slots) * wave(r.ctas) + (rest ? wave((rest + sms - 1) / sms) : 0.0);
}

// The gram's splits of n: two CTAs an SM if the tiles were 64 x 64, at least 256 rows each.  They and
// the order in which they are summed fix the result's last bits, so they follow from the shape alone
// and not from the tile: a solve that keeps an unconverged pair carries a last bit of its basis to the
// sixth digit of that pair.
int64_t gram_splits(int64_t n, int64_t m, int64_t k, int sms) {
  const int64_t want = 2LL * sms / (((m + 63) / 64) * ((k + 63) / 64));
  return std::max<int64_t>(1, std::min<int64_t>(want, (n + 255) / 256));
}

// Its CTAs are long: those past the first wave start as others end, with no gap between.
template <typename T>
double gram_time(const Rate &r, int64_t n, int64_t m, int64_t k, bool upper, int64_t splits, int sms) {
  int64_t tiles = 0;
  for (int64_t x = 0; x < m; x += T::M)
    for (int64_t y = 0; y < k; y += T::N) tiles += !(upper && below<T>((int)x, (int)y));
  const int64_t ctas = tiles * splits, chunks = ((n + splits - 1) / splits + kDepth - 1) / kDepth;
  const double each = ctas <= r.ctas * sms ? (double)((ctas + sms - 1) / sms) : (double)ctas / sms;
  return (chunks + 2) * std::max(r.alone, each * r.shared);
}

}  // namespace dmma

void dgemm_update(cudaStream_t st, int num_sms, int64_t n, int64_t m, int64_t p, const double *X,
                  int64_t ldx, const double *C, int64_t ldc, bool transC, double *Y, int64_t ldy,
                  double alpha, double beta) {
  using namespace dmma;
  if (n == 0 || p == 0) return;
  require(m <= INT32_MAX && p <= INT32_MAX, SMA_ERR_ARG, "product too wide");
  auto run = [&](auto tile) {
    using T = typename decltype(tile)::Self;
    if (transC) launch_update<true, T>(st, n, m, p, X, ldx, C, ldc, Y, ldy, alpha, beta);
    else launch_update<false, T>(st, n, m, p, X, ldx, C, ldc, Y, ldy, alpha, beta);
  };
  auto time = [&](auto tile, const Rate &r) {
    using T = typename decltype(tile)::Self;
    return tiles_time(r, (n + T::M - 1) / T::M * ((p + T::N - 1) / T::N), (m + kDepth - 1) / kDepth, num_sms);
  };
  // in place one CTA has to read a row of X before it is written: no tile narrower than p
  const bool in_place = (uintptr_t)X < (uintptr_t)(Y + n * ldy) && (uintptr_t)Y < (uintptr_t)(X + n * ldx);
  const double small = in_place && p > 32 ? 1e300 : time(Small{}, kSmall);
  if (p <= 32) {  // half of a wide tile would be padding
    if (small <= time(Narrow{}, kNarrow)) run(Small{});
    else run(Narrow{});
  } else if (m <= 128) {
    if (small <= time(Short{}, kShort)) run(Small{});
    else run(Short{});
  } else {
    if (small <= time(Wide{}, kWide)) run(Small{});
    else run(Wide{});
  }
}

void dgemm_gram(cudaStream_t st, int num_sms, int64_t n, int64_t m, int64_t k, const double *X,
                int64_t ldx, const double *Y, int64_t ldy, double *C, int64_t ldc, double alpha,
                double beta, DevBuf<double> &work, bool upper) {
  using namespace dmma;
  if (m == 0 || k == 0) return;
  require(m <= INT32_MAX && k <= INT32_MAX, SMA_ERR_ARG, "product too wide");
  upper = upper && m == k;
  const int64_t splits = gram_splits(n, m, k, num_sms);
  auto run = [&](auto tile) {
    using T = typename decltype(tile)::Self;
    launch_gram<T>(st, num_sms, n, m, k, X, ldx, Y, ldy, C, ldc, alpha, beta, work, upper, splits);
  };
  auto time = [&](auto tile, const Rate &r) {
    using T = typename decltype(tile)::Self;
    return gram_time<T>(r, n, m, k, upper, splits, num_sms);
  };
  const double small = time(Small{}, kSmall);
  if (k <= 16) {
    run(Tiny{});
  } else if (k <= 32) {
    if (small <= time(Narrow{}, kNarrow)) run(Small{});
    else run(Narrow{});
  } else {
    if (small <= time(Wide{}, kWide)) run(Small{});
    else run(Wide{});
  }
}

}  // namespace sma
