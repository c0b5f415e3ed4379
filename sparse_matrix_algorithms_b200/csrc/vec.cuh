// Vector loads/stores of V consecutive elements, V*sizeof(T) = 4..32 bytes, each ONE access:
// a 32-byte vector is a 256-bit load or store (sm_100), so that a warp's request covers whole
// 128-byte lines -- two 16-byte halves at a 32-byte stride touch every line twice.  Read-only
// data goes through the non-coherent path; it is written only by earlier kernel launches.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

namespace sma {

// KEEP = false: the line is not kept in L1 (rows that one thread reads once)
template <bool KEEP, int BYTES>
__device__ __forceinline__ void ld_words(const void *p, unsigned (&w)[BYTES / 4]) {
  static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16 || BYTES == 32, "vector width");
  if constexpr (BYTES == 32) {
    if constexpr (KEEP)
      asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]),
            "=r"(w[7])
          : "l"(p));
    else
      asm("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
          : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]),
            "=r"(w[7])
          : "l"(p));
  } else if constexpr (BYTES == 16) {
    if constexpr (KEEP)
      asm("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];"
          : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p));
    else
      asm("ld.global.nc.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];"
          : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p));
  } else if constexpr (BYTES == 8) {
    if constexpr (KEEP) asm("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "l"(p));
    else
      asm("ld.global.nc.L1::no_allocate.v2.b32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "l"(p));
  } else {
    if constexpr (KEEP) asm("ld.global.nc.b32 %0, [%1];" : "=r"(w[0]) : "l"(p));
    else asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(w[0]) : "l"(p));
  }
}

template <typename T, int V, bool KEEP = true>
__device__ __forceinline__ void ldv(const T *__restrict__ p, T (&f)[V]) {
  unsigned w[V * sizeof(T) / 4];
  ld_words<KEEP, V * (int)sizeof(T)>(p, w);
  memcpy(f, w, sizeof(w));
}

// An index through which every address after the wait for the previous kernel is formed: ties the
// loads there, which the compiler could otherwise hoist past the wait.
__device__ __forceinline__ uint32_t after_wait(uint32_t i) {
  asm volatile("" : "+r"(i)::"memory");
  return i;
}
__device__ __forceinline__ int64_t after_wait(int64_t i) {
  asm volatile("" : "+l"(i)::"memory");
  return i;
}

// ldv where ok, else zeros: the access itself is predicated, nothing branches.
template <typename T, int V>
__device__ __forceinline__ void ldv_if(bool ok, const T *__restrict__ p, T (&f)[V]) {
  constexpr int kBytes = V * (int)sizeof(T);
  unsigned w[kBytes / 4];
#pragma unroll
  for (int i = 0; i < kBytes / 4; ++i) w[i] = 0u;
  if constexpr (kBytes == 32)
    asm("{\n .reg .pred p;\n setp.ne.u32 p, %9, 0;\n"
        " @p ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n}"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]),
          "+r"(w[7])
        : "l"(p), "r"((unsigned)ok));
  else if constexpr (kBytes == 16)
    asm("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n"
        " @p ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];\n}"
        : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]) : "l"(p), "r"((unsigned)ok));
  else if constexpr (kBytes == 8)
    asm("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p ld.global.nc.v2.b32 {%0, %1}, [%2];\n}"
        : "+r"(w[0]), "+r"(w[1]) : "l"(p), "r"((unsigned)ok));
  else
    asm("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p ld.global.nc.b32 %0, [%1];\n}"
        : "+r"(w[0]) : "l"(p), "r"((unsigned)ok));
  memcpy(f, w, sizeof(w));
}

template <typename T, int V>
__device__ __forceinline__ void stv(T *__restrict__ p, const T (&f)[V]) {
  constexpr int kBytes = V * (int)sizeof(T);
  unsigned w[kBytes / 4];
  memcpy(w, f, sizeof(w));
  if constexpr (kBytes == 32)
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]),
                 "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  else if constexpr (kBytes == 16)
    asm volatile("st.global.v4.b32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(w[0]), "r"(w[1]),
                 "r"(w[2]), "r"(w[3]) : "memory");
  else if constexpr (kBytes == 8)
    asm volatile("st.global.v2.b32 [%0], {%1, %2};" ::"l"(p), "r"(w[0]), "r"(w[1]) : "memory");
  else
    asm volatile("st.global.b32 [%0], %1;" ::"l"(p), "r"(w[0]) : "memory");
}

// Brings the line into L2 without holding a register for it.
__device__ __forceinline__ void prefetch_l2(const void *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Programmatic dependent launch: wait until the grids this one depends on have completed and
// their writes are visible; let the next grid in the stream be scheduled.  The second always
// comes AFTER the first: a grid then starts while its predecessor runs, but never while its
// predecessor's predecessor still does, so no cache line that an older step read into L1 can
// outlive the write that replaced it.  Launched without the attribute both are no-ops.
__device__ __forceinline__ void pdl_wait_then_trigger() {
  asm volatile("griddepcontrol.wait;\n griddepcontrol.launch_dependents;" ::: "memory");
}

// Round-to-nearest products and sums that the compiler never contracts into FMAs.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

// One element of a Clenshaw step's epilogue, ck*q + alpha*acc + beta*s - t, evaluated left
// to right as the reference's broadcast TMP .= c_k .* Q .+ alpha .* AX .+ beta .* B1 .- B2
// (chebyshev_subspace_iteration.jl:576-580) with every product and sum rounded on its own.
// Left to the compiler, ck*q + alpha*acc may be fused either way round into an FMA, and
// different kernels would then round differently; with this form every kernel that takes a
// step -- CSR, segmented, stencil, persistent, matrix-free axpy -- writes the same bits.
// HQ, HS, HB: whether the q, s and t terms are present.
template <bool HQ, bool HS, bool HB, typename T>
__device__ __forceinline__ T clenshaw_combine(T acc, T q, T s, T t, T ck, T alpha, T beta) {
  T x = mul_rn(alpha, acc);
  if constexpr (HQ) x = add_rn(mul_rn(ck, q), x);
  if constexpr (HS) x = add_rn(x, mul_rn(beta, s));
  if constexpr (HB) x = sub_rn(x, t);
  return x;
}

}  // namespace sma
