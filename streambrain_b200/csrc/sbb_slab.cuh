// Copies of the operand slabs of the contraction kernels into shared memory (cp.async).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sbb {

// One copy into shared memory; not valid: nothing is read, the destination is filled with zeros.
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, bool valid) {
  static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async copies 4, 8 or 16 bytes");
  const int bytes = valid ? BYTES : 0;
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(bytes), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A thread's share of the k-slabs of both operands: N copies of V elements per slab into the stage buffers, zero-filled
// outside the operands.  A is [K x Mdim] MN-major (element (k, m) at A[k*lda + m]) or, S::KMAJOR, [Mdim x K] (at
// A[m*lda + k]); B is [K x Ndim] MN-major; the shape S has the tile (BM x BN, slabs of BK), the block's THREADS and the row
// strides LDA and LDB of the buffers.  V > 1: all row starts and V-element chunks are 16-byte aligned (checked by the host).
// A thread's copies of one operand lie RA (RB) rows of its memory layout apart in the same column, so one pointer and one
// count of what is left per operand are all it keeps.
template <typename T, class S, int V>
struct Slab {
  static constexpr bool KMAJOR = S::KMAJOR;
  static constexpr int CA = (KMAJOR ? S::BK : S::BM) / V, CB = S::BN / V;   // copies per row
  static constexpr int RA = S::THREADS / CA, RB = S::THREADS / CB;          // rows per pass of the block
  static constexpr int NA = S::BM * S::BK / V / S::THREADS, N = NA + S::BK * S::BN / V / S::THREADS;
  static_assert(S::THREADS % CA == 0 && S::THREADS % CB == 0, "whole rows per pass");
  const T *pa, *pb;          // the first copy of the next slab
  long lda, ldb;
  uint32_t da, db;           // its place in stage 0
  int rows_a, left_a, left_b;   // rows of A at and below the first copy's (K-major); k left from the first copies on
  __device__ __forceinline__ Slab(const T *A, long lda_, const T *Bm, long ldb_, long m0, long Mdim, long n0, long Ndim,
                                  int kbeg, int kend, const T *As, const T *Bs)
      : lda(lda_), ldb(ldb_) {
    const int ra = threadIdx.x / CA, ca = threadIdx.x % CA * V, rb = threadIdx.x / CB, cb = threadIdx.x % CB * V;
    const long m = m0 + (KMAJOR ? ra : ca);
    pa = A + (KMAJOR ? m * lda + kbeg + ca : (long)(kbeg + ra) * lda + m);
    pb = Bm + (long)(kbeg + rb) * ldb + n0 + cb;
    rows_a = (int)min(Mdim - m, (long)S::BM);
    left_a = kend - kbeg - (KMAJOR ? ca : ra);
    if (!KMAJOR && m >= Mdim) left_a = 0;
    left_b = n0 + cb < Ndim ? kend - kbeg - rb : 0;
    da = (uint32_t)__cvta_generic_to_shared(As + ra * S::LDA + ca);
    db = (uint32_t)__cvta_generic_to_shared(Bs + rb * S::LDB + cb);
  }
  // Copy t of the next slab, into the stage that starts at element a (b) of the buffers.
  __device__ __forceinline__ void copy(int t, int a, int b, const T *A, const T *Bm) const {
    if (t < NA) {
      const bool ok = KMAJOR ? t * RA < rows_a && left_a > 0 : t * RA < left_a;
      cp_async<V * (int)sizeof(T)>(da + (uint32_t)(a + t * RA * S::LDA) * (uint32_t)sizeof(T), ok ? pa + t * RA * lda : A, ok);
    } else if (t < N) {
      const bool ok = (t - NA) * RB < left_b;
      cp_async<V * (int)sizeof(T)>(db + (uint32_t)(b + (t - NA) * RB * S::LDB) * (uint32_t)sizeof(T),
                                   ok ? pb + (t - NA) * RB * ldb : Bm, ok);
    }
  }
  __device__ __forceinline__ void advance() {
    pa += KMAJOR ? (long)S::BK : S::BK * lda;
    pb += S::BK * ldb;
    left_a -= S::BK;
    left_b -= S::BK;
  }
};

}  // namespace sbb
