// General-shape CUDA kernels of the BCPNN layer train step (float and double).
//
// These are the contractions for any N, M, B (odd sizes, unaligned rows) and for
// float64, and the softmax, the column vectors and the element-wise kernels of
// every path.  The tcgen05 tile kernels for aligned float32 shapes, the kernels
// for layers of few units or forward passes of few samples, and the mask update
// have files of their own.
//
// Data layout: every matrix is row-major and contiguous.  x[B,N], y[B,M],
// weights/Cij[N,M], wmask[N,H] bytes.  Both contractions of the step read their
// operands "MN-major" (contiguous along the output dimension) except the forward
// product's x, which is contiguous along the reduction dimension in memory and in
// shared memory alike.
#include "sbb_kernels.cuh"
#include "sbb_f64_mma.cuh"
#include "sbb_launch.cuh"
#include "sbb_math.cuh"
#include "sbb_tc_ptx.cuh"

#include <atomic>
#include <math.h>
#include <stdlib.h>
#include <string.h>

namespace sbb {

static std::atomic<unsigned long long> g_launches{0};
unsigned long long kernel_launches() { return g_launches.load(); }
void count_launches(int n) { g_launches += (unsigned long long)n; }
static inline cudaError_t launched(int n = 1) {
  g_launches += (unsigned long long)n;
  return cudaGetLastError();
}

template <typename T>
TraceParams<T> make_trace_params(double taupdt, double cthr, long batch) {
  TraceParams<T> p;
  p.taupdt = (T)taupdt;
  // The reference forms (1.0 - taupdt) in double from the REAL-rounded taupdt and
  // rounds the result to REAL (kernels_openmp_internal.cc:101).
  p.one_minus = (T)(1.0 - (double)p.taupdt);
  p.batch = (T)batch;
  p.cthr = (T)cthr;
  p.cthr4 = p.cthr * p.cthr * p.cthr * p.cthr;
  return p;
}
template TraceParams<float> make_trace_params<float>(double, double, long);
template TraceParams<double> make_trace_params<double>(double, double, long);

// ----------------------------------------------------------------------------
// 16-byte vector helpers.
// ----------------------------------------------------------------------------
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  using type = float4;
  static constexpr int N = 4;
};
template <>
struct Vec16<double> {
  using type = double2;
  static constexpr int N = 2;
};

__device__ __forceinline__ void unpack(const float4 &v, float *r) {
  r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
}
__device__ __forceinline__ void unpack(const double2 &v, double *r) {
  r[0] = v.x; r[1] = v.y;
}
__device__ __forceinline__ float4 pack(const float *r) { return make_float4(r[0], r[1], r[2], r[3]); }
__device__ __forceinline__ double2 pack(const double *r) { return make_double2(r[0], r[1]); }

// Four consecutive elements from / to memory.  `vec` says the address is 16-byte
// aligned and all four are in range; otherwise `valid` (1..4) elements are touched.
__device__ __forceinline__ void load4(const float *p, float *r, bool vec, int valid) {
  if (vec && valid == 4) {
    unpack(*reinterpret_cast<const float4 *>(p), r);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = c < valid ? p[c] : 0.f;
  }
}
__device__ __forceinline__ void load4(const double *p, double *r, bool vec, int valid) {
  if (vec && valid == 4) {
    unpack(*reinterpret_cast<const double2 *>(p), r);
    unpack(*reinterpret_cast<const double2 *>(p + 2), r + 2);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = c < valid ? p[c] : 0.0;
  }
}
__device__ __forceinline__ void store4(float *p, const float *r, bool vec, int valid) {
  if (vec && valid == 4) {
    *reinterpret_cast<float4 *>(p) = pack(r);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < valid) p[c] = r[c];
  }
}
__device__ __forceinline__ void store4(double *p, const double *r, bool vec, int valid) {
  if (vec && valid == 4) {
    *reinterpret_cast<double2 *>(p) = pack(r);
    *reinterpret_cast<double2 *>(p + 2) = pack(r + 2);
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (c < valid) p[c] = r[c];
  }
}

static inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ----------------------------------------------------------------------------
// Tiled float32 contraction: C[Mdim, Ndim] = A^T-or-A * B over k in [k0, k1), on the FMA pipe; it serves rows that the
// tensor-core kernels' copies cannot address.  128 x 128 output tile per 256-thread CTA, 8 x 8 micro-tile per thread split
// into two 4-wide halves in each dimension (rows ty*4+r and 64+ty*4+r; columns tx*4+c and 64+tx*4+c) so shared-memory reads
// are conflict-free 16-byte loads and global stores are 16 bytes per thread, 256 contiguous bytes per half-warp.  The slabs
// arrive by cp.async, three of four stages in flight, and the multiplications are the two-wide FMA (two columns; each half
// rounds like a single FMA): one issue slot for two leaves the others to the operand reads and copies.
// 1001 x 6001 -> 2257, odd rows: forward 690 -> 586 us, trace 778 -> 570 us against register-staged slabs (46 TFLOP/s; a
// warp of 4 x 8 threads, which halves the shared-memory passes, changes nothing).
// ----------------------------------------------------------------------------
struct Tile {
  static constexpr int BM = 128, BN = 128, BK = 16, THREADS = 256, STAGES = 4;
  static constexpr int LDA_K = BK + 4, LDA_M = BM + 4, LDB = BN + 4;
  static constexpr int A_STAGE = BM * LDA_K > BK * LDA_M ? BM * LDA_K : BK * LDA_M, B_STAGE = BK * LDB;
  static constexpr size_t SMEM_BYTES = (size_t)STAGES * (A_STAGE + B_STAGE) * sizeof(float);
};
template <bool A_KMAJOR>
struct TileShape : Tile {
  static constexpr bool KMAJOR = A_KMAJOR;
  static constexpr int LDA = A_KMAJOR ? LDA_K : LDA_M;
};

__device__ __forceinline__ void lds4(const float *p, float *r) { unpack(*reinterpret_cast<const float4 *>(p), r); }
__device__ __forceinline__ void lds4(const double *p, double *r) {
  unpack(*reinterpret_cast<const double2 *>(p), r);
  unpack(*reinterpret_cast<const double2 *>(p + 2), r + 2);
}

// Row / column of micro-tile entry e (0..7) inside the 128-wide tile.
__device__ __forceinline__ int micro_index(int t, int e) { return (e < 4 ? 0 : 64) + t * 4 + (e & 3); }

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo);
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// grid.x = row tiles of the output, grid.y = column tiles (swapped when cols_fastest: the fastest dimension walks the tiles
// that share the larger re-used operand), grid.z = k-splits.  k-split z covers [z*kper, min(K,(z+1)*kper)), kper a multiple
// of the slab depth.
template <bool A_KMAJOR, int V, class Epilogue>
__global__ void __launch_bounds__(Tile::THREADS, 2)
    contraction_kernel(const float *__restrict__ A, long lda, const float *__restrict__ Bm, long ldb, long Mdim, long Ndim,
                       int K, int kper, bool cols_fastest, Epilogue ep) {
  after_previous();
  using S = TileShape<A_KMAJOR>;
  using L = Slab<float, S, V>;
  extern __shared__ __align__(16) float tile_smem[];
  float *As = tile_smem, *Bs = tile_smem + S::STAGES * S::A_STAGE;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const long m0 = (long)(cols_fastest ? blockIdx.y : blockIdx.x) * S::BM;
  const long n0 = (long)(cols_fastest ? blockIdx.x : blockIdx.y) * S::BN;
  const int kbeg = blockIdx.z * kper;
  const int kend = min(K, kbeg + kper);
  const int nk = kend > kbeg ? (kend - kbeg + S::BK - 1) / S::BK : 0;
  L slab(A, lda, Bm, ldb, m0, Mdim, n0, Ndim, kbeg, kend, As, Bs);
#pragma unroll
  for (int s = 0; s < S::STAGES - 1; ++s) {
#pragma unroll
    for (int c = 0; c < L::N; ++c) slab.copy(c, s * S::A_STAGE, s * S::B_STAGE, A, Bm);
    slab.advance();
    cp_async_commit();
  }
  uint64_t acc[8][4];   // pairs of neighbouring columns
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0;
  int cur = 0, fill = S::STAGES - 1;
#pragma unroll 1
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<S::STAGES - 2>();   // slab kt has landed (for this thread's copies; the barrier covers the others')
    __syncthreads();                  // ... and everyone has finished with the stage refilled below
    const float *as = As + cur * S::A_STAGE, *bs = Bs + cur * S::B_STAGE;
    constexpr int PER_STEP = (L::N + S::BK / 2 - 1) / (S::BK / 2);
#pragma unroll
    for (int k2 = 0; k2 < S::BK; k2 += 2) {
      float a[2][8];
      if constexpr (A_KMAJOR) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float2 v = *reinterpret_cast<const float2 *>(as + micro_index(ty, r) * S::LDA + k2);
          a[0][r] = v.x;
          a[1][r] = v.y;
        }
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if constexpr (!A_KMAJOR) {
          lds4(as + (k2 + k) * S::LDA + ty * 4, a[k]);
          lds4(as + (k2 + k) * S::LDA + 64 + ty * 4, a[k] + 4);
        }
        uint64_t b[4];
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(bs + (k2 + k) * S::LDB + tx * 4);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2 *>(bs + (k2 + k) * S::LDB + 64 + tx * 4);
        b[0] = b0.x, b[1] = b0.y, b[2] = b1.x, b[3] = b1.y;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const uint64_t aa = pack2(a[k][r], a[k][r]);
#pragma unroll
          for (int c = 0; c < 4; ++c) fma2(acc[r][c], aa, b[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < PER_STEP; ++c)   // a few of a later slab's copies between the multiplications
        slab.copy(k2 / 2 * PER_STEP + c, fill * S::A_STAGE, fill * S::B_STAGE, A, Bm);
    }
    slab.advance();
    cp_async_commit();
    fill = cur;
    cur = cur + 1 < S::STAGES ? cur + 1 : 0;
  }
  cp_async_wait<0>();
  float out[8][8];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      out[r][2 * c] = __uint_as_float((uint32_t)acc[r][c]);
      out[r][2 * c + 1] = __uint_as_float((uint32_t)(acc[r][c] >> 32));
    }
  ep(out, m0, n0, ty, tx, (int)blockIdx.z);
}

// The same contraction for float32 outputs of few 128 x 128 tiles: a 32 x 64 tile per CTA of four warps, each 8 rows x 64
// columns (a lane owns columns lane and lane + 32, so every global access of a warp is 32 neighbouring elements whatever the
// row length, and its reads of A are broadcasts).  Such launches are bound by latency and by the SMs they leave idle, not by
// arithmetic: the slabs arrive by 4-byte cp.async (any alignment) with three of four stages in flight, and what the epilogue
// reads is requested before the main loop.  Each output is the same chain of FMAs over ascending k as in the kernel above.
// (In float64 it is what SBB_F64_CONTRACTION=dfma runs, with the general epilogue's division and library logarithm, to
// compare the FP64 tensor-core kernels with: 1568 -> 30 x 100 at batch 128, forward pass 82 us against 43, train step without
// a mask update 142 against 70.)
// ROWS: rows of a warp.  Eight; four, and twice the warps, in trace steps that leave the schedulers idle, up to two blocks to an SM,
// or four and few slabs (an element's logarithm and division are some hundred dependent instructions, and a thread has two of
// them per row): 1001 x 481 at batch 97 13.2 -> 10.7 us, 1211 x 39 at 40 8.0 -> 5.6, 231 x 3108 at 47 (392 blocks) 11.2 -> 9.5; 1843 x 424 at
// 5485 (406 blocks) 328 -> 372, so not there.  The forward product gains nothing (9.1 and 9.4).
template <typename T, bool A_KMAJOR, int ROWS>
struct SmallShape {
  static constexpr bool KMAJOR = A_KMAJOR;
  static constexpr int BM = 32, BN = 64, BK = 32, STAGES = 4, THREADS = 32 / ROWS * 32;
  static constexpr int LDA = 32 + 4, LDB = BN;   // K-major A as [m][k], MN-major as [k][m]: 16-byte rows
  static constexpr int A_STAGE = 32 * LDA, B_STAGE = BK * LDB;
  static constexpr size_t SMEM_BYTES = (size_t)STAGES * (A_STAGE + B_STAGE) * sizeof(T);
};

// grid.x = column tiles, grid.y = row tiles, grid.z = k-splits
template <typename T, bool A_KMAJOR, int ROWS, class Epilogue>
__global__ void __launch_bounds__(SmallShape<T, A_KMAJOR, ROWS>::THREADS)
    small_contraction_kernel(const T *__restrict__ A, long lda, const T *__restrict__ Bm, long ldb, long Mdim, long Ndim, int K,
                             int kper, Epilogue ep) {
  after_previous();
  using S = SmallShape<T, A_KMAJOR, ROWS>;
  using L = Slab<T, S, 1>;
  extern __shared__ __align__(16) unsigned char small_smem[];
  T *As = reinterpret_cast<T *>(small_smem), *Bs = As + S::STAGES * S::A_STAGE;
  const int w8 = (threadIdx.x >> 5) * ROWS, lane = threadIdx.x & 31;
  const long m0 = (long)blockIdx.y * S::BM, n0 = (long)blockIdx.x * S::BN;
  const int kbeg = blockIdx.z * kper;
  const int kend = min(K, kbeg + kper);
  const int nk = kend > kbeg ? (kend - kbeg + S::BK - 1) / S::BK : 0;
  L slab(A, lda, Bm, ldb, m0, Mdim, n0, Ndim, kbeg, kend, As, Bs);
#pragma unroll
  for (int s = 0; s < S::STAGES - 1; ++s) {
    if (s < nk) {
#pragma unroll
      for (int c = 0; c < L::N; ++c) slab.copy(c, s * S::A_STAGE, s * S::B_STAGE, A, Bm);
      slab.advance();
    }
    cp_async_commit();
  }
  typename Epilogue::template Strip<ROWS> strip(ep, m0 + w8, n0 + lane, lane);
  T acc[ROWS][2];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r][0] = acc[r][1] = (T)0;
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<S::STAGES - 2>();   // slab kt has landed
    __syncthreads();                  // ... for every thread, and the stage refilled below is free
    const int nx = kt + S::STAGES - 1;
    if (nx < nk) {
#pragma unroll
      for (int c = 0; c < L::N; ++c)
        slab.copy(c, nx % S::STAGES * S::A_STAGE, nx % S::STAGES * S::B_STAGE, A, Bm);
      slab.advance();
    }
    cp_async_commit();
    const T *as = As + kt % S::STAGES * S::A_STAGE, *bs = Bs + kt % S::STAGES * S::B_STAGE + lane;
#pragma unroll
    for (int k4 = 0; k4 < S::BK; k4 += 4) {
      T a[ROWS][4];   // [row][k]
      if constexpr (A_KMAJOR) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) lds4(as + (w8 + r) * S::LDA + k4, a[r]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          T v[ROWS];
#pragma unroll
          for (int r = 0; r < ROWS; r += 4) lds4(as + (k4 + k) * S::LDA + w8 + r, v + r);
#pragma unroll
          for (int r = 0; r < ROWS; ++r) a[r][k] = v[r];
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const T b0 = bs[(k4 + k) * S::LDB], b1 = bs[(k4 + k) * S::LDB + 32];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          acc[r][0] = fma(a[r][k], b0, acc[r][0]);
          acc[r][1] = fma(a[r][k], b1, acc[r][1]);
        }
      }
    }
  }
  cp_async_wait<0>();
  strip.finish(ep, acc, m0 + w8, n0 + lane, (int)blockIdx.z);
}

// Epilogue: partial[z, m, n] = acc  (forward product) or delta[m, n] = acc.
template <typename T>
struct StoreEpilogue {
  T *out;
  long rows, cols;   // logical extent of one [rows, cols] slice
  long ld;           // row stride of out
  long zstride;      // elements between k-split slices
  bool vec;
  // The micro-tiles of the large-tile kernel.
  __device__ __forceinline__ void operator()(T (&acc)[8][8], long m0, long n0, int ty, int tx, int z) const {
    T *base = out + (long)z * zstride;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const long m = m0 + micro_index(ty, r);
      if (m >= rows) continue;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const long n = n0 + g * 64 + tx * 4;
        const long left = cols - n;
        if (left <= 0) continue;
        store4(base + m * ld + n, &acc[r][g * 4], vec, left >= 4 ? 4 : (int)left);
      }
    }
  }
  // ROWS rows from m on, columns n and n + 32 of the small-tile kernel.
  template <int ROWS>
  struct Strip {
    __device__ __forceinline__ Strip(const StoreEpilogue &, long, long, int) {}
    __device__ __forceinline__ void finish(const StoreEpilogue &e, T (&acc)[ROWS][2], long m, long n, int z) const {
      T *p = e.out + (long)z * e.zstride + m * e.ld + n;
#pragma unroll
      for (int r = 0; r < ROWS; ++r, p += e.ld) {
        if (m + r < e.rows && n < e.cols) p[0] = acc[r][0];
        if (m + r < e.rows && n + 32 < e.cols) p[32] = acc[r][1];
      }
    }
  };
};

// Epilogue of the fused trace step: moving average of Cij, log-ratio weight,
// threshold and mask zeroing.  Each Cij element is read once and written once.
template <typename T>
struct TraceEpilogue {
  const T *Ci;
  const T *Cj;
  T *Cij;
  T *W;
  const uint8_t *wmask;  // [N, H] or null
  long row0;             // global row of tile row 0
  long row_end;          // global row limit
  long M, H, Mc;
  TraceParams<T> p;
  bool vec;
  const T *rci, *rcj;    // reciprocals of Ci and Cj (float64 tensor-core kernel)
  __device__ __forceinline__ void operator()(T (&acc)[8][8], long m0, long n0, int ty, int tx, int) const {
    T cj[8];
    int hc[8];
    bool cj_low[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const long j = n0 + micro_index(tx, c);
      const bool in = j < M;
      cj[c] = in ? Cj[j] : (T)1;
      cj_low[c] = cj[c] < p.cthr;
      hc[c] = in ? (int)(j / Mc) : 0;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const long i = row0 + m0 + micro_index(ty, r);
      if (i >= row_end) continue;
      const T ci = Ci[i];
      const bool skip = ci < p.cthr;
      const uint8_t *mrow = wmask ? wmask + i * H : nullptr;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        constexpr int GW = 4;
        const long j = n0 + g * 64 + tx * 4;
        const long left = M - j;
        if (left <= 0) continue;
        const int valid = left >= GW ? GW : (int)left;
        T c4[GW], w4[GW];
        load4(Cij + i * M + j, c4, vec, valid);
#pragma unroll
        for (int c = 0; c < GW; ++c) {
          if (c < valid) {
            const T cij = trace_ema(c4[c], acc[r][g * GW + c], p);
            c4[c] = cij;
            T w = (T)0;
            if (!skip && !cj_low[g * GW + c] && (mrow == nullptr || mrow[hc[g * GW + c]] != 0))
              w = log_ratio(cij, ci, cj[g * GW + c], p.cthr4);
            w4[c] = w;
          }
        }
        store4(Cij + i * M + j, c4, vec, valid);
        store4(W + i * M + j, w4, vec, valid);
      }
    }
  }
  // ROWS rows from m on, columns n and n + 32 of the small-tile kernel: everything the epilogue reads is requested before the
  // main loop, and its arithmetic (the same as above) is one row at a time from one copy of the code, the rows rotating
  // through slot 0: unrolled, sixteen logarithms and divisions come from a cold instruction cache.
  template <int ROWS>
  struct Strip {
    T old[ROWS][2], ci, cj[2];   // ci: lane r holds row r's
    unsigned on = 0;          // bit 2 * r + c: the mask keeps the element's weight
    __device__ __forceinline__ Strip(const TraceEpilogue &e, long m, long n, int lane) {
      const long i0 = e.row0 + m, i = i0 + (lane & (ROWS - 1));
      ci = i < e.row_end ? e.Ci[i] : (T)0;
      const T *src = e.Cij + i0 * e.M + n;
      const uint8_t *mrow[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const long j = n + 32 * c < e.M ? n + 32 * c : 0;
        cj[c] = e.Cj[j];
        mrow[c] = e.wmask ? e.wmask + i0 * e.H + (unsigned)j / (unsigned)e.Mc : nullptr;
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r, src += e.M)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const bool in = i0 + r < e.row_end && n + 32 * c < e.M;
          old[r][c] = in ? src[32 * c] : (T)0;
          if (in && (mrow[c] == nullptr || mrow[c][r * e.H] != 0)) on |= 1u << (2 * r + c);
        }
    }
    __device__ __forceinline__ void finish(const TraceEpilogue &e, T (&acc)[ROWS][2], long m, long n, int) {
      const long i0 = e.row0 + m;
      const int rows = (int)min((long)ROWS, e.row_end - i0);
      T *pc = e.Cij + i0 * e.M + n, *pw = e.W + i0 * e.M + n;
#pragma unroll 1
      for (int r = 0; r < rows; ++r, pc += e.M, pw += e.M) {
        const T row = __shfl_sync(0xffffffffu, ci, r);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (n + 32 * c < e.M) {
            const T cij = trace_ema(old[0][c], acc[0][c], e.p);
            T w = (T)0;
            if (!(row < e.p.cthr) && !(cj[c] < e.p.cthr) && (on >> (2 * r + c) & 1u)) w = log_ratio(cij, row, cj[c], e.p.cthr4);
            pc[32 * c] = cij;
            pw[32 * c] = w;
          }
#pragma unroll
          for (int k = 0; k < ROWS - 1; ++k) {
            acc[k][c] = acc[k + 1][c];
            old[k][c] = old[k + 1][c];
          }
        }
      }
    }
  };
};

// ----------------------------------------------------------------------------
// float64 on the FP64 tensor-core instruction (sbb_f64_mma.cuh): the same two epilogues, fed with the
// accumulator pairs of the mma.sync fragment layout (element (m, n) and (m, n + 1), n even).
// ----------------------------------------------------------------------------
struct StorePairs {
  static constexpr bool LATE = false;
  double *out;
  long rows, cols, ld, zstride;
  bool vec;
  __device__ __forceinline__ void prefetch(long, long, int) const {}
  __device__ __forceinline__ void tile(const double (&acc)[4][4][2], long m_first, long n_first, int z) const {
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      const long m = m_first + mi * 8;
      if (m >= rows) continue;
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const long n = n_first + ni * 8;
        if (n >= cols) continue;
        double *p = out + (long)z * zstride + m * ld + n;
        if (vec) {
          *reinterpret_cast<double2 *>(p) = make_double2(acc[mi][ni][0], acc[mi][ni][1]);   // cols is even
        } else {
          p[0] = acc[mi][ni][0];
          if (n + 1 < cols) p[1] = acc[mi][ni][1];
        }
      }
    }
  }
};

// The fused trace epilogue on accumulator pairs.  Its memory accesses are what it waits for, so they are arranged in two
// phases: first every load the thread needs (its 16 pairs of the old trace, the mask bytes, the reciprocals of Ci and Cj;
// the trace block was requested into L2 before the main loop), folded into the accumulators as they arrive; then the
// arithmetic and the stores.  With a load, a logarithm and two stores per pair in turn, the sixteen dependent memory round
// trips per thread left the tensor pipe idle half of the time.  The second phase is one row of the thread's block at a time
// from one copy of the code (the accumulators rotate): unrolled it was 32 logarithms long and ran from a cold instruction
// cache.  1568 x 3000, batch 128: 96 us with that, a 64-bit division per column and a float64 division per row and column.
struct TracePairs {
  static constexpr bool LATE = true;   // that kernel is column_vectors_kernel, which writes the reciprocals, or a copy of old traces
  const double *rci, *rcj;   // reciprocals of Ci and Cj, 0 below the threshold
  double *Cij, *W;
  const uint8_t *wmask;
  long row0, row_end, M, H, Mc;
  TraceParams<double> p;
  double inv_batch;
  bool vec;
  __device__ __forceinline__ void prefetch(long m_warp, long n_warp, int lane) const {
    // the warp's 32 x 32 block of Cij: 256 bytes per row, two 128-byte lines, one request per line
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int line = lane + 32 * k;
      const long i = row0 + m_warp + (line >> 1), n = n_warp + (line & 1) * 16;
      if (i < row_end && n < M) asm volatile("prefetch.global.L2 [%0];" ::"l"(Cij + i * M + n));
    }
  }
  __device__ __forceinline__ void tile(double (&acc)[4][4][2], long m_first, long n_first, int) const {
    // ---- phase 1: loads
    double rj[4][2], ri[4];
    unsigned on = 0;   // bit 8*mi + 2*ni + e: the element keeps a weight (row, column and mask allow it)
    unsigned col_on = 0, second = 0;   // bit 2*ni + e: column at or above the threshold; in the second hypercolumn
    const unsigned mc = (unsigned)Mc, last = (unsigned)(M - 1);
    const unsigned h0 = min((unsigned)n_first, last) / mc, next = (h0 + 1) * mc;
    bool two = true;   // the thread's columns (25 apart at most) lie in two hypercolumns
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const long j = n_first + ni * 8 + e;
        rj[ni][e] = j < M ? __ldg(rcj + j) : 0.0;
        if ((unsigned)j >= next) second |= 1u << (2 * ni + e);
        if (j < M && (unsigned)j >= next + mc) two = false;
      }
    }
    const unsigned h1 = h0 + 1 < (unsigned)H ? h0 + 1 : h0;
    uint8_t m0[4], m1[4];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      const long i = row0 + m_first + mi * 8;
      const bool in = i < row_end;
      ri[mi] = in ? __ldg(rci + i) : 0.0;
      m0[mi] = wmask == nullptr ? 1 : (in ? wmask[i * H + h0] : 0);
      m1[mi] = wmask == nullptr ? 1 : (in ? wmask[i * H + h1] : 0);
    }
    const double scale = inv_batch * p.taupdt;
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      const long i = row0 + m_first + mi * 8;
      const bool row_in = i < row_end;
      double2 old[4];
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const long n = n_first + ni * 8;
        old[ni] = make_double2(0.0, 0.0);
        if (row_in && n < M) {
          const double *cp = Cij + i * M + n;
          if (vec) old[ni] = *reinterpret_cast<const double2 *>(cp);
          else old[ni] = make_double2(cp[0], n + 1 < M ? cp[1] : 0.0);
        }
      }
      // the moving average, with the batch mean and the averaging weight folded into one factor (the reciprocal
      // of the batch size is exact for powers of two, one rounding more otherwise); a NaN clamps to zero
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const double a0 = fma(old[ni].x, p.one_minus, acc[mi][ni][0] * scale);
        const double a1 = fma(old[ni].y, p.one_minus, acc[mi][ni][1] * scale);
        acc[mi][ni][0] = a0 > 0.0 ? a0 : 0.0;
        acc[mi][ni][1] = a1 > 0.0 ? a1 : 0.0;
      }
    }
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (rj[ni][e] != 0.0) col_on |= 1u << (2 * ni + e);
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      unsigned row = (m0[mi] != 0 ? ~second : 0u) | (m1[mi] != 0 ? second : 0u);
      if (!two) {   // hypercolumns narrower than the thread's columns: every byte
        row = 0;
        const long i = row0 + m_first + mi * 8;
        if (i < row_end) {
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const unsigned j = (unsigned)(n_first + ni * 8 + e);
              if (j <= last && (wmask == nullptr || wmask[i * H + j / mc] != 0)) row |= 1u << (2 * ni + e);
            }
        }
      }
      if (ri[mi] != 0.0) on |= (row & col_on & 0xFFu) << (8 * mi);
    }
    // ---- phase 2: weights and stores, a row of the block at a time.  Cij / (Ci * Cj) by the reciprocals: three roundings
    // more than the division, a few 1e-16 on the weight.
#pragma unroll 1
    for (int mi = 0; mi < 4; ++mi) {
      const long i = row0 + m_first + mi * 8;
      if (i < row_end) {
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          const long n = n_first + ni * 8;
          if (n >= M) continue;
          const double n0 = acc[0][ni][0], n1 = acc[0][ni][1];
          double w0 = 0.0, w1 = 0.0;
          if (on & (1u << (2 * ni))) w0 = f64mma::log_positive((n0 < p.cthr4 ? p.cthr4 : n0) * (ri[0] * rj[ni][0]));
          if (on & (2u << (2 * ni))) w1 = f64mma::log_positive((n1 < p.cthr4 ? p.cthr4 : n1) * (ri[0] * rj[ni][1]));
          double *cp = Cij + i * M + n, *wp = W + i * M + n;
          if (vec) {
            *reinterpret_cast<double2 *>(cp) = make_double2(n0, n1);
            *reinterpret_cast<double2 *>(wp) = make_double2(w0, w1);
          } else {
            cp[0] = n0;
            wp[0] = w0;
            if (n + 1 < M) {
              cp[1] = n1;
              wp[1] = w1;
            }
          }
        }
      }
      on >>= 8;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        ri[q] = ri[q + 1];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          acc[q][ni][0] = acc[q + 1][ni][0];
          acc[q][ni][1] = acc[q + 1][ni][1];
        }
      }
    }
  }
};

static StorePairs to_pairs(const StoreEpilogue<double> &e) { return StorePairs{e.out, e.rows, e.cols, e.ld, e.zstride, e.vec}; }
static TracePairs to_pairs(const TraceEpilogue<double> &e) {
  TracePairs t{};
  t.rci = e.rci;
  t.rcj = e.rcj;
  t.Cij = e.Cij;
  t.W = e.W;
  t.wmask = e.wmask;
  t.row0 = e.row0;
  t.row_end = e.row_end;
  t.M = e.M;
  t.H = e.H;
  t.Mc = e.Mc;
  t.p = e.p;
  t.inv_batch = 1.0 / e.p.batch;
  t.vec = e.vec;
  return t;
}


constexpr size_t kMostSmem = 232448;   // of one block; an SM has 1 KB more, and every block takes 1 KB besides its own

// Dynamic shared memory to ask for, so that no SM gets more blocks than an even spread over the SMs gives it: blocks are
// placed while the kernel before still runs on some of them (programmatic launches), and with room for two or more on an SM
// some got two while others got none.  float64 trace step 2048 -> 8 x 64 at batch 1024, 128 blocks: 86 or 156 us, by the device
// and the state of the SMs, without it; 86 with it.
static size_t spread_smem(size_t own, long blocks) {
  const long sms = sm_count(), per = (blocks + sms - 1) / sms;
  if (per < 1 || per > 8) return own;
  const size_t least = ((kMostSmem + 1024) / (size_t)(per + 1) - 1024) / 128 * 128 + 128;   // (no more than that: other kernels' blocks
  return least > own ? least : own;                                                          // still fit beside them)
}

// More than 48 KB of dynamic shared memory is asked for once per kernel and device.
template <class K>
static cudaError_t allow_smem(K kernel, bool (&configured)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && configured[dev]) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
  if (e == cudaSuccess && dev >= 0 && dev < 64) configured[dev] = true;
  return e;
}

template <bool A_KMAJOR, int BM, bool DEEP, int V, class Pairs>
static cudaError_t launch_f64_mma_tiles(const double *A, long lda, const double *Bm, long ldb, long Mdim, long Ndim,
                                        int K, int splits, bool cols_fastest, Pairs ep, cudaStream_t st) {
  namespace F = f64mma;
  using C = F::Cfg<BM, DEEP>;
  auto kernel = F::contraction_kernel<A_KMAJOR, BM, DEEP, V, Pairs>;
  static bool configured[64] = {false};
  const cudaError_t e = allow_smem(kernel, configured);
  if (e != cudaSuccess) return e;
  const unsigned mt = (unsigned)((Mdim + BM - 1) / BM), nt = (unsigned)((Ndim + F::BN - 1) / F::BN);
  if (cols_fastest && mt > 65535u) cols_fastest = false;
  dim3 grid(cols_fastest ? nt : mt, cols_fastest ? mt : nt, (unsigned)splits);
  if (grid.y > 65535u || grid.z > 65535u) return cudaErrorInvalidConfiguration;
  const int slabs = (K + F::BK - 1) / F::BK;
  const int kper = (slabs + splits - 1) / splits * F::BK;
  launch_next(kernel, grid, C::THREADS, spread_smem(C::SMEM_BYTES, (long)mt * nt * splits), st, A, lda, Bm, ldb, Mdim, Ndim, K, kper, cols_fastest, ep);
  return launched();
}

// Row tiles of 128 unless the fullest SM has fewer rows to do in tiles of 64: 1568 x 3000 outputs are 611 tiles of 128
// rows, five on some SMs, or 1175 tiles of 64 rows, at most eight.  The forward product's tiles on as many SMs
// take the deep pipeline (the trace step's few-tile launches have one short chain of slabs, which it does not help).
template <bool A_KMAJOR, int V, class Pairs>
static cudaError_t launch_f64_mma(const double *A, long lda, const double *Bm, long ldb, long Mdim, long Ndim, int K,
                                  int splits, bool cols_fastest, Pairs ep, cudaStream_t st) {
  namespace F = f64mma;
  const long nt = (Ndim + F::BN - 1) / F::BN, sms = sm_count();
  auto ctas = [&](long bm) { return ((Mdim + bm - 1) / bm) * nt * splits; };
  auto rows = [&](long bm) { return (ctas(bm) + sms - 1) / sms * bm; };
  if (rows(64) < rows(128)) {
    if constexpr (A_KMAJOR) {
      if (ctas(64) <= sms)
        return launch_f64_mma_tiles<A_KMAJOR, 64, true, V>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, cols_fastest, ep, st);
    }
    return launch_f64_mma_tiles<A_KMAJOR, 64, false, V>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, cols_fastest, ep, st);
  }
  if constexpr (A_KMAJOR) {
    if (ctas(128) <= sms)
      return launch_f64_mma_tiles<A_KMAJOR, 128, true, V>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, cols_fastest, ep, st);
  }
  return launch_f64_mma_tiles<A_KMAJOR, 128, false, V>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, cols_fastest, ep, st);
}

// When the 32 x 64 tiles take over, in 128 x 128 tiles.  Forward products: below half an SM's worth; 28 tiles 18.5 -> 9.1
// us, but 92 tiles 19.0 -> 20.6.  And up to 64 samples (launch_contraction), of whose large tiles half or more is padding: 4999 x
// 2989 at batch 32 92 -> 42 us, at 64 93 -> 72, at 96 94 -> 105; 42265 x 150 74 -> 35, 75 -> 47, 76 -> 60.  Trace steps, whose epilogue is a logarithm and a division per output: below one per SM; 32
// tiles 35.6 -> 12.8 us, 96 tiles 36.5 -> 28.3, but 216 tiles 55.0 -> 54.7 at batch 97 and 125 -> 136 at batch 512.
static bool small_tiles(long tiles, bool forward) { return (forward ? 2 : 1) * tiles < sm_count(); }

template <typename T, bool A_KMAJOR, int ROWS, class Ep>
static cudaError_t launch_small_tiles(const T *A, long lda, const T *Bm, long ldb, long Mdim, long Ndim, int K,
                                            int splits, int kper, Ep ep, cudaStream_t st) {
  using S = SmallShape<T, A_KMAJOR, ROWS>;
  auto kernel = small_contraction_kernel<T, A_KMAJOR, ROWS, Ep>;
  static bool configured[64] = {false};
  const cudaError_t e = allow_smem(kernel, configured);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((Ndim + S::BN - 1) / S::BN), (unsigned)((Mdim + S::BM - 1) / S::BM), (unsigned)splits);
  if (grid.y > 65535u || grid.z > 65535u) return cudaErrorInvalidConfiguration;
  launch_next(kernel, grid, S::THREADS, spread_smem(S::SMEM_BYTES, (long)grid.x * grid.y * splits), st, A, lda, Bm, ldb, Mdim, Ndim, K, kper, ep);
  return launched();
}
template <typename T, bool A_KMAJOR, class Ep>
static cudaError_t launch_small_contraction(const T *A, long lda, const T *Bm, long ldb, long Mdim, long Ndim, int K,
                                            int splits, int kper, Ep ep, cudaStream_t st) {
  using S = SmallShape<T, A_KMAJOR, 8>;
  const long blocks = ((Ndim + S::BN - 1) / S::BN) * ((Mdim + S::BM - 1) / S::BM) * splits;
  if constexpr (!A_KMAJOR) {
    if (blocks <= 2 * sm_count() || (blocks <= 4 * sm_count() && K <= 512)) return launch_small_tiles<T, A_KMAJOR, 4>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, kper, ep, st);
  }
  return launch_small_tiles<T, A_KMAJOR, 8>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, kper, ep, st);
}

template <bool A_KMAJOR, int V, class Ep>
static cudaError_t launch_tiles(const float *A, long lda, const float *Bm, long ldb, long Mdim, long Ndim, int K,
                                int splits, int kper, bool cols_fastest, Ep ep, cudaStream_t st) {
  auto kernel = contraction_kernel<A_KMAJOR, V, Ep>;
  static bool configured[64] = {false};
  const cudaError_t e = allow_smem(kernel, configured);
  if (e != cudaSuccess) return e;
  const unsigned mt = (unsigned)((Mdim + 127) / 128), nt = (unsigned)((Ndim + 127) / 128);
  if (cols_fastest && mt > 65535u) cols_fastest = false;
  const dim3 grid(cols_fastest ? nt : mt, cols_fastest ? mt : nt, (unsigned)splits);
  if (grid.y > 65535u || grid.z > 65535u) return cudaErrorInvalidConfiguration;
  launch_next(kernel, grid, Tile::THREADS, spread_smem(Tile::SMEM_BYTES, (long)mt * nt * splits), st, A, lda, Bm, ldb, Mdim, Ndim, K, kper, cols_fastest, ep);
  return launched();
}

// SBB_F64_CONTRACTION=dfma keeps float64 off the FP64 tensor-core instruction (read once).
static bool f64_mma_enabled() {
  static const bool on = [] {
    const char *e = getenv("SBB_F64_CONTRACTION");
    return !(e != nullptr && strcmp(e, "dfma") == 0);
  }();
  return on;
}

template <typename T, bool A_KMAJOR, class Ep>
static cudaError_t launch_contraction(const T *A, long lda, const T *Bm, long ldb, long Mdim, long Ndim, int K,
                                      int splits, int kper, bool vec, bool cols_fastest, Ep ep, cudaStream_t st) {
  const long mt = (Mdim + 127) / 128, nt = (Ndim + 127) / 128;
  if (mt <= 0 || nt <= 0 || K <= 0) return cudaSuccess;
  // `vec`: every operand row starts on a 16-byte boundary and holds a whole number of 16-byte pieces
  if constexpr (std::is_same<T, double>::value) {
    if (!f64_mma_enabled() && Mdim <= 65535L * SmallShape<T, A_KMAJOR, 8>::BM)   // (its row tiles are grid.y)
      return launch_small_contraction<T, A_KMAJOR>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, kper, ep, st);
    if (vec && lda % 2 == 0 && ldb % 2 == 0)
      return launch_f64_mma<A_KMAJOR, 2>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, cols_fastest, to_pairs(ep), st);
    return launch_f64_mma<A_KMAJOR, 1>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, cols_fastest, to_pairs(ep), st);
  } else {
    if (small_tiles(mt * nt * splits, A_KMAJOR) || (A_KMAJOR && Mdim <= 64))
      return launch_small_contraction<T, A_KMAJOR>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, kper, ep, st);
    if (vec) return launch_tiles<A_KMAJOR, 4>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, kper, cols_fastest, ep, st);
    return launch_tiles<A_KMAJOR, 1>(A, lda, Bm, ldb, Mdim, Ndim, K, splits, kper, cols_fastest, ep, st);
  }
}

// ----------------------------------------------------------------------------
// Forward product (split over k so that small batches still fill the GPU).
// ----------------------------------------------------------------------------
int sm_count() {
  static std::atomic<int> known{0};
  int n = known.load(std::memory_order_relaxed);
  if (n == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
    known.store(n, std::memory_order_relaxed);
  }
  return n;
}

// k-splits of the forward product.  float32: output tiles of 128 x 128 until two CTAs per SM are busy, at least eight slabs
// each.  float64 (128 x 64 tiles, slabs of 16): the split whose fullest SM has the least to do, in slabs, counting each
// partial sum's way to memory and back (16 bytes per output at about 4 TB/s against about 1.05 us per slab of a tile, and
// two fifths of that for its turn in the sum); 47
// tiles of 98 slabs: three splits on 141 SMs, 33 slabs each, half of the partial sums that two CTAs per SM need for 34.
template <typename T>
int forward_splits(long B, long N, long M) {
  const long sms = sm_count();
  if (sizeof(T) == 8) {
    const long tiles = ((B + 127) / 128) * ((M + f64mma::BN - 1) / f64mma::BN), slabs = (N + f64mma::BK - 1) / f64mma::BK;
    const double per_split = (double)B * M / 262144.0 + 0.4;
    const long slots = B <= 64 ? 2 * sms : sms;   // batches of one 64-row tile: two of its four-warp CTAs keep an SM busy
    int best = 1;
    double least = 0;
    for (long s = 1; s <= 64 && (s == 1 || slabs / s >= 4); ++s) {
      const double cost = (double)((tiles * s + slots - 1) / slots) * ((slabs + s - 1) / s) + per_split * s;
      if (s == 1 || cost < least) least = cost, best = (int)s;
    }
    return best;
  }
  const long tiles = ((B + 127) / 128) * ((M + 127) / 128);
  const long want = 2 * sms;
  long s = tiles >= want ? 1 : want / (tiles > 0 ? tiles : 1);
  const long slabs = (N + Tile::BK - 1) / Tile::BK;
  const long max_s = slabs / 8 > 0 ? slabs / 8 : 1;
  if (s > max_s) s = max_s;
  if (s > 64) s = 64;
  if (s < 1) s = 1;
  return (int)s;
}
template int forward_splits<float>(long, long, long);
template int forward_splits<double>(long, long, long);

template <typename T>
cudaError_t launch_forward_product(const T *x, const T *w, T *partial, long B, long N, long M, int splits,
                                   cudaStream_t st) {
  constexpr int V = Vec16<T>::N;
  const long slabs = (N + Tile::BK - 1) / Tile::BK;
  const int kper = (int)((slabs + splits - 1) / splits) * Tile::BK;
  const bool vec = (N % V == 0) && (M % V == 0) && aligned16(x) && aligned16(w);
  StoreEpilogue<T> ep{partial, B, M, M, B * M, (M % V == 0) && aligned16(partial)};
  return launch_contraction<T, true>(x, N, w, M, B, M, (int)N, splits, kper, vec, false, ep, st);
}
template cudaError_t launch_forward_product<float>(const float *, const float *, float *, long, long, long, int,
                                                   cudaStream_t);
template cudaError_t launch_forward_product<double>(const double *, const double *, double *, long, long, long, int,
                                                    cudaStream_t);

// ----------------------------------------------------------------------------
// out = sum_s partial[s] + bias, then softmax per hypercolumn: one warp or part of a warp per (row, hypercolumn) group.
// ----------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T subwarp_max(T v, int width) {
  for (int off = width >> 1; off > 0; off >>= 1) {
    const T o = __shfl_xor_sync(0xffffffffu, v, off, width);
    v = o > v ? o : v;
  }
  return v;
}
template <typename T>
__device__ __forceinline__ T subwarp_sum(T v, int width) {
  for (int off = width >> 1; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off, width);
  return v;
}

// Groups of any size (what the kernels below do not take): a lane owns the entries sub, sub + width, ... of its group and keeps
// them in `out`.
template <typename T>
__global__ void __launch_bounds__(256)
    reduce_bias_softmax_kernel(const T *partial, int splits, long slice, const T *__restrict__ bias, T *out,
                               long groups, long H, long Mc, int width) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const int sub = lane % width;
  const long warp = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long g = warp * (32 / width) + lane / width;
  const bool live = g < groups;
  const long base = g * Mc;            // offset of the group inside [rows, H*Mc]
  const long col0 = (g % H) * Mc;      // first column of the group
  T mx = -INFINITY;
  if (live)
    for (long j = sub; j < Mc; j += width) {
      T s = partial[base + j];
      for (int z = 1; z < splits; ++z) s += partial[(long)z * slice + base + j];
      if (bias) s += bias[col0 + j];
      out[base + j] = s;
      mx = s > mx ? s : mx;
    }
  mx = subwarp_max(mx, width);
  T sum = (T)0;
  if (live)
    for (long j = sub; j < Mc; j += width) {
      const T e = sbb_exp(out[base + j] - mx);
      out[base + j] = e;
      sum += e;
    }
  sum = subwarp_sum(sum, width);
  if (live)
    for (long j = sub; j < Mc; j += width) out[base + j] = out[base + j] / sum;
}

// Softmax of a group of up to 32 * NC entries by one warp: lane l holds entries l, l + 32, ..., entry e of it exists when
// e < FULL or e * 32 < left (-inf otherwise), and dst points at its first one.
template <typename T, int NC, int FULL>
__device__ __forceinline__ void warp_softmax(T (&v)[NC], int left, T *dst) {
  if constexpr (sizeof(T) == 8) {
    T mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < NC; ++e) mx = v[e] > mx ? v[e] : mx;
    mx = subwarp_max(mx, 32);
    T sum = (T)0;
    // one copy of the float64 exponential (the entries rotate through slot 0): unrolled, a kernel of a few microseconds
    // spends most of them fetching instructions
#pragma unroll 1
    for (int e = 0; e < NC; ++e) {
      const T x = e * 32 < left ? sbb_exp(v[0] - mx) : (T)0;
      sum += x;
#pragma unroll
      for (int q = 0; q + 1 < NC; ++q) v[q] = v[q + 1];
      v[NC - 1] = x;
    }
    sum = subwarp_sum(sum, 32);
    const DivideBy<T> by(sum);
    // (128 samples, 784 -> 15 x 200: the forward pass takes 27.5 us, and 28.8 with a multiplication by 1 / sum, which rounds
    // once more than the division)
    bool covered = true;
#pragma unroll
    for (int e = 0; e < NC; ++e) covered = covered && by.covers(v[e]);
    if (!covered) {   // rare: one copy of the division, as of the exponential
#pragma unroll 1
      for (int e = 0; e < NC; ++e) {
        if (e * 32 < left) dst[e * 32] = v[0] / sum;
#pragma unroll
        for (int q = 0; q + 1 < NC; ++q) v[q] = v[q + 1];
      }
      return;
    }
#pragma unroll
    for (int e = 0; e < NC; ++e)
      if (e < FULL || e * 32 < left) dst[e * 32] = by.quotient(v[e]);
  } else {
    // What bounds the kernel in float32 is the issue of instructions, so each entry gets as few as it can: no test for the
    // entries that every lane has, the maximum of the lanes in one instruction, one test for all entries of whether the
    // short division covers them, and that division two entries at a time (100 groups of 300 at batch 1024: 520 instructions
    // a group of 300 and 68.0 us without these, 37.6 us so).
    float mx = -INFINITY;
#pragma unroll
    for (int e = 0; e < NC; ++e) mx = fmaxf(v[e], mx);   // (NaNs lose, and of -0 and 0 either will do)
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(mx) : "f"(mx));
    float sum = 0.f;
    uint32_t least = 0xffffffffu;   // of bits(v) - 1: zeros wrap to the top
#pragma unroll
    for (int e = 0; e < NC; ++e) {
      v[e] = e < FULL || e * 32 < left ? sbb_exp(v[e] - mx) : 0.f;
      sum += v[e];
      least = min(least, __float_as_uint(v[e]) - 1u);
    }
    sum = subwarp_sum(sum, 32);
    const DivideBy<float> by(sum);
    if (by.plain || least < __float_as_uint(DivideBy<float>::MIN) - 1u) {   // rare
#pragma unroll 1
      for (int e = 0; e < NC; ++e) {
        if (e * 32 < left) dst[e * 32] = by(v[0]);
#pragma unroll
        for (int q = 0; q + 1 < NC; ++q) v[q] = v[q + 1];
      }
      return;
    }
    const uint64_t y = pair_of(by.y, by.y), minus_d = pair_of(-by.d, -by.d);
#pragma unroll
    for (int e = 0; e < NC; e += 2) {
      const uint64_t p = pair_of(v[e], v[e + 1]), q = mul_pair(p, y);
      const float2 r = halves(fma_pair(fma_pair(q, minus_d, p), y, q));   // DivideBy::quotient
      if (e < FULL || e * 32 < left) dst[e * 32] = r.x;
      if (e + 1 < FULL || (e + 1) * 32 < left) dst[(e + 1) * 32] = r.y;
    }
  }
}

// The same for groups of more than 16 entries (one whole warp per group) with every per-element index a
// compile-time multiple of 32 from three pointers formed once: the general kernel above spends most of its
// instructions on 64-bit index arithmetic (about 100 per element at Mc = 300, which made it issue-bound: 183 us
// for 246 MB at the 1568 -> 100 x 300 layer at batch 1024; 37.6 us here, 6.5 TB/s).
template <typename T, int NC, int FULL, bool SPLIT>
__global__ void __launch_bounds__(256)
    softmax_warp_kernel(const T *partial, int splits, long slice, const T *__restrict__ bias, T *out, uint32_t groups,
                        uint32_t H, int Mc) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const uint32_t g = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (g >= groups) return;   // whole warps leave together
  const T *src = partial + (long)g * Mc + lane;
  const T *bs = bias ? bias + (long)(g % H) * Mc + lane : nullptr;
  T *dst = out + (long)g * Mc + lane;
  const int left = Mc - lane;   // entry e of this lane exists when e < FULL or e * 32 < left
  T v[NC];
  // (entries inside, partial sums outside: all entries' loads are in flight at once.  With the loops the other way round
  // each partial sum was a round trip to memory of its own: 11.2 us for 128 x 15 groups of 200 doubles in six partial
  // sums)
#pragma unroll
  for (int e = 0; e < NC; ++e) {
    v[e] = e < FULL || e * 32 < left ? src[e * 32] : -INFINITY;
    if (!SPLIT && bs && (e < FULL || e * 32 < left)) v[e] += bs[e * 32];
  }
  if (SPLIT) {
    if constexpr (sizeof(T) == 4) {
#pragma unroll 2
      for (int z = 1; z < splits; ++z) {
        const T *sz = src + (long)z * slice;
        T d[NC];
#pragma unroll
        for (int e = 0; e < NC; ++e) d[e] = e < FULL || e * 32 < left ? sz[e * 32] : (T)0;
#pragma unroll
        for (int e = 0; e < NC; ++e) v[e] += d[e];
      }
    } else {   // (more registers, for the many parts of a float64 batch; in float32, seven parts, a 1001 x 481 step took 45.7 us with them, 41.0 so)
      constexpr int AHEAD = NC <= 4 ? 8 : NC <= 12 ? 4 : 2;
      T d[AHEAD][NC];
#pragma unroll 1
      for (int z = 1; z < splits; z += AHEAD) {
        const T *sz = src + (long)z * slice;
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
#pragma unroll
          for (int e = 0; e < NC; ++e) d[a][e] = z + a < splits && (e < FULL || e * 32 < left) ? sz[a * slice + e * 32] : (T)0;
#pragma unroll
        for (int a = 0; a < AHEAD; ++a)
#pragma unroll
          for (int e = 0; e < NC; ++e) v[e] += d[a][e];
      }
    }
  }
  if (SPLIT && bs) {
#pragma unroll
    for (int e = 0; e < NC; ++e)
      if (e < FULL || e * 32 < left) v[e] += bs[e * 32];
  }
  warp_softmax<T, NC, FULL>(v, left, dst);
}

// The same for few groups with many partial sums: a block per group, a thread per entry while the partial sums are added (in
// the same order), then the group's softmax by the first warp as above.  With a warp per group, 64 groups of 207 entries in 64
// partial sums took 24.8 us, two dependent rounds of loads per pair of partial sums; 8.6 us so.
template <typename T, int NC>
__global__ void __launch_bounds__(256)
    softmax_block_kernel(const T *__restrict__ partial, int splits, long slice, const T *__restrict__ bias, T *__restrict__ out, int H,
                         int Mc) {
  after_previous();
  __shared__ T support[NC * 32];
  const long base = (long)blockIdx.x * Mc;
  const T *bs = bias ? bias + (blockIdx.x % (unsigned)H) * (long)Mc : nullptr;
  for (int j = threadIdx.x; j < Mc; j += 256) {
    constexpr int U = 16;
    const T *p = partial + base + j;
    T s = p[0];
    for (int z = 1; z < splits; z += U) {
      T d[U];
#pragma unroll
      for (int u = 0; u < U; ++u) d[u] = z + u < splits ? p[(z + u) * slice] : (T)0;
#pragma unroll
      for (int u = 0; u < U; ++u) s = z + u < splits ? s + d[u] : s;
    }
    support[j] = bs ? s + bs[j] : s;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int left = Mc - (int)threadIdx.x;
  T v[NC];
#pragma unroll
  for (int e = 0; e < NC; ++e) v[e] = e * 32 < left ? support[threadIdx.x + e * 32] : -INFINITY;
  warp_softmax<T, NC, 0>(v, left, out + base + threadIdx.x);
}

// And for groups of up to 16 entries, one to a lane: 2^log2 lanes per group.  1524 x 82 groups of 5 doubles took 15.3 us in the
// general kernel, most of it index arithmetic in 64 bits, 8.7 us here; 627 x 96 groups of 16 floats 16.7 and 14.0.
template <typename T>
__global__ void __launch_bounds__(256)
    softmax_lanes_kernel(const T *partial, int splits, long slice, const T *__restrict__ bias, T *out,   // (may be the same)
                         uint32_t groups, uint32_t H, uint32_t Mc, int log2) {
  after_previous();
  const int width = 1 << log2;
  const uint32_t at = blockIdx.x * 256u + threadIdx.x, g = at >> log2, sub = at & (uint32_t)(width - 1);
  const bool live = g < groups && sub < Mc;
  const uint32_t i = g * Mc + sub;
  T v = -INFINITY;
  if (live) {
    constexpr int U = 8;
    const T *p = partial + i;
    v = p[0];
    for (int z = 1; z < splits; z += U) {
      T d[U];
#pragma unroll
      for (int u = 0; u < U; ++u) d[u] = z + u < splits ? p[(z + u) * slice] : (T)0;
#pragma unroll
      for (int u = 0; u < U; ++u) v = z + u < splits ? v + d[u] : v;
    }
    if (bias) v += bias[g % H * Mc + sub];
  }
  T mx = v > -INFINITY ? v : -INFINITY;
  mx = subwarp_max(mx, width);
  const T e = live ? sbb_exp(v - mx) : (T)0;
  const T sum = subwarp_sum(e, width);
  if (live) out[i] = e / sum;
}

// out[r, j] = sum_s partial[s, r, j] + bias[j]   (no softmax)
template <typename T>
__global__ void __launch_bounds__(256)
    reduce_bias_kernel(const T *partial, int splits, long slice, const T *__restrict__ bias, T *out, long total,
                       long M) {
  after_previous();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  T s = partial[idx];
  for (int z = 1; z < splits; ++z) s += partial[(long)z * slice + idx];
  if (bias) s += bias[idx % M];
  out[idx] = s;
}

template <typename T>
cudaError_t launch_reduce_bias_softmax(const T *partial, int splits, const T *bias, T *out, long rows, long H,
                                       long Mc, int softmax, cudaStream_t st) {
  const long M = H * Mc;
  const long total = rows * M;
  if (total == 0) return cudaSuccess;
  if (!softmax) {
    if (splits == 1 && bias == nullptr && partial == out) return cudaSuccess;
    launch_next(reduce_bias_kernel<T>, (unsigned)((total + 255) / 256), 256, 0, st, partial, splits, total, bias, out, total, M);
    return launched();
  }
  int width = 32;
  while (width > 1 && (width >> 1) >= Mc) width >>= 1;
  const long groups = rows * H;
  const long per_lane = (Mc + width - 1) / width;
  if (width == 32 && per_lane <= 16 && groups < (1l << 31)) {
    // few groups, many partial sums: a block per group.  (128 x 30 groups of 100 in six parts stay with a warp each.)
    if (splits >= 8 && groups <= 4 * sm_count()) {
      if (per_lane <= 8) launch_next(softmax_block_kernel<T, 8>, (unsigned)groups, 256, 0, st, partial, splits, total, bias, out, (int)H, (int)Mc);
      else launch_next(softmax_block_kernel<T, 16>, (unsigned)groups, 256, 0, st, partial, splits, total, bias, out, (int)H, (int)Mc);
      return launched();
    }
    // one warp per group: the lean kernel (same arithmetic, same summation order)
#define SBB_SOFTMAX_WARP(NC, FULL)                                                                                     \
  do {                                                                                                            \
    if (splits > 1)                                                                                               \
      launch_next(softmax_warp_kernel<T, NC, FULL, true>, (unsigned)((groups + 7) / 8), 256, 0, st, partial, splits, total, bias, out, \
                                                                                    (uint32_t)groups, (uint32_t)H, (int)Mc);    \
    else                                                                                                          \
      launch_next(softmax_warp_kernel<T, NC, FULL, false>, (unsigned)((groups + 7) / 8), 256, 0, st, partial, splits, total, bias, out, \
                                                                                     (uint32_t)groups, (uint32_t)H, (int)Mc);   \
  } while (0)
    // (float32: slots in pairs, and a test for the last pair's entries alone.  100 groups of 300 at batch 1024, 10 slots: 68.0 us
    // with 12 slots and a test in each, 37.6 so.  In float64 more kernels than these gain nothing: the exponential takes the time)
    constexpr bool F32 = sizeof(T) == 4;
    if (per_lane <= 2) SBB_SOFTMAX_WARP(2, 0);
    else if (per_lane <= 4) SBB_SOFTMAX_WARP(4, F32 ? 2 : 0);
    else if (F32 && per_lane <= 6) SBB_SOFTMAX_WARP(F32 ? 6 : 8, F32 ? 4 : 0);
    else if (per_lane <= 8) SBB_SOFTMAX_WARP(8, F32 ? 6 : 0);
    else if (F32 && per_lane <= 10) SBB_SOFTMAX_WARP(F32 ? 10 : 12, F32 ? 8 : 0);
    else if (per_lane <= 12) SBB_SOFTMAX_WARP(12, F32 ? 10 : 0);
    else SBB_SOFTMAX_WARP(16, F32 ? 12 : 0);
#undef SBB_SOFTMAX_WARP
    return launched();
  }
  if (width < 32 && groups * width < (1l << 31) && total < (1l << 31)) {
    int log2 = 0;
    while ((1 << log2) < width) ++log2;
    launch_next(softmax_lanes_kernel<T>, (unsigned)((groups * width + 255) / 256), 256, 0, st, partial, splits, total, bias, out,
                (uint32_t)groups, (uint32_t)H, (uint32_t)Mc, log2);
    return launched();
  }
  const long per_warp = 32 / width, warps = (groups + per_warp - 1) / per_warp;
  launch_next(reduce_bias_softmax_kernel<T>, (unsigned)((warps + 7) / 8), 256, 0, st, partial, splits, total, bias, out, groups, H, Mc, width);
  return launched();
}
template cudaError_t launch_reduce_bias_softmax<float>(const float *, int, const float *, float *, long, long, long,
                                                       int, cudaStream_t);
template cudaError_t launch_reduce_bias_softmax<double>(const double *, int, const double *, double *, long, long,
                                                        long, int, cudaStream_t);

// ----------------------------------------------------------------------------
// Column sums over the batch.
// Block = 32 columns x 8 row lanes; rows are summed in a fixed order.
// ----------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    colsum_kernel(const T *__restrict__ a, long B, long cols, T *sums, T *lo) {
  after_previous();
  __shared__ T part[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long col = (long)blockIdx.x * 32 + tx;
  T s = (T)0;
  if (col < cols) {
    long b = ty;
    for (; b + 24 < B; b += 32) {
      const T v0 = __ldg(a + b * cols + col), v1 = __ldg(a + (b + 8) * cols + col);
      const T v2 = __ldg(a + (b + 16) * cols + col), v3 = __ldg(a + (b + 24) * cols + col);
      s += v0; s += v1; s += v2; s += v3;
      if (lo) {   // the operand's low parts for the split product of the tensor-core contraction that follows
        lo[b * cols + col] = tf32_lo(v0);
        lo[(b + 8) * cols + col] = tf32_lo(v1);
        lo[(b + 16) * cols + col] = tf32_lo(v2);
        lo[(b + 24) * cols + col] = tf32_lo(v3);
      }
    }
    for (; b < B; b += 8) {
      const T v = __ldg(a + b * cols + col);
      s += v;
      if (lo) lo[b * cols + col] = tf32_lo(v);
    }
  }
  part[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && col < cols) {
    T t = part[0][tx];
#pragma unroll
    for (int r = 1; r < 8; ++r) t += part[r][tx];
    sums[col] = t;
  }
}

template <typename T>
cudaError_t launch_colsum(const T *a, long B, long cols, T *sums, cudaStream_t st, T *lo) {
  if (cols == 0) return cudaSuccess;
  launch_next(colsum_kernel<T>, (unsigned)((cols + 31) / 32), 256, 0, st, a, B, cols, sums, lo);
  return launched();
}
template cudaError_t launch_colsum<float>(const float *, long, long, float *, cudaStream_t, float *);
template cudaError_t launch_colsum<double>(const double *, long, long, double *, cudaStream_t, double *);

// What a train step derives from the column sums of its batch, for both operands in one launch: Ci and Cj, their
// reciprocals (rc != null; 0 below the threshold) and, from Cj, gain and bias (kbi != null).  The sums are formed in the
// order of colsum_kernel.  Bound by latency for small layers, by HBM otherwise: sixteen loads per thread in flight.  (The two
// column sums, the reciprocals and the bias were four launches, 2 x 3.3 + 1.9 + 1.9 us at 1568 + 3000 columns, batch 128;
// 3.7 us now.  1568 + 30000 columns, batch 1024: 67 -> 28 us.)
template <typename T, bool few>
__global__ void __launch_bounds__(256)
    column_vectors_kernel(ColumnVectors<T> x, ColumnVectors<T> y, long B, TraceParams<T> p, BiasParams<T> nb, unsigned x_blocks) {
  after_previous();
  __shared__ T part[8][33];
  const bool is_x = blockIdx.x < x_blocks;
  const ColumnVectors<T> &o = is_x ? x : y;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long col = (long)(is_x ? blockIdx.x : blockIdx.x - x_blocks) * 32 + tx;
  T s = (T)0;
  if (col < o.cols) {
    constexpr int U = 16;
    const T *src = o.a + col;
    long b = ty;
    if (few) {   // long batches of few columns: sixteen loads of each of few blocks do not keep memory busy (88 + 528 columns at
                 // batch 5851: 20.7 -> 12 us)
      constexpr int D = 64;
      for (; b + 8 * (D - 1) < B; b += 8 * D) {
        T v[D];
#pragma unroll
        for (int u = 0; u < D; ++u) v[u] = __ldg(src + (b + 8 * u) * o.cols);
#pragma unroll
        for (int u = 0; u < D; ++u) s += v[u];
      }
    }
    for (; b + 8 * (U - 1) < B; b += 8 * U) {
      T v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = __ldg(src + (b + 8 * u) * o.cols);
#pragma unroll
      for (int u = 0; u < U; ++u) s += v[u];
    }
    T v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = b + 8 * u < B ? __ldg(src + (b + 8 * u) * o.cols) : (T)0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (b + 8 * u < B) s += v[u];
  }
  part[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && col < o.cols) {
    T t = part[0][tx];
#pragma unroll
    for (int r = 1; r < 8; ++r) t += part[r][tx];
    const T c = trace_ema(o.c[col], t, p);
    o.c[col] = c;
    if (o.rc != nullptr) o.rc[col] = c < p.cthr ? (T)0 : (T)1 / c;
    if (!is_x && nb.kbi != nullptr)
      bias_regularized(nb.bias[col], nb.kbi[col], c, p.cthr, nb.khalf, nb.pmin4, nb.k, nb.taubdt);
  }
}
template <typename T>
cudaError_t launch_column_vectors(const ColumnVectors<T> &x, const ColumnVectors<T> &y, long B, TraceParams<T> p,
                                  BiasParams<T> bias, cudaStream_t st) {
  const unsigned xb = (unsigned)((x.cols + 31) / 32), yb = (unsigned)((y.cols + 31) / 32);
  if (xb + yb == 0) return cudaSuccess;
  if (B >= 1024 && xb + yb <= 2 * (unsigned)sm_count()) launch_next(column_vectors_kernel<T, true>, xb + yb, 256, 0, st, x, y, B, p, bias, xb);
  else launch_next(column_vectors_kernel<T, false>, xb + yb, 256, 0, st, x, y, B, p, bias, xb);
  return launched();
}
template cudaError_t launch_column_vectors<float>(const ColumnVectors<float> &, const ColumnVectors<float> &, long,
                                                  TraceParams<float>, BiasParams<float>, cudaStream_t);
template cudaError_t launch_column_vectors<double>(const ColumnVectors<double> &, const ColumnVectors<double> &, long,
                                                   TraceParams<double>, BiasParams<double>, cudaStream_t);

template <typename T>
__global__ void vector_ema_kernel(T *c, const T *__restrict__ sums, long n, TraceParams<T> p) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) c[i] = trace_ema(c[i], sums[i], p);
}
template <typename T>
cudaError_t launch_vector_ema(T *c, const T *sums, long n, TraceParams<T> p, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  vector_ema_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(c, sums, n, p);
  return launched();
}
template cudaError_t launch_vector_ema<float>(float *, const float *, long, TraceParams<float>, cudaStream_t);
template cudaError_t launch_vector_ema<double>(double *, const double *, long, TraceParams<double>, cudaStream_t);

// ----------------------------------------------------------------------------
// Trace step: fused (x^T y in the contraction, traces and weights in its
// epilogue) and split (raw x^T y, then an element-wise tail).
// ----------------------------------------------------------------------------
// The float32 trace step of few samples: no tile of products to form, so a warp walks `rows` rows of 32 columns.  A lane owns a
// column, whose activations (and column data) stay in registers; lane r loads row r's inputs, which reach the others by
// shuffles.  Four rows' old traces are in flight while the four before are worked on, one after the other from one copy of the
// arithmetic.  Each sum is the chain of FMAs over ascending samples that the tile kernels form.
template <int NB>
__global__ void __launch_bounds__(256)
    trace_few_kernel(const float *__restrict__ x, long ldx, const float *__restrict__ y, int B, TraceEpilogue<float> e, unsigned column_warps,
                     int rows) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const unsigned warp = blockIdx.x * 8u + (threadIdx.x >> 5);
  const long i0 = e.row0 + (long)(warp / column_warps) * rows;
  if (i0 >= e.row_end) return;
  const int here = e.row_end - i0 < rows ? (int)(e.row_end - i0) : rows;
  const unsigned j = warp % column_warps * 32u + lane;
  const bool live = j < (unsigned)e.M;
  const unsigned col = live ? j : 0u;   // (loads need no branch)
  float yv[NB], xv[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    yv[b] = b < B ? y[(long)b * e.M + col] : 0.f;
    xv[b] = b < B && lane < here ? x[(long)b * ldx + i0 + lane] : 0.f;
  }
  const float my_ci = lane < here ? e.Ci[i0 + lane] : 0.f, cj = e.Cj[col];
  const bool column_on = !(cj < e.p.cthr);
  float *c = e.Cij + i0 * e.M + col, *w = e.W + i0 * e.M + col;
  const uint8_t *mask = e.wmask ? e.wmask + i0 * e.H + col / (unsigned)e.Mc : nullptr;
  constexpr int U = 4;
  float old[U], next[U];
  bool on[U], next_on[U];
  auto fetch = [&](int r0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = r0 + u < here;
      next[u] = in ? c[(long)(r0 + u) * e.M] : 0.f;
      next_on[u] = mask == nullptr || (in && mask[(long)(r0 + u) * e.H] != 0);
    }
  };
  fetch(0);
#pragma unroll 1
  for (int r0 = 0; r0 < here; r0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      old[u] = next[u];
      on[u] = next_on[u];
    }
    fetch(r0 + U);
    const int last = here < r0 + U ? here : r0 + U;
#pragma unroll 1
    for (int r = r0; r < last; ++r) {
      float sum = 0.f;
#pragma unroll
      for (int b = 0; b < NB; ++b) sum = fmaf(__shfl_sync(0xffffffffu, xv[b], r), yv[b], sum);
      const float ci = __shfl_sync(0xffffffffu, my_ci, r);
      const float v = trace_ema(old[0], sum, e.p);
      const float g = on[0] && column_on && !(ci < e.p.cthr) ? log_ratio(v, ci, cj, e.p.cthr4) : 0.f;
      if (live) {
        c[(long)r * e.M] = v;
        w[(long)r * e.M] = g;
      }
#pragma unroll
      for (int u = 0; u + 1 < U; ++u) {
        old[u] = old[u + 1];
        on[u] = on[u + 1];
      }
    }
  }
}
// What bounds it is the issue of instructions, some hundred for the two divisions and the logarithm of an element, and two more for
// each sample.  Train step without a mask update, tiles -> this, at 4, 8 and 16 samples: 3202 x 7398 177 -> 95, 178 -> 116,
// 178 -> 154 us; 2217 x 1425 35.9 -> 21.0, 36.0 -> 23.2, 36.0 -> 27.1; 26849 x 49 23.1 -> 16.3, 23.2 -> 16.4, 23.2 -> 15.9; 1211 x 39
// 7.2 -> 7.1, 7.3 -> 6.9, 7.2 -> 6.9.  The same kernel for 24 samples loses: 190 -> 254, 38.7 -> 49.4, 26.2 -> 26.0, 7.2 -> 7.0.
constexpr long kFewTrace = 16;   // most samples
static bool few_trace_fits(long B, long rows, long M) {
  return B >= 1 && B <= kFewTrace && M < (1l << 31) && ((M + 31) / 32) * ((rows + 3) / 4) < (1l << 31);
}
static cudaError_t launch_trace_few(const float *x, long ldx, const float *y, long B, const TraceEpilogue<float> &e, cudaStream_t st) {
  const long n = e.row_end - e.row0, column_warps = (e.M + 31) / 32;
  int rows = 32;   // (fewer where that leaves fewer than sixteen warps to an SM)
  while (rows > 4 && ((n + rows - 1) / rows) * column_warps < 16l * sm_count()) rows >>= 1;
  const unsigned blocks = (unsigned)((((n + rows - 1) / rows) * column_warps + 7) / 8);
  auto launch = [&](auto kernel) { launch_next(kernel, blocks, 256, 0, st, x, ldx, y, (int)B, e, (unsigned)column_warps, rows); };
  if (B <= 4) launch(trace_few_kernel<4>);
  else if (B <= 8) launch(trace_few_kernel<8>);
  else launch(trace_few_kernel<16>);
  return launched();
}

template <typename T>
cudaError_t launch_trace_update_fused(const T *x, const T *y, long B, long N, long M, long H, long Mc, const T *Ci,
                                      const T *Cj, const T *rci, const T *rcj, T *Cij, T *w, const uint8_t *wmask,
                                      TraceParams<T> p, long row_begin, long row_end, cudaStream_t st) {
  constexpr int V = Vec16<T>::N;
  if (row_end <= row_begin) return cudaSuccess;
  const bool vec = (N % V == 0) && (M % V == 0) && (row_begin % V == 0) && ((row_end - row_begin) % V == 0) &&
                   aligned16(x) && aligned16(y);
  TraceEpilogue<T> ep{Ci, Cj, Cij, w, wmask, row_begin, row_end, M, H, Mc, p,
                      (M % V == 0) && aligned16(Cij) && aligned16(w), rci, rcj};
  if constexpr (std::is_same<T, float>::value)
    if (few_trace_fits(B, row_end - row_begin, M)) return launch_trace_few(x, N, y, B, ep, st);
  const int kper = (int)((B + Tile::BK - 1) / Tile::BK) * Tile::BK;
  return launch_contraction<T, false>(x + row_begin, N, y, M, row_end - row_begin, M, (int)B, 1, kper, vec, true, ep, st);
}
template cudaError_t launch_trace_update_fused<float>(const float *, const float *, long, long, long, long, long,
                                                      const float *, const float *, const float *, const float *, float *, float *,
                                                      const uint8_t *, TraceParams<float>, long, long, cudaStream_t);
template cudaError_t launch_trace_update_fused<double>(const double *, const double *, long, long, long, long, long,
                                                       const double *, const double *, const double *, const double *, double *,
                                                       double *,
                                                       const uint8_t *, TraceParams<double>, long, long,
                                                       cudaStream_t);

template <typename T>
cudaError_t launch_outer_product(const T *x, const T *y, long B, long N, long M, T *delta, long row_begin,
                                 long row_end, cudaStream_t st) {
  constexpr int V = Vec16<T>::N;
  if (row_end <= row_begin) return cudaSuccess;
  const bool vec = (N % V == 0) && (M % V == 0) && (row_begin % V == 0) && ((row_end - row_begin) % V == 0) &&
                   aligned16(x) && aligned16(y);
  StoreEpilogue<T> ep{delta + row_begin * M, row_end - row_begin, M, M, 0, (M % V == 0) && aligned16(delta)};
  const int kper = (int)((B + Tile::BK - 1) / Tile::BK) * Tile::BK;
  return launch_contraction<T, false>(x + row_begin, N, y, M, row_end - row_begin, M, (int)B, 1, kper, vec, true, ep, st);
}
template cudaError_t launch_outer_product<float>(const float *, const float *, long, long, long, float *, long, long,
                                                 cudaStream_t);
template cudaError_t launch_outer_product<double>(const double *, const double *, long, long, long, double *, long,
                                                  long, cudaStream_t);

// One thread per four consecutive columns, walking kApplyRows rows: the column data (Cj, the
// hypercolumn of each column) is set up once per thread, rows only add Ci and the mask byte.
constexpr int kApplyRows = 8;
// FAST (float32 only): the tensor-core path's arithmetic (see sbb_math.cuh), so that the data-parallel
// step and the fused single-device step of that path compute the same values from the same sums.
template <typename T, bool FAST>
__global__ void __launch_bounds__(256)
    trace_apply_kernel(const T *__restrict__ delta, long M, long H, long Mc, const T *__restrict__ Ci,
                       const T *__restrict__ Cj, T *Cij, T *W, const uint8_t *__restrict__ wmask, TraceParams<T> p,
                       int ema, long row_begin, long row_end, bool vec) {
  const long j = ((long)blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (j >= M) return;
  const long left = M - j;
  const int valid = left >= 4 ? 4 : (int)left;
  T cj[4];
  bool col_on[4];
  long hc[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    cj[c] = c < valid ? Cj[j + c] : (T)1;
    col_on[c] = c < valid && !(cj[c] < p.cthr);
    hc[c] = wmask ? (j + (c < valid ? c : 0)) / Mc : 0;
    if (FAST) cj[c] = (T)1 / cj[c];   // from here on the reciprocal
  }
  const T ema_scale = p.taupdt / p.batch;
  const bool one_hc = hc[0] == hc[3] && hc[0] == hc[1] && hc[0] == hc[2];
  const long r0 = row_begin + (long)blockIdx.x * kApplyRows;
  const long r1 = r0 + kApplyRows < row_end ? r0 + kApplyRows : row_end;
  for (long i = r0; i < r1; ++i) {
    T ci = Ci[i];
    const bool row_on = !(ci < p.cthr);
    if (FAST) ci = (T)1 / ci;
    bool on[4];
    if (wmask == nullptr) {
#pragma unroll
      for (int c = 0; c < 4; ++c) on[c] = row_on && col_on[c];
    } else if (one_hc) {
      const bool m = wmask[i * H + hc[0]] != 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) on[c] = row_on && col_on[c] && m;
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) on[c] = row_on && col_on[c] && wmask[i * H + hc[c]] != 0;
    }
    T c4[4], d4[4], w4[4];
    load4(Cij + i * M + j, c4, vec, valid);
    if (ema) load4(delta + i * M + j, d4, vec, valid);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c < valid) {
        T cij = c4[c];
        if constexpr (FAST) {
          if (ema) cij = trace_ema_fast(c4[c], d4[c], p.one_minus, ema_scale);
          w4[c] = on[c] ? log_ratio_fast(cij, ci, cj[c], p.cthr4) : 0.f;
        } else {
          if (ema) cij = trace_ema(c4[c], d4[c], p);
          w4[c] = on[c] ? log_ratio(cij, ci, cj[c], p.cthr4) : (T)0;
        }
        c4[c] = cij;
      }
    }
    if (ema) store4(Cij + i * M + j, c4, vec, valid);
    store4(W + i * M + j, w4, vec, valid);
  }
}

template <typename T>
cudaError_t launch_trace_apply(const T *delta, long N, long M, long H, long Mc, const T *Ci, const T *Cj, T *Cij,
                               T *w, const uint8_t *wmask, TraceParams<T> p, int ema, long row_begin, long row_end,
                               cudaStream_t st, bool fast) {
  (void)N;
  constexpr int V = Vec16<T>::N;
  if (row_end <= row_begin || M == 0) return cudaSuccess;
  const long qpr = (M + 3) / 4;
  const bool vec = (M % V == 0) && aligned16(Cij) && aligned16(w) && (!ema || aligned16(delta));
  const long row_groups = (row_end - row_begin + kApplyRows - 1) / kApplyRows;
  const int threads = qpr >= 256 ? 256 : (int)((qpr + 31) / 32 * 32);
  const dim3 grid((unsigned)row_groups, (unsigned)((qpr + threads - 1) / threads));
  if constexpr (std::is_same<T, float>::value) {
    if (fast && p.cthr4 >= 1e-30f) {
      trace_apply_kernel<float, true><<<grid, threads, 0, st>>>(delta, M, H, Mc, Ci, Cj, Cij, w, wmask, p, ema, row_begin,
                                                                row_end, vec);
      return launched();
    }
  }
  trace_apply_kernel<T, false><<<grid, threads, 0, st>>>(delta, M, H, Mc, Ci, Cj, Cij, w, wmask, p, ema, row_begin,
                                                         row_end, vec);
  return launched();
}
template cudaError_t launch_trace_apply<float>(const float *, long, long, long, long, const float *, const float *,
                                               float *, float *, const uint8_t *, TraceParams<float>, int, long, long,
                                               cudaStream_t, bool);
template cudaError_t launch_trace_apply<double>(const double *, long, long, long, long, const double *,
                                                const double *, double *, double *, const uint8_t *,
                                                TraceParams<double>, int, long, long, cudaStream_t, bool);

// ----------------------------------------------------------------------------
// The trace step of a long batch whose outputs are few tiles: the batch is cut into `splits` parts, whose products are
// formed side by side (a fused launch would sum each output over the whole batch on a few SMs), and this adds them up and does
// what the fused epilogues do.  The arithmetic is that of the path: reciprocals and lg2 behind the tensor-core product
// (FAST), the reciprocals and logarithm of the float64 kernel, divisions and the library's logarithm otherwise.
// 88 -> 2 x 264 at batch 5851, train step: float32 165 us fused, 31 so; float64 235 and 50.
// ----------------------------------------------------------------------------
template <typename T, int V, bool FAST>
__global__ void __launch_bounds__(256)
    split_trace_kernel(const T *__restrict__ partial, int splits, long slice, int M, int H, int Mc, const T *__restrict__ Ci,
                       const T *__restrict__ Cj, const T *__restrict__ rci, const T *__restrict__ rcj, T *Cij, T *W,
                       const uint8_t *__restrict__ wmask, TraceParams<T> p) {
  after_previous();
  const long at = ((long)blockIdx.x * 256 + threadIdx.x) * V;
  if (at >= slice) return;
  const long i = at / M;
  const int j = (int)(at - i * M);
  struct alignas(sizeof(T) * V) Piece {
    T v[V];
  };
  Piece c = *reinterpret_cast<const Piece *>(Cij + at), w;
  const uint8_t *mrow = wmask ? wmask + i * H : nullptr;
  bool on[V];
  T cj[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    on[v] = mrow == nullptr || mrow[(unsigned)(j + v) / (unsigned)Mc] != 0;
    cj[v] = (FAST || sizeof(T) == 8 ? rcj : Cj)[j + v];
  }
  const T ci = (FAST || sizeof(T) == 8 ? rci : Ci)[i];
  T s[V];
#pragma unroll
  for (int v = 0; v < V; ++v) s[v] = (T)0;
  constexpr int U = 8;   // parts in flight
  for (int z = 0; z < splits; z += U) {
    Piece d[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (z + u < splits) d[u] = *reinterpret_cast<const Piece *>(partial + (long)(z + u) * slice + at);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (z + u < splits)
#pragma unroll
        for (int v = 0; v < V; ++v) s[v] += d[u].v[v];
  }
#pragma unroll
  for (int v = 0; v < V; ++v) {
    T x;
    if constexpr (FAST) {
      x = trace_ema_fast(c.v[v], s[v], p.one_minus, p.taupdt / p.batch);
      w.v[v] = on[v] && ci != 0.f && cj[v] != 0.f ? log_ratio_fast(x, ci, cj[v], p.cthr4) : 0.f;
    } else if constexpr (sizeof(T) == 8) {
      x = fma(c.v[v], p.one_minus, s[v] * (1.0 / p.batch * p.taupdt));
      x = x > 0.0 ? x : 0.0;
      w.v[v] = on[v] && ci != 0.0 && cj[v] != 0.0 ? f64mma::log_positive((x < p.cthr4 ? p.cthr4 : x) * (ci * cj[v])) : 0.0;
    } else {
      x = trace_ema(c.v[v], s[v], p);
      w.v[v] = on[v] && !(ci < p.cthr) && !(cj[v] < p.cthr) ? log_ratio(x, ci, cj[v], p.cthr4) : (T)0;
    }
    c.v[v] = x;
  }
  *reinterpret_cast<Piece *>(Cij + at) = c;
  *reinterpret_cast<Piece *>(W + at) = w;
}

template <typename T>
cudaError_t launch_split_trace(const T *partial, int splits, long N, long M, long H, long Mc, const T *Ci, const T *Cj,
                               const T *rci, const T *rcj, T *Cij, T *w, const uint8_t *wmask, TraceParams<T> p, bool fast,
                               cudaStream_t st) {
  const long slice = N * M;
  constexpr int V = Vec16<T>::N;
  const bool vec = M % V == 0 && aligned16(partial) && aligned16(Cij) && aligned16(w);
  auto launch = [&](auto kernel, int v) {
    launch_next(kernel, (unsigned)((slice / v + 255) / 256), 256, 0, st, partial, splits, slice, (int)M, (int)H, (int)Mc, Ci, Cj, rci,
                rcj, Cij, w, wmask, p);
  };
  if constexpr (sizeof(T) == 4) {
    if (fast) {   // (the tensor-core path's rows are multiples of 16 bytes)
      launch(split_trace_kernel<T, V, true>, V);
      return launched();
    }
  }
  if (vec) launch(split_trace_kernel<T, V, false>, V);
  else launch(split_trace_kernel<T, 1, false>, 1);
  return launched();
}
template cudaError_t launch_split_trace<float>(const float *, int, long, long, long, long, const float *, const float *,
                                               const float *, const float *, float *, float *, const uint8_t *,
                                               TraceParams<float>, bool, cudaStream_t);
template cudaError_t launch_split_trace<double>(const double *, int, long, long, long, long, const double *, const double *,
                                                const double *, const double *, double *, double *, const uint8_t *,
                                                TraceParams<double>, bool, cudaStream_t);

// partial[s, N, M]: the products of the parts of the batch.
template <typename T>
cudaError_t launch_split_product(const T *x, const T *y, long B, long N, long M, int splits, T *partial, cudaStream_t st) {
  constexpr int V = Vec16<T>::N;
  const bool vec = N % V == 0 && M % V == 0 && aligned16(x) && aligned16(y);
  StoreEpilogue<T> ep{partial, N, M, M, N * M, M % V == 0 && aligned16(partial)};
  const long slabs = (B + Tile::BK - 1) / Tile::BK;
  return launch_contraction<T, false>(x, N, y, M, N, M, (int)B, splits, (int)((slabs + splits - 1) / splits) * Tile::BK, vec, true,
                                      ep, st);
}
template cudaError_t launch_split_product<float>(const float *, const float *, long, long, long, int, float *, cudaStream_t);
template cudaError_t launch_split_product<double>(const double *, const double *, long, long, long, int, double *, cudaStream_t);

// Parts the batch of a trace step is cut into (1: the fused kernel), from what a launch takes in microseconds: slabs of a part
// times the time of one with so many blocks to an SM, and for the parts the second launch and the way of the partial sums to
// memory and back.  Measured (train step without a mask update, fused -> best of 2 to 48 parts -> the rule's): float32 501 x 301
// at batch 1001 41 -> 23 -> 24, 207 x 9 at 4000 136 -> 22 -> 21; float64 88 x 528 at 5851 235 -> 50 -> 50, 501 x 301 at 1001 54 ->
// 24 -> 24, 256 x 256 at 2048 90 -> 24 -> 26, 5000 x 50 at 3000 148 -> 101 -> 103.  With more tiles than blocks fit it loses:
// float64 2048 x 512 at 1024 86 -> 90.  Its sums are the more exact ones (1843 x 424 at 5485: 5e-8 of the trace against 2e-7).
template <typename T>
int trace_splits(long B, long N, long M) {
  // (float32 layers of many inputs keep the order of their sums, as few_plan's: 1843 x 424 at batch 5485 moved single weights by
  // 7e-4 of their mean square in two steps, 12566 x 102 at 1444 the activations by 2e-5)
  if (B < 128 || (sizeof(T) == 4 && N > 1024)) return 1;
  const long sms = sm_count();
  auto ceil_div = [](long a, long b) { return (a + b - 1) / b; };
  auto per_slab = [&](long blocks, long per_sm, double one, double two, double full) {   // us, by the blocks an SM has
    if (blocks <= sms) return one;
    if (blocks <= 2 * sms) return two;
    return full * (double)ceil_div(blocks, per_sm * sms);
  };
  auto cost = [&](long s) {
    if (sizeof(T) == 8) return ceil_div(ceil_div(B, 16), s) * per_slab(ceil_div(N, 64) * ceil_div(M, 64) * s, 3, 0.9, 1.0, 1.5);
    const long tiles = ceil_div(N, 128) * ceil_div(M, 128) * s;
    if (small_tiles(tiles, false)) return ceil_div(ceil_div(B, 32), s) * per_slab(ceil_div(N, 32) * ceil_div(M, 64) * s, 4, 1.2, 1.5, 2.0);
    return ceil_div(ceil_div(B, 16), s) * per_slab(tiles, 2, 1.9, 3.4, 3.4);
  };
  int best = 1;
  const double fused = cost(1);
  double least = 0.85 * fused;
  for (long s = 2; s <= 48 && B / s >= 64; ++s) {
    if (s * N * M > (1l << 26)) break;
    const double c = cost(s) + 4.0 + (double)(s * N * M) * (2 * sizeof(T)) / 3e6;
    if (c < least) least = c, best = (int)s;
  }
  const long slabs = ceil_div(B, Tile::BK);
  return (int)ceil_div(slabs, ceil_div(slabs, best));   // no empty part
}
template int trace_splits<float>(long, long, long);
template int trace_splits<double>(long, long, long);

// Un-fused trace update in the NumPy operation order: (1-t)*C + t*(sum/B).
template <typename T>
__global__ void counters_apply_kernel(T *c, const T *__restrict__ sums, long n, T taupdt, T batch) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const T v = ((T)1 - taupdt) * c[i] + taupdt * (sums[i] / batch);
  c[i] = v > (T)0 ? v : (T)0;
}
template <typename T>
cudaError_t launch_counters_apply(T *c, const T *sums, long n, T taupdt, T batch, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  counters_apply_kernel<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(c, sums, n, taupdt, batch);
  return launched();
}
template cudaError_t launch_counters_apply<float>(float *, const float *, long, float, float, cudaStream_t);
template cudaError_t launch_counters_apply<double>(double *, const double *, long, double, double, cudaStream_t);

// ----------------------------------------------------------------------------
// Bias kernels and small element-wise helpers.
// ----------------------------------------------------------------------------
template <typename T>
__global__ void update_bias_kernel(T *bias, const T *__restrict__ Cj, T cthr, long M) {
  const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < M) bias[j] = Cj[j] < cthr ? sbb_log((T)2 * cthr) : sbb_log(Cj[j]);
}
template <typename T>
cudaError_t launch_update_bias(T *bias, const T *Cj, T cthr, long M, cudaStream_t st) {
  if (M == 0) return cudaSuccess;
  update_bias_kernel<T><<<(unsigned)((M + 255) / 256), 256, 0, st>>>(bias, Cj, cthr, M);
  return launched();
}
template cudaError_t launch_update_bias<float>(float *, const float *, float, long, cudaStream_t);
template cudaError_t launch_update_bias<double>(double *, const double *, double, long, cudaStream_t);

template <typename T>
BiasParams<T> make_bias(T *bias, T *kbi, T khalf, T pmin, T taubdt) {
  const T pmin4 = pmin / (T)4;
  return BiasParams<T>{bias, kbi, khalf, pmin4, (khalf - (T)1) * (pmin4 * pmin4), taubdt};
}
template BiasParams<float> make_bias<float>(float *, float *, float, float, float);
template BiasParams<double> make_bias<double>(double *, double *, double, double, double);

template <typename T>
__global__ void update_bias_regularized_kernel(T *bias, T *kbi, const T *__restrict__ Cj, T cthr, T khalf, T pmin4,
                                               T k, T taubdt, long M) {
  const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  bias_regularized(bias[j], kbi[j], Cj[j], cthr, khalf, pmin4, k, taubdt);
}
template <typename T>
cudaError_t launch_update_bias_regularized(T *bias, T *kbi, const T *Cj, T cthr, T khalf, T pmin, T taubdt, long M,
                                           cudaStream_t st) {
  if (M == 0) return cudaSuccess;
  const BiasParams<T> b = make_bias<T>(bias, kbi, khalf, pmin, taubdt);
  update_bias_regularized_kernel<T><<<(unsigned)((M + 255) / 256), 256, 0, st>>>(bias, kbi, Cj, cthr, khalf, b.pmin4, b.k,
                                                                                  taubdt, M);
  return launched();
}
template cudaError_t launch_update_bias_regularized<float>(float *, float *, const float *, float, float, float,
                                                           float, long, cudaStream_t);
template cudaError_t launch_update_bias_regularized<double>(double *, double *, const double *, double, double,
                                                            double, double, long, cudaStream_t);

template <typename T>
__global__ void add_bias_kernel(T *a, const T *__restrict__ bias, long total, long M) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < total) a[idx] += bias[idx % M];
}
template <typename T>
cudaError_t launch_add_bias(T *a, const T *bias, long rows, long M, cudaStream_t st) {
  const long total = rows * M;
  if (total == 0) return cudaSuccess;
  add_bias_kernel<T><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a, bias, total, M);
  return launched();
}
template cudaError_t launch_add_bias<float>(float *, const float *, long, long, cudaStream_t);
template cudaError_t launch_add_bias<double>(double *, const double *, long, long, cudaStream_t);

template <typename T>
__global__ void apply_mask_kernel(T *w, const uint8_t *__restrict__ wmask, long total, long M, long H, long Mc) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const long i = idx / M, j = idx % M;
  if (!wmask[i * H + j / Mc]) w[idx] = (T)0;
}
template <typename T>
cudaError_t launch_apply_mask(T *w, const uint8_t *wmask, long N, long M, long H, long Mc, cudaStream_t st) {
  const long total = N * M;
  if (total == 0) return cudaSuccess;
  apply_mask_kernel<T><<<(unsigned)((total + 255) / 256), 256, 0, st>>>(w, wmask, total, M, H, Mc);
  return launched();
}
template cudaError_t launch_apply_mask<float>(float *, const uint8_t *, long, long, long, long, cudaStream_t);
template cudaError_t launch_apply_mask<double>(double *, const uint8_t *, long, long, long, long, cudaStream_t);



// ----------------------------------------------------------------------------
// Evaluation helper: rows whose predicted class equals the labelled class
// (first maximum wins, as numpy.argmax).
// ----------------------------------------------------------------------------
template <typename T>
__global__ void count_correct_kernel(const T *__restrict__ pred, const T *__restrict__ labels, long rows, long classes,
                                     unsigned long long *count) {
  after_previous();
  const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  bool hit = false;
  if (r < rows) {
    long ap = 0, al = 0;
    T vp = pred[r * classes], vl = labels[r * classes];
    for (long c = 1; c < classes; ++c) {
      const T p = pred[r * classes + c], l = labels[r * classes + c];
      if (p > vp) { vp = p; ap = c; }
      if (l > vl) { vl = l; al = c; }
    }
    hit = ap == al;
  }
  const unsigned ballot = __ballot_sync(0xffffffffu, hit);
  if ((threadIdx.x & 31) == 0 && ballot) atomicAdd(count, (unsigned long long)__popc(ballot));
}
template <typename T>
cudaError_t launch_count_correct(const T *pred, const T *labels, long rows, long classes, unsigned long long *count,
                                 cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  launch_next(count_correct_kernel<T>, (unsigned)((rows + 255) / 256), 256, 0, st, pred, labels, rows, classes, count);
  return launched();
}
template cudaError_t launch_count_correct<float>(const float *, const float *, long, long, unsigned long long *,
                                                 cudaStream_t);
template cudaError_t launch_count_correct<double>(const double *, const double *, long, long, unsigned long long *,
                                                  cudaStream_t);

// ----------------------------------------------------------------------------
// Batch assembly: dst[r, :] = src[order[first + r], :] (order null: the identity).  One
// warp copies one row in 16-byte pieces when the row pitch allows, else element-wise.
// HBM-bound: rows * cols * sizeof(T) read and written.
// ----------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    gather_rows_kernel(const T *__restrict__ src, const long *__restrict__ order, long first, long rows, long cols,
                       T *__restrict__ dst, int vec16) {
  after_previous();
  const long warp = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long nwarps = ((long)gridDim.x * blockDim.x) >> 5;
  for (long r = warp; r < rows; r += nwarps) {
    const long from = order ? order[first + r] : first + r;
    const T *s = src + from * cols;
    T *d = dst + r * cols;
    if (vec16) {
      const long pieces = cols * (long)sizeof(T) / 16;
      const uint4 *s4 = reinterpret_cast<const uint4 *>(s);
      uint4 *d4 = reinterpret_cast<uint4 *>(d);
      for (long k = lane; k < pieces; k += 32) d4[k] = __ldg(s4 + k);
    } else {
      for (long k = lane; k < cols; k += 32) d[k] = s[k];
    }
  }
}
template <typename T>
cudaError_t launch_gather_rows(const T *src, const long *order, long first, long rows, long cols, T *dst,
                               cudaStream_t st) {
  if (rows <= 0) return cudaSuccess;
  const int vec16 = (cols * (long)sizeof(T)) % 16 == 0 && aligned16(src) && aligned16(dst);
  const long blocks = (rows + 7) / 8;   // eight warps per block, one row per warp and pass
  const int cap = sm_count() * 8;
  launch_next(gather_rows_kernel<T>, (unsigned)(blocks < cap ? blocks : cap), 256, 0, st, src, order, first, rows, cols, dst,
                                                                                 vec16);
  return launched();
}
template cudaError_t launch_gather_rows<float>(const float *, const long *, long, long, long, float *, cudaStream_t);
template cudaError_t launch_gather_rows<double>(const double *, const long *, long, long, long, double *,
                                                cudaStream_t);

// ----------------------------------------------------------------------------
// Row-sharded layer over peer-mapped memory.  Every rank owns a block of input rows of
// the layer (those rows of the weights, of Cij and of Ci).  Per step the ranks exchange the
// matching COLUMNS of their input batches, so that every owner holds its columns of the
// whole global batch; each owner then forms its part of every sample's support, the parts
// are summed across the ranks, and the owner updates its rows from the global batch.
// The pointer tables below hold, per destination rank, an address in that rank's memory
// (the rank's own entry is a local address).
// ----------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) peer_broadcast_kernel(const T *__restrict__ src, long n, PeerTable dst) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const T v = src[i];
    for (int d = 0; d < dst.n; ++d) static_cast<T *>(dst.ptr[d])[i] = v;
  }
}
template <typename T>
cudaError_t launch_peer_broadcast(const T *src, long n, const PeerTable &dst, cudaStream_t st) {
  if (n <= 0 || dst.n <= 0) return cudaSuccess;
  const long blocks = (n + 255) / 256;
  peer_broadcast_kernel<T><<<(unsigned)(blocks < 1184 ? blocks : 1184), 256, 0, st>>>(src, n, dst);
  return launched();
}
template cudaError_t launch_peer_broadcast<float>(const float *, long, const PeerTable &, cudaStream_t);
template cudaError_t launch_peer_broadcast<double>(const double *, long, const PeerTable &, cudaStream_t);
template cudaError_t launch_peer_broadcast<uint4>(const uint4 *, long, const PeerTable &, cudaStream_t);

// Column block o of x[B, N] (columns [o * block, min(N, (o + 1) * block))) goes to rank o as a dense
// [B, width_o] matrix at dst.ptr[o].  V = elements moved per thread (a 16-byte vector when the shapes allow).
// Blocks of 128 threads with few registers, so that the kernel can run on a side stream beside a
// tensor-core contraction, whose one CTA per SM leaves room for little else.
template <typename T, int V>
__global__ void __launch_bounds__(128)
    scatter_columns_kernel(const T *__restrict__ x, long B, long N, long block, PeerTable dst) {
  struct alignas(sizeof(T) * V) Pack {
    T v[V];
  };
  const long per_row = N / V;
  const long total = B * per_row;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
    const long b = t / per_row;
    const long c = (t - b * per_row) * V;
    const long o = c / block;
    const long first = o * block;
    const long width = first + block <= N ? block : N - first;
    const Pack v = *reinterpret_cast<const Pack *>(x + b * N + c);
    *reinterpret_cast<Pack *>(static_cast<T *>(dst.ptr[o]) + b * width + (c - first)) = v;
  }
}
template <typename T>
cudaError_t launch_scatter_columns(const T *x, long B, long N, long block, const PeerTable &dst, cudaStream_t st) {
  if (B <= 0 || N <= 0) return cudaSuccess;
  constexpr int V = Vec16<T>::N;
  // a vector never straddles two owners when both N and the block width are multiples of V
  bool vec = N % V == 0 && block % V == 0 && aligned16(x);
  for (int d = 0; d < dst.n; ++d) vec = vec && aligned16(dst.ptr[d]);
  const long total = vec ? B * (N / V) : B * N;
  const long blocks = (total + 127) / 128;
  const unsigned grid = (unsigned)(blocks < 2368 ? blocks : 2368);
  if (vec) scatter_columns_kernel<T, V><<<grid, 128, 0, st>>>(x, B, N, block, dst);
  else scatter_columns_kernel<T, 1><<<grid, 128, 0, st>>>(x, B, N, block, dst);
  return launched();
}
template cudaError_t launch_scatter_columns<float>(const float *, long, long, long, const PeerTable &, cudaStream_t);
template cudaError_t launch_scatter_columns<double>(const double *, long, long, long, const PeerTable &, cudaStream_t);

// out[i] = sum over s (in order) of partial[s * n + i]
template <typename T>
__global__ void __launch_bounds__(256) sum_partials_kernel(const T *__restrict__ partial, int splits, long n, T *out) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    T s = partial[i];
    for (int k = 1; k < splits; ++k) s += partial[(long)k * n + i];
    out[i] = s;
  }
}
template <typename T>
cudaError_t launch_sum_partials(const T *partial, int splits, long n, T *out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const long blocks = (n + 255) / 256;
  sum_partials_kernel<T><<<(unsigned)(blocks < 2368 ? blocks : 2368), 256, 0, st>>>(partial, splits, n, out);
  return launched();
}
template cudaError_t launch_sum_partials<float>(const float *, int, long, float *, cudaStream_t);
template cudaError_t launch_sum_partials<double>(const double *, int, long, double *, cudaStream_t);

}  // namespace sbb

// ----------------------------------------------------------------------------
// Measured float64 rates of the device, for the roofline of the float64 kernels:
// a register-resident DFMA loop and a loop of mma.sync.m8n8k4 (the float64 tensor-core
// instruction).  Both keep every operand in registers; the result is stored once so
// that the loops are not removed.
// ----------------------------------------------------------------------------
namespace sbb {
namespace {
__global__ void __launch_bounds__(256) dfma_rate_kernel(double *out, int iters) {
  double a[8];
  const double x = 1.0 + 1e-9 * threadIdx.x, y = 1e-9;
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = (double)k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = fma(a[k], x, y);
  }
  double s = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += a[k];
  if (s == 12345.678) out[0] = s;   // never true: keeps the loop alive
}
__global__ void __launch_bounds__(256) dmma_rate_kernel(double *out, int iters) {
  double c[4][2];
  const double a = 1.0 + 1e-9 * threadIdx.x, b = 1e-9;
#pragma unroll
  for (int k = 0; k < 4; ++k) c[k][0] = c[k][1] = (double)k;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                   : "+d"(c[k][0]), "+d"(c[k][1])
                   : "d"(a), "d"(b));
  }
  double s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) s += c[k][0] + c[k][1];
  if (s == 12345.678) out[0] = s;
}
}  // namespace

// TFLOP/s of both loops on the current device (CUDA events, best of three launches).
cudaError_t measure_fp64_rates(double *dfma_tflops, double *dmma_tflops) {
  double *out = nullptr;
  cudaError_t e = cudaMalloc(&out, sizeof(double));
  if (e != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int blocks = sm_count() * 4, iters = 20000;
  double best[2] = {0.0, 0.0};
  for (int which = 0; which < 2; ++which)
    for (int rep = 0; rep < 4; ++rep) {
      cudaEventRecord(e0, 0);
      if (which == 0) dfma_rate_kernel<<<blocks, 256>>>(out, iters);
      else dmma_rate_kernel<<<blocks, 256>>>(out, iters);
      cudaEventRecord(e1, 0);
      e = cudaEventSynchronize(e1);
      if (e != cudaSuccess) break;
      launched();
      float ms = 0.f;
      cudaEventElapsedTime(&ms, e0, e1);
      // DFMA: 8 FMAs per thread and iteration; DMMA: 4 instructions of 8 x 8 x 4 FMAs per warp and iteration
      const double flops = which == 0 ? 2.0 * 8 * iters * 256.0 * blocks : 2.0 * 4 * 256 * iters * 8.0 * blocks;
      const double tf = flops / (ms * 1e-3) / 1e12;
      if (rep > 0 && tf > best[which]) best[which] = tf;
    }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (e != cudaSuccess) return e;
  *dfma_tflops = best[0];
  *dmma_tflops = best[1];
  return cudaGetLastError();
}
}  // namespace sbb
