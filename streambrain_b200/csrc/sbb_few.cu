// Forward pass for a few samples: contraction, bias and softmax in one launch.
//
// One sample reads all weights for one multiplication each, so what counts is how fast they stream and what comes after:
// 1568 x 3000 weights are 18.8 MB, 2 us out of L2.  The tiled kernels spent 12.0 + 5.1 us on it in two launches, 127 of
// 128 rows of every tile padding.  Here a block owns a few whole hypercolumns and a range of inputs, every thread streams
// 16-byte pieces of the weights with sixteen of them in flight, and the block that finishes a group of hypercolumns last
// adds up the ranges and takes the softmax.
#include "sbb_kernels.cuh"
#include "sbb_launch.cuh"
#include "sbb_math.cuh"

namespace sbb {

void count_launches(int n);   // sbb_kernels.cu

namespace {

constexpr int kFewThreads = 256;
// Inputs of a thread beyond which its weights stream, two batches of eight in flight, and the inputs wait in shared memory: in
// registers, one per weight in flight and sample, they leave room for one block on an SM.  Three float64 samples 3370 -> 75 x
// 213 206 -> 131 us; the one or two batches of a smaller range lose by the inputs' own trip (one sample 1568 -> 30 x 100 8.8 ->
// 12.4 us).
constexpr int kFewStream = 64;

template <typename T, int V>
struct alignas(sizeof(T) * V) Piece {
  T v[V];
};

// `cols` = columns of a block (whole hypercolumns), `lanes` = threads across them, kFewThreads / lanes inputs at a time.
template <typename T, int V, int R, bool STREAM>
__global__ void __launch_bounds__(kFewThreads)
    few_forward_kernel(const T *__restrict__ x, const T *__restrict__ W, const T *__restrict__ bias, T *__restrict__ out,
                       T *partial, int *tickets, int N, int M, int Mc, int cols, int lanes, int range) {
  after_previous();
  __shared__ T s_sum[kFewThreads * V * R];
  __shared__ int s_last;
  T *s_support = s_sum;   // (the sums have been read by then)
  const int c0 = blockIdx.x * cols, width = min(cols, M - c0);
  const int k0 = blockIdx.y * range, k1 = min(N, k0 + range);
  const int groups = kFewThreads / lanes, g = threadIdx.x / lanes, c = (threadIdx.x % lanes) * V;
  T acc[R][V];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int v = 0; v < V; ++v) acc[r][v] = (T)0;
  const bool active = g < groups && c < width;
  if constexpr (STREAM) {
    constexpr int U = 8;
    // inputs in shared memory at a time; each fill begins with the first group of threads again, so a range of several fills that
    // `groups` does not divide is summed in another order than from registers
    constexpr int KT = sizeof(T) * R <= 16 ? 1024 : 512;
    __shared__ T s_x[R][KT];
    for (int t0 = k0; t0 < k1; t0 += KT) {
      const int t1 = min(k1, t0 + KT);
      const T *wp = W + c0 + c;
      auto load = [&](Piece<T, V> (&w)[U], int k) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u * groups < t1) w[u] = *reinterpret_cast<const Piece<T, V> *>(wp + (long)(k + u * groups) * M);
      };
      auto multiply = [&](const Piece<T, V> (&w)[U], int k) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u * groups < t1)
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int v = 0; v < V; ++v) acc[r][v] = fma(s_x[r][k + u * groups - t0], w[u].v[v], acc[r][v]);
      };
      Piece<T, V> a[U], b[U];
      int k = t0 + g;
      if (active) load(a, k);
      if (t0 > k0) __syncthreads();   // the inputs before these have been read
#pragma unroll
      for (int r = 0; r < R; ++r)
        for (int t = threadIdx.x; t < t1 - t0; t += kFewThreads) s_x[r][t] = x[(long)r * N + t0 + t];
      __syncthreads();
      if (active)
        for (; k < t1; k += 2 * U * groups) {
          load(b, k + U * groups);
          multiply(a, k);
          load(a, k + 2 * U * groups);
          multiply(b, k + U * groups);
        }
    }
  } else if (active) {
    constexpr int U = R <= 2 ? 16 : 8;   // (as registers allow with two blocks on an SM: four float32 samples 1568 -> 30 x 100 19.3 -> 17.5 us)
    const T *wp = W + c0 + c;
    for (int k = k0 + g; k < k1; k += U * groups) {
      Piece<T, V> w[U];
      T xv[U][R];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kk = k + u * groups;
        if (kk < k1) {
          w[u] = *reinterpret_cast<const Piece<T, V> *>(wp + (long)kk * M);
#pragma unroll
          for (int r = 0; r < R; ++r) xv[u][r] = __ldg(x + (long)r * N + kk);
        } else {
#pragma unroll
          for (int v = 0; v < V; ++v) w[u].v[v] = (T)0;
#pragma unroll
          for (int r = 0; r < R; ++r) xv[u][r] = (T)0;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int v = 0; v < V; ++v) acc[r][v] = fma(xv[u][r], w[u].v[v], acc[r][v]);
    }
  }
  if (active)
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int v = 0; v < V; ++v) s_sum[(g * R + r) * lanes * V + c + v] = acc[r][v];
  __syncthreads();
  for (int t = threadIdx.x; t < R * width; t += kFewThreads) {
    const int r = t / width, j = t % width;
    T s = s_sum[r * lanes * V + j];
    for (int q = 1; q < groups; ++q) s += s_sum[(q * R + r) * lanes * V + j];
    partial[((long)blockIdx.y * R + r) * M + c0 + j] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(tickets + blockIdx.x, 1) == (int)gridDim.y - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x == 0) tickets[blockIdx.x] = 0;
  for (int t = threadIdx.x; t < R * width; t += kFewThreads) {
    const T *p = partial + (long)(t / width) * M + c0 + t % width;
    T s = (T)0;
#pragma unroll 16
    for (int q = 0; q < (int)gridDim.y; ++q) s += __ldcg(p + (long)q * R * M);
    s_support[t] = s + bias[c0 + t % width];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int t = threadIdx.x >> 5; t < R * (width / Mc); t += kFewThreads / 32) {   // a warp per sample and hypercolumn
    T *v = s_support + t * Mc;   // (width is a multiple of Mc: samples follow one another in whole hypercolumns)
    T mx = -INFINITY;
    for (int j = lane; j < Mc; j += 32) mx = v[j] > mx ? v[j] : mx;
    for (int off = 16; off > 0; off >>= 1) {
      const T o = __shfl_xor_sync(0xffffffffu, mx, off);
      mx = o > mx ? o : mx;
    }
    T sum = (T)0;
    for (int j = lane; j < Mc; j += 32) {
      const T e = sbb_exp(v[j] - mx);
      v[j] = e;
      sum += e;
    }
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const int per = width / Mc;
    T *dst = out + (long)(t / per) * M + c0 + (t % per) * Mc;
    for (int j = lane; j < Mc; j += 32) dst[j] = v[j] / sum;
  }
}

struct FewPlan {
  int vec, cols, lanes, chunks, ranges, range;
  bool stream;
};
template <typename T>
bool few_plan(const void *W, long B, long N, long H, long Mc, FewPlan &p) {
  const long M = H * Mc;
  if (B < 1 || B > kFewSamples || N < 1 || N >= (1l << 30) || M >= (1l << 30)) return false;
  // In float32 the tiled kernel's sums differ in the sixth digit for tens of thousands of inputs, and a layer that trains
  // on its activations amplifies that: those stay with it, and a forward pass does not tell whether a train step follows.
  // What that costs a pure forward pass, N -> 30 x 100, tiled against this kernel: one sample 37.6 and 19.2 us at 8192
  // inputs, 125 and 68 at 30000, 208 and 119 at 55296; four samples 38.0 and 45.3, 128 and 124, 213 and 215.
  if (sizeof(T) == 4 && N > 4096) return false;
  p.vec = 16 / (int)sizeof(T);
  if (M % p.vec != 0 || (reinterpret_cast<uintptr_t>(W) & 15u) != 0) p.vec = 1;
  // whole hypercolumns per block, their start on a vector boundary: a quarter of the threads across them (wider blocks need
  // more ranges to fill the chip, and the last block reads a partial sum per range)
  const long most = (long)kFewThreads * p.vec;
  long hcs = most / 4 / Mc > 0 ? most / 4 / Mc : 1;
  if (hcs > H) hcs = H;
  while (hcs > 1 && (hcs * Mc) % p.vec != 0) --hcs;
  if ((hcs * Mc) % p.vec != 0) {
    if (hcs * Mc != M) p.vec = 1;
    hcs = kFewThreads / Mc / 4 > 0 ? kFewThreads / Mc / 4 : 1;
    if (hcs > H) hcs = H;
  }
  const long cols = hcs * Mc;
  if (cols > (long)kFewThreads * p.vec) return false;
  p.cols = (int)cols;
  p.lanes = (int)((cols + p.vec - 1) / p.vec);
  p.chunks = (int)((H + hcs - 1) / hcs);
  // two blocks per SM, at least sixteen inputs per thread
  const long groups = kFewThreads / p.lanes;
  long ranges = (2 * sm_count() + p.chunks - 1) / p.chunks;
  const long most_ranges = (N + 16 * groups - 1) / (16 * groups);
  if (ranges > most_ranges) ranges = most_ranges;
  if (ranges > 64) ranges = 64;
  p.range = (int)((N + ranges - 1) / ranges);
  p.ranges = (int)((N + p.range - 1) / p.range);
  p.stream = p.range / groups > kFewStream;
  return true;
}

}  // namespace

template <typename T>
bool few_samples(const T *W, long B, long N, long H, long Mc, size_t *scratch_elems) {
  FewPlan p;
  if (!few_plan<T>(W, B, N, H, Mc, p)) return false;
  *scratch_elems = (size_t)p.ranges * (size_t)B * (size_t)(H * Mc);
  return true;
}
template bool few_samples<float>(const float *, long, long, long, long, size_t *);
template bool few_samples<double>(const double *, long, long, long, long, size_t *);

template <typename T>
cudaError_t launch_few_forward(const T *x, const T *W, const T *bias, T *out, long B, long N, long H, long Mc, T *partial,
                               int *tickets, cudaStream_t st) {
  FewPlan p;
  if (!few_plan<T>(W, B, N, H, Mc, p)) return cudaErrorNotSupported;
  const dim3 grid((unsigned)p.chunks, (unsigned)p.ranges);
  constexpr int V = 16 / (int)sizeof(T);
#define SBB_FEW(VV, R, S) \
  launch_next(few_forward_kernel<T, VV, R, S>, grid, kFewThreads, 0, st, x, W, bias, out, partial, tickets, (int)N, (int)(H * Mc), (int)Mc, \
              p.cols, p.lanes, p.range)
#define SBB_FEW_R(R) \
  if (p.vec == 1 && p.stream) SBB_FEW(1, R, true); \
  else if (p.vec == 1) SBB_FEW(1, R, false); \
  else if (p.stream) SBB_FEW(V, R, true); \
  else SBB_FEW(V, R, false)
  if (B == 1) {
    SBB_FEW_R(1);
  } else if (B == 2) {
    SBB_FEW_R(2);
  } else if (B == 3) {
    SBB_FEW_R(3);
  } else {
    SBB_FEW_R(4);
  }
#undef SBB_FEW_R
#undef SBB_FEW
  count_launches(1);
  return cudaGetLastError();
}
template cudaError_t launch_few_forward<float>(const float *, const float *, const float *, float *, long, long, long, long,
                                               float *, int *, cudaStream_t);
template cudaError_t launch_few_forward<double>(const double *, const double *, const double *, double *, long, long, long, long,
                                                double *, int *, cudaStream_t);

}  // namespace sbb
