// Layers with few units (the 10-class output layer above all): both halves of a step as one launch each.
//
// Such a layer is nothing but latency: 3000 x 10 weights are 120 kB, the whole step some 2 MB of traffic and 15 MFLOP.
// The tiled contraction kernels spend it on 128-column tiles that are nine tenths padding and on one dependent round
// trip to memory per k-slab, and the column sums, the reduction with the softmax and the bias are launches of their
// own: the 3000 -> 10 layer at batch 128 took 20.4 + 5.7 us for the forward pass and 31.0 + 2 x 2.6 us for the train
// step.  Here every thread has all its loads of the inputs in flight at once.
#include "sbb_kernels.cuh"
#include "sbb_launch.cuh"
#include "sbb_math.cuh"

#include <cooperative_groups.h>

namespace sbb {

void count_launches(int n);   // sbb_kernels.cu

namespace {

inline cudaError_t launched() {
  count_launches(1);
  return cudaGetLastError();
}

// ----------------------------------------------------------------------------
// out[b, :] = softmax per hypercolumn of (x[b, :] W + bias), M <= MP units.  WARPS warps share R samples: each thread
// takes every (32 * WARPS)-th input, keeps R x MP sums, and shuffles and one pass through shared memory add them up.
// Where the samples fill few SMs a cluster of up to eight blocks (gridDim.y) shares the inputs of R samples, and a single sample
// keeps four inputs' weights in flight a thread: a step of the layer 30000 -> 10 at batch 64 72 -> 46 us, 9001 -> 10 at batch 4
// 17.5 -> 12.7 (as long as the calling thread takes for the two launches).
// ----------------------------------------------------------------------------
template <typename T, int MP, int R, int WARPS>
__global__ void __launch_bounds__(256)
    narrow_forward_kernel(const T *__restrict__ x, const T *__restrict__ W, const T *__restrict__ bias, T *__restrict__ out,
                          long B, int N, int M, int Mc) {
  after_previous();
  namespace cg = cooperative_groups;
  constexpr int SETS = 8 / WARPS;   // groups of R samples per block
  __shared__ T part[8][R][MP], support[SETS][R][MP];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int set = wid / WARPS;
  const int ranks = WARPS == 8 ? (int)gridDim.y : 1, rank = WARPS == 8 ? (int)blockIdx.y : 0;   // of the cluster
  const int span = (N + ranks - 1) / ranks, n0 = rank * span, n1 = min(N, n0 + span);           // this block's inputs
  const long b0 = ((long)blockIdx.x * SETS + set) * R;
  T acc[R][MP];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < MP; ++j) acc[r][j] = (T)0;
  constexpr int STEP = 32 * WARPS;
  constexpr int ROW = MP * (int)sizeof(T);
  constexpr int U = R > 2 || ROW > 128 ? 1 : R == 1 ? (256 / ROW < 4 ? 256 / ROW : 4) : ROW > 64 ? 1 : ROW > 32 ? 2 : 4;   // inputs in flight per thread, as registers allow
  for (int k0 = n0 + (wid % WARPS) * 32 + lane; k0 < n1; k0 += U * STEP) {
    T xv[U][R], w[U][MP];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * STEP;
#pragma unroll
      for (int r = 0; r < R; ++r) xv[u][r] = k < n1 && b0 + r < B ? x[(b0 + r) * N + k] : (T)0;
#pragma unroll
      for (int j = 0; j < MP; ++j) w[u][j] = k < n1 && j < M ? W[(long)k * M + j] : (T)0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int j = 0; j < MP; ++j) acc[r][j] = fma(xv[u][r], w[u][j], acc[r][j]);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int j = 0; j < MP; ++j) {
      T v = acc[r][j];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (lane == 0) part[wid][r][j] = v;
    }
  __syncthreads();
  // the support of (sample, unit), then the softmax of its hypercolumn
  for (int t = threadIdx.x; t < SETS * R * M; t += 256) {
    const int s = t / (R * M), r = t / M % R, j = t % M;
    T v = part[s * WARPS][r][j];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) v += part[s * WARPS + w][r][j];
    support[s][r][j] = ranks > 1 ? v : v + bias[j];
  }
  if (WARPS == 8 && ranks > 1) {
    cg::this_cluster().sync();
    if (rank != 0) {
      cg::this_cluster().sync();   // (the first block still reads this one's sums)
      return;
    }
    T v = (T)0;
    const int t = threadIdx.x, r = t / M, j = t % M;
    if (t < R * M) {
      T d[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) d[q] = q < ranks ? *cg::this_cluster().map_shared_rank(&support[0][r][j], q) : (T)0;
#pragma unroll
      for (int q = 0; q < 8; ++q) v += d[q];
    }
    cg::this_cluster().sync();
    if (t < R * M) support[0][r][j] = v + bias[j];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < SETS * R * M; t += 256) {
    const int s = t / (R * M), r = t / M % R, j = t % M;
    const long b = ((long)blockIdx.x * SETS + s) * R + r;
    if (b >= B) continue;
    const T *v = support[s][r] + j / Mc * Mc;
    T mx = v[0];
    for (int q = 1; q < Mc; ++q) mx = v[q] > mx ? v[q] : mx;
    T sum = (T)0;
    for (int q = 0; q < Mc; ++q) sum += sbb_exp(v[q] - mx);
    out[b * M + j] = sbb_exp(v[j % Mc] - mx) / sum;
  }
}

// ----------------------------------------------------------------------------
// The whole train step but the mask: Ci, Cj, Cij, weights, and (kbi != null) the regularised bias.  A block owns 32
// inputs: lane = input, warp = every eighth sample; the targets pass through shared memory, where all lanes read the same
// word.  Every block forms the new Cj for itself (it reads all targets anyway); the old one stays in place until the
// last block writes the new one and the bias.  CL > 1: a cluster of CL blocks shares the 32 inputs, each takes a part of the
// batch, and the first adds up their sums out of shared memory.  One block's pass over the batch is a chain of loads: 664 -> 2
// x 8 float64 units at batch 5453 took 89 us on 21 of 148 SMs, 29 us in clusters of four.
// ----------------------------------------------------------------------------
template <typename T, int MP>
struct NarrowTrain {
  static constexpr int STAGE = sizeof(T) * MP <= 128 ? 128 : 64;   // samples of the targets in shared memory at a time
  static constexpr int CH = sizeof(T) == 4 && MP > 16 ? 16 : (sizeof(T) == 8 ? 8 : MP);   // units reduced at a time
};

template <typename T, int MP, int CL>
__global__ void __launch_bounds__(256)
    narrow_train_kernel(const T *__restrict__ x, const T *__restrict__ y, long B, int N, int M, int H, int Mc, T *Ci, T *Cj,
                        T *Cij, T *W, const uint8_t *__restrict__ wmask, TraceParams<T> p, BiasParams<T> nb, int *ticket) {
  after_previous();
  constexpr int STAGE = NarrowTrain<T, MP>::STAGE, CH = NarrowTrain<T, MP>::CH;
  constexpr int NCH = MP / CH, E = 32 * CH / 256;   // outputs per thread: NCH chunks of E
  namespace cg = cooperative_groups;
  const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
  const long part = CL > 1 ? (B + CL - 1) / CL : B, b0 = rank * part, b1 = b0 + part < B ? b0 + part : B;   // its samples
  struct Sums {
    T xy[32][MP], x[32], y[MP];
  };
  __shared__ Sums sums[1];   // this block's, for the cluster's first
  __shared__ __align__(16) T ys[STAGE][MP];
  __shared__ T red[8][32][CH + 1], redx[8][32];
  __shared__ T cj_new[MP], ci_new[32];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long i0 = (long)(blockIdx.x / CL) * 32, i = i0 + lane;
  const int rows = (int)(N - i0 < 32 ? N - i0 : 32);
  constexpr int U = STAGE / 8;             // a warp's samples of a stage
  constexpr int UY = STAGE * MP / 256;     // a thread's targets of a stage
  T xv[U], yv[UY];
  auto fetch = [&](long c0) {
#pragma unroll
    for (int u = 0; u < U; ++u) xv[u] = c0 + wid + 8 * u < b1 && i < N ? x[(c0 + wid + 8 * u) * N + i] : (T)0;
#pragma unroll
    for (int u = 0; u < UY; ++u) {
      const int t = threadIdx.x + 256 * u, b = t / MP, j = t % MP;
      yv[u] = c0 + b < b1 && j < M ? y[(c0 + b) * M + j] : (T)0;
    }
  };
  fetch(b0);
  // the old state too is on its way before the sums are formed
  T old[NCH][E], c_old = (T)0;
  uint8_t bit[NCH][E];
#pragma unroll
  for (int c = 0; c < NCH; ++c)
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int t = threadIdx.x + 256 * e, r = t / CH, j = c * CH + t % CH;
      const bool in = r < rows && j < M;
      old[c][e] = in ? Cij[(i0 + r) * M + j] : (T)0;
      bit[c][e] = in && wmask != nullptr ? wmask[(i0 + r) * H + j / Mc] : (uint8_t)1;
    }
  if (threadIdx.x < 32) {
    if ((int)threadIdx.x < rows) c_old = Ci[i0 + threadIdx.x];
  } else if ((int)threadIdx.x - 32 < M) {
    c_old = Cj[threadIdx.x - 32];
  }
  T acc[MP], sx = (T)0, sy = (T)0;
#pragma unroll
  for (int j = 0; j < MP; ++j) acc[j] = (T)0;
  for (long c0 = b0; c0 < b1; c0 += STAGE) {
    const int len = (int)(b1 - c0 < STAGE ? b1 - c0 : STAGE);
    if (c0 > b0) __syncthreads();   // the previous stage has been read
    T xs[U];
#pragma unroll
    for (int u = 0; u < U; ++u) xs[u] = xv[u];
#pragma unroll
    for (int u = 0; u < UY; ++u) (&ys[0][0])[threadIdx.x + 256 * u] = yv[u];
    __syncthreads();
    if (c0 + STAGE < b1) fetch(c0 + STAGE);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      sx += xs[u];   // (samples past the end are zero)
#pragma unroll
      for (int j = 0; j < MP; ++j) acc[j] = fma(xs[u], ys[wid + 8 * u][j], acc[j]);
    }
    // column sums of the targets: 256 / MP threads per column
    for (int b = threadIdx.x / MP; b < len; b += 256 / MP) sy += ys[b][threadIdx.x % MP];
  }
  // the sum over the cluster of a value at the same place of every block's `sums`
  auto total = [&](const T *mine) {
    T v[CL];
#pragma unroll
    for (int q = 0; q < CL; ++q) v[q] = *cg::this_cluster().map_shared_rank(mine, q);
    T t = v[0];
#pragma unroll
    for (int q = 1; q < CL; ++q) t += v[q];
    return t;
  };
  redx[wid][lane] = sx;
  __syncthreads();
  T *ysum = &ys[0][0];   // [256 / MP][MP]
  ysum[threadIdx.x] = sy;
  __syncthreads();
  if constexpr (CL > 1) {
    if (threadIdx.x < 32) {
      T s = redx[0][threadIdx.x];
#pragma unroll
      for (int w = 1; w < 8; ++w) s += redx[w][threadIdx.x];
      sums[0].x[threadIdx.x] = s;
    } else if ((int)threadIdx.x - 32 < MP) {
      const int j = threadIdx.x - 32;
      T s = ysum[j];
#pragma unroll 4
      for (int k = 1; k < 256 / MP; ++k) s += ysum[k * MP + j];
      sums[0].y[j] = s;
    }
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      if (c > 0) __syncthreads();
#pragma unroll
      for (int j = 0; j < CH; ++j) red[wid][lane][j] = acc[c * CH + j];
      __syncthreads();
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int t = threadIdx.x + 256 * e, r = t / CH;
        T s = red[0][r][t % CH];
#pragma unroll
        for (int w = 1; w < 8; ++w) s += red[w][r][t % CH];
        sums[0].xy[r][c * CH + t % CH] = s;
      }
    }
    cg::this_cluster().sync();
    if (rank != 0) {
      cg::this_cluster().sync();   // (the first block still reads this one's sums)
      return;
    }
  }
  if (threadIdx.x < 32) {
    if ((int)threadIdx.x < rows) {
      T s;
      if constexpr (CL > 1) {
        s = total(&sums[0].x[threadIdx.x]);
      } else {
        s = redx[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < 8; ++w) s += redx[w][threadIdx.x];
      }
      const T c = trace_ema(c_old, s, p);
      Ci[i0 + threadIdx.x] = c;
      ci_new[threadIdx.x] = c;
    }
  } else if ((int)threadIdx.x - 32 < M) {
    const int j = threadIdx.x - 32;
    T s;
    if constexpr (CL > 1) {
      s = total(&sums[0].y[j]);
    } else {
      s = ysum[j];
#pragma unroll 4
      for (int k = 1; k < 256 / MP; ++k) s += ysum[k * MP + j];
    }
    cj_new[j] = trace_ema(c_old, s, p);
  }
  if constexpr (CL > 1) __syncthreads();
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    if constexpr (CL == 1) {
      if (c > 0) __syncthreads();
#pragma unroll
      for (int j = 0; j < CH; ++j) red[wid][lane][j] = acc[c * CH + j];
      __syncthreads();
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int t = threadIdx.x + 256 * e, r = t / CH, j = c * CH + t % CH;
      if (r >= rows || j >= M) continue;
      T s;
      if constexpr (CL > 1) {
        s = total(&sums[0].xy[r][j]);
      } else {
        s = red[0][r][t % CH];
#pragma unroll
        for (int w = 1; w < 8; ++w) s += red[w][r][t % CH];
      }
      const T v = trace_ema(old[c][e], s, p);
      const T ci = ci_new[r], cj = cj_new[j];
      const bool on = !(ci < p.cthr) && !(cj < p.cthr) && bit[c][e] != 0;
      const long at = (i0 + r) * M + j;
      Cij[at] = v;
      W[at] = on ? log_ratio(v, ci, cj, p.cthr4) : (T)0;
    }
  }
  if constexpr (CL > 1) cg::this_cluster().sync();
  // the block that finishes last: no other one needs the old Cj any more (the others of its cluster have long read it)
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(ticket, 1) == (int)gridDim.x / CL - 1;
  }
  __syncthreads();
  if (!s_last) return;
  if (threadIdx.x == 0) *ticket = 0;
  if ((int)threadIdx.x < M) {
    const T cj = cj_new[threadIdx.x];
    Cj[threadIdx.x] = cj;
    if (nb.kbi != nullptr) bias_regularized(nb.bias[threadIdx.x], nb.kbi[threadIdx.x], cj, p.cthr, nb.khalf, nb.pmin4, nb.k, nb.taubdt);
  }
}

// Samples a thread keeps sums for: 64 registers of them in float32; one in float64 (narrow_forward admits no batch that would
// share its reads of the weights).
constexpr int narrow_samples(long M, size_t elem) { return elem == 8 ? 1 : M <= 8 ? 8 : M <= 16 ? 4 : 2; }

template <typename T, int MP>
cudaError_t forward_mp(const T *x, const T *W, const T *bias, T *out, long B, long N, long M, long Mc, cudaStream_t st) {
  constexpr int RMAX = narrow_samples(MP, sizeof(T));
  // few samples: one per block (or warp), so that all SMs take part; more of them share each read of the weights
  const long sms = sm_count(), per = (B + 2 * sms - 1) / (2 * sms);
  unsigned ranks = B * 8 <= sms ? 8 : B * 4 <= sms ? 4 : B * 2 <= sms ? 2 : 1;   // (one sample a block then, on SMs of their own)
  while (ranks > 1 && N < 512 * (long)ranks) ranks /= 2;
  const bool alone = narrow_alone(B, N);
#define SBB_NARROW_FWD(R)                                                                                              \
  do {                                                                                                                 \
    if (alone)                                                                                                         \
      launch_next(narrow_forward_kernel<T, MP, R, 1>, (unsigned)((B + 8 * R - 1) / (8 * R)), 256, 0, st, x, W, bias, out, B, (int)N, (int)M, (int)Mc); \
    else if (ranks > 1)                                                                                                \
      launch_clusters(narrow_forward_kernel<T, MP, R, 8>, dim3((unsigned)((B + R - 1) / R), ranks), dim3(1, ranks, 1), 256, 0, st, x, W, bias, out, B, (int)N, (int)M, (int)Mc); \
    else                                                                                                               \
      launch_next(narrow_forward_kernel<T, MP, R, 8>, (unsigned)((B + R - 1) / R), 256, 0, st, x, W, bias, out, B, (int)N, (int)M, (int)Mc); \
  } while (0)
  if (per <= 1 || RMAX == 1) SBB_NARROW_FWD(1);
  else if (per <= 2 || RMAX == 2) SBB_NARROW_FWD((RMAX < 2 ? RMAX : 2));
  else if (per <= 4 || RMAX == 4) SBB_NARROW_FWD((RMAX < 4 ? RMAX : 4));
  else SBB_NARROW_FWD(RMAX);
#undef SBB_NARROW_FWD
  return launched();
}

}  // namespace

// Up to 32 units; beyond that the tiles of the contraction kernels are full enough.  The forward pass reads all weights
// once per block of samples: with very many samples that is more L2 traffic than the tiled kernels cause.
bool narrow_layer(long N, long M) { return M <= 32 && N < (1l << 30); }
// Not enough inputs to share among the warps of a block, or samples enough without (500 -> 31 at batch 128, a step: 37 us alone,
// 25 shared).
bool narrow_alone(long B, long N) { return N <= 64 || (N <= 512 && B > 2 * sm_count()); }
bool narrow_forward(long B, long N, long M, size_t elem) {
  // float64: a block of one sample reads all weights 8 bytes at a time, rows apart, and the cost grows with samples x inputs; the
  // tiles of the FP64 tensor-core kernel read them once but wait for more inputs one after the other.  Where the line lies
  // depends on the row's length: a unit costs twice as much in rows of 64 bytes (8 units) as in those of 72 to 88, in rows of 128
  // (16 units) four times.  Measured, us, here and in tiles.  7 units: 20000 inputs at batch 8 6 and 22, at 256 29 and 34; 30001 at 256 43 and 44.  8
  // units: 8192 at 64 12.9 and 15.5, 3000 at 180 16.4 and 10.5, 8192 at 256 38 and 15.  10 units: 20000 at 8 9.1 and 20.4, 8192 at 128
  // 16.4 and 15.4, at 256 22.9 and 15.6.  11 units: 20000 at 32 15.5 and 23.3, 3000 at 256 13.0 and 12.2.  12 to 15 units: 1000 at
  // 128 6.4 to 7.3 and 7.7 to 8.5, 8192 at 64 14.4 to 16.4 and 15.5 to 17.1, 3000 at 128 11.5 to 13.2 and 10.8 to 11.8.  16 units:
  // 1000 at 64 12.2 and 7.7.  Up to four samples the other way is the kernel for few samples: 5000 -> 7 4.5 here and 6.5 there, 5000
  // -> 11 5.7 and 9.1, 1000 -> 11 5.4 and 4.6, 1000 -> 15 6.4 and 5.6, 20000 -> 10 9.0 and 8.1.
  if (elem == 8) {
    if (!narrow_layer(N, M) || M > 15 || B > 256) return false;
    if (B <= kFewSamples) return M <= 7 ? N <= 32768 : M <= 11 && N <= 8192;
    return B * N <= (M <= 7 ? 1l << 23 : M == 8 ? 1l << 19 : M <= 10 ? 1l << 20 : M == 11 ? 5l << 17 : B <= 64 ? 1l << 19 : 1l << 17);
  }
  const long r = narrow_samples(M, 4);
  return narrow_layer(N, M) && ((B + r - 1) / r) * N * M <= (1l << 28);
}

template <typename T>
cudaError_t launch_narrow_forward(const T *x, const T *W, const T *bias, T *out, long B, long N, long M, long Mc,
                                  cudaStream_t st) {
  if (M <= 8) return forward_mp<T, 8>(x, W, bias, out, B, N, M, Mc, st);
  if constexpr (sizeof(T) == 8) {
    return M <= 16 ? forward_mp<T, 16>(x, W, bias, out, B, N, M, Mc, st) : cudaErrorNotSupported;
  } else {
    if (M <= 16) return forward_mp<T, 16>(x, W, bias, out, B, N, M, Mc, st);
    return forward_mp<T, 32>(x, W, bias, out, B, N, M, Mc, st);
  }
}
template cudaError_t launch_narrow_forward<float>(const float *, const float *, const float *, float *, long, long, long, long,
                                                  cudaStream_t);
template cudaError_t launch_narrow_forward<double>(const double *, const double *, const double *, double *, long, long, long,
                                                   long, cudaStream_t);

template <typename T>
cudaError_t launch_narrow_train(const T *x, const T *y, long B, long N, long M, long H, long Mc, T *Ci, T *Cj, T *Cij, T *W,
                                const uint8_t *wmask, TraceParams<T> p, BiasParams<T> nb, int *ticket, cudaStream_t st) {
  const unsigned blocks = (unsigned)((N + 31) / 32);
  // Clusters where they find SMs of their own and every block a stage of samples: 664 inputs, float64, batch 5453 89 -> 29 us,
  // 300 inputs, float32, batch 1024 14.3 -> 6.8; without that room they lose (3000 inputs at batch 1024 21 -> 46 in eights).
  const long stages = (B + 127) / 128;
  const long sms = sm_count();
  const int cl = blocks * 8 <= sms && stages >= 8 ? 8 : blocks * 4 <= sms && stages >= 4 ? 4 : blocks * 2 <= sms && stages >= 4 ? 2 : 1;
#define SBB_NARROW_TRAIN(MP)                                                                                            \
  do {                                                                                                                  \
    if (cl == 8)                                                                                                        \
      launch_clusters(narrow_train_kernel<T, MP, 8>, blocks * 8, dim3(8, 1, 1), 256, 0, st, x, y, B, (int)N, (int)M, (int)H, (int)Mc, Ci, Cj, Cij, W, wmask, p, nb, ticket); \
    else if (cl == 4)                                                                                                   \
      launch_clusters(narrow_train_kernel<T, MP, 4>, blocks * 4, dim3(4, 1, 1), 256, 0, st, x, y, B, (int)N, (int)M, (int)H, (int)Mc, Ci, Cj, Cij, W, wmask, p, nb, ticket); \
    else if (cl == 2)                                                                                                   \
      launch_clusters(narrow_train_kernel<T, MP, 2>, blocks * 2, dim3(2, 1, 1), 256, 0, st, x, y, B, (int)N, (int)M, (int)H, (int)Mc, Ci, Cj, Cij, W, wmask, p, nb, ticket); \
    else                                                                                                                \
      launch_next(narrow_train_kernel<T, MP, 1>, blocks, 256, 0, st, x, y, B, (int)N, (int)M, (int)H, (int)Mc, Ci, Cj, Cij, W, wmask, p, nb, ticket); \
  } while (0)
  if (M <= 8) SBB_NARROW_TRAIN(8);
  else if (M <= 16) SBB_NARROW_TRAIN(16);
  else SBB_NARROW_TRAIN(32);
#undef SBB_NARROW_TRAIN
  return launched();
}
template cudaError_t launch_narrow_train<float>(const float *, const float *, long, long, long, long, long, float *, float *,
                                                float *, float *, const uint8_t *, TraceParams<float>, BiasParams<float>, int *,
                                                cudaStream_t);
template cudaError_t launch_narrow_train<double>(const double *, const double *, long, long, long, long, long, double *,
                                                 double *, double *, double *, const uint8_t *, TraceParams<double>,
                                                 BiasParams<double>, int *, cudaStream_t);

}  // namespace sbb
