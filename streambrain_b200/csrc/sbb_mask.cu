// Structural plasticity: the mutual-information score of every connection of one hypercolumn, the swaps of silent
// and active connections it decides, and the weights of the rows a swap touched.
#include "sbb_kernels.cuh"
#include "sbb_launch.cuh"
#include "sbb_math.cuh"

#include <math.h>
#include <type_traits>

namespace sbb {

void count_launches(int n);   // sbb_kernels.cu
static inline cudaError_t launched(int n = 1) {
  count_launches(n);
  return cudaGetLastError();
}

template <typename T>
struct Pick {
  T v;
  long i;  // -1 = empty
};
// Maximum with ties to the larger index / minimum with ties to the larger index:
// the outcome of a front-to-back scan that replaces on >= (resp. <=).
template <typename T>
__device__ __forceinline__ Pick<T> pick_max(Pick<T> a, Pick<T> b) {
  if (b.i < 0) return a;
  if (a.i < 0) return b;
  return (b.v > a.v || (b.v == a.v && b.i > a.i)) ? b : a;
}
template <typename T>
__device__ __forceinline__ Pick<T> pick_min(Pick<T> a, Pick<T> b) {
  if (b.i < 0) return a;
  if (a.i < 0) return b;
  return (b.v < a.v || (b.v == a.v && b.i > a.i)) ? b : a;
}
template <typename T>
__device__ __forceinline__ Pick<T> shfl_pick(Pick<T> p, int off) {
  Pick<T> o;
  o.v = __shfl_xor_sync(0xffffffffu, p.v, off);
  o.i = __shfl_xor_sync(0xffffffffu, p.i, off);
  return o;
}

// Single CTA.  Every iteration scans all rows: among silent connections
// (mask 0) the highest score, among active ones (mask 1) the lowest, both with
// the reference's sequential-scan semantics: ties go to the last index, and a
// NaN score can only be selected when it belongs to the first candidate of its
// class (a scan never replaces its holder with a NaN, nor a NaN holder at all).
template <typename T>
__global__ void __launch_bounds__(1024)
    mask_swap_kernel(uint8_t *wmask, const T *__restrict__ nom, int *csum, long N, long M, long H, long Mc, long h,
                     long iterations, T *rewrite_w,
                     const uint8_t *__restrict__ old_col, const T *__restrict__ Ci, const T *__restrict__ Cj,
                     const T *__restrict__ Cij, T cthr, T cthr4) {
  __shared__ Pick<T> s_max[32], s_min[32];
  __shared__ long s_first0[32], s_first1[32];
  __shared__ int s_done;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if (threadIdx.x == 0) s_done = 0;
  __syncthreads();
  for (long it = 0; it < iterations; ++it) {
    Pick<T> bmax{(T)0, -1}, bmin{(T)0, -1};
    long first0 = N, first1 = N;
    for (long j = threadIdx.x; j < N; j += blockDim.x) {
      const uint8_t m = wmask[j * H + h];
      const T sc = (T)((double)nom[j] / (1.0 + (double)csum[j]));
      if (m == 0) {
        first0 = j < first0 ? j : first0;
        if (sc == sc) bmax = pick_max(bmax, Pick<T>{sc, j});
      } else if (m == 1) {
        first1 = j < first1 ? j : first1;
        if (sc == sc) bmin = pick_min(bmin, Pick<T>{sc, j});
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      bmax = pick_max(bmax, shfl_pick(bmax, off));
      bmin = pick_min(bmin, shfl_pick(bmin, off));
      const long f0 = __shfl_xor_sync(0xffffffffu, first0, off);
      const long f1 = __shfl_xor_sync(0xffffffffu, first1, off);
      first0 = f0 < first0 ? f0 : first0;
      first1 = f1 < first1 ? f1 : first1;
    }
    if (lane == 0) {
      s_max[wid] = bmax;
      s_min[wid] = bmin;
      s_first0[wid] = first0;
      s_first1[wid] = first1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < nwarps; ++w) {
        bmax = pick_max(bmax, s_max[w]);
        bmin = pick_min(bmin, s_min[w]);
        first0 = s_first0[w] < first0 ? s_first0[w] : first0;
        first1 = s_first1[w] < first1 ? s_first1[w] : first1;
      }
      long imax0 = N, imin1 = N;
      T vmax0 = (T)0, vmin1 = (T)0;
      if (first0 < N) {
        const T sf = (T)((double)nom[first0] / (1.0 + (double)csum[first0]));
        if (sf != sf) { imax0 = first0; vmax0 = sf; }
        else { imax0 = bmax.i; vmax0 = bmax.v; }
      }
      if (first1 < N) {
        const T sf = (T)((double)nom[first1] / (1.0 + (double)csum[first1]));
        if (sf != sf) { imin1 = first1; vmin1 = sf; }
        else { imin1 = bmin.i; vmin1 = bmin.v; }
      }
      if (imax0 == N || imin1 == N || vmax0 < vmin1) {
        s_done = 1;
      } else {
        wmask[imax0 * H + h] = 1;
        wmask[imin1 * H + h] = 0;
        csum[imax0] += 1;
        csum[imin1] -= 1;
      }
    }
    __syncthreads();
    if (s_done) break;
  }
  if (rewrite_w == nullptr) return;
  // rows whose mask bit changed get new weights in hypercolumn h (at most 2 * iterations rows)
  for (long j = threadIdx.x; j < N; j += blockDim.x) {
    const uint8_t now = wmask[j * H + h];
    if (now == old_col[j]) continue;
    const T ci = Ci[j];
    for (long jj = 0; jj < Mc; ++jj) {
      const long col = h * Mc + jj;
      const T cj = Cj[col];
      T v = (T)0;
      if (now != 0 && !(ci < cthr) && !(cj < cthr)) v = log_ratio(Cij[j * M + col], ci, cj, cthr4);
      rewrite_w[j * M + col] = v;
    }
  }
}

// ---- one launch per mask update ------------------------------------------------------------
// Only the two rows of a swap change their score, so the row chosen in iteration t is always among the t+1 best
// of its class in the initial ordering or a row moved by an earlier swap.  Every block scores its rows; the block
// that finishes last lists the `iterations` best silent rows (highest score, ties to the larger index) and the
// `iterations` worst active rows, and one warp applies the swaps to them in registers.
//
// Latency is what bounds it (the scores of 1568 rows are 0.6 MB of the trace matrix), and with it the code: most of it
// runs once per launch, from a cold instruction cache, so loops over logarithms are not unrolled.
//
// Scores are mapped to unsigned keys whose integer order is the class order (silent rows: score
// descending first = larger key; active rows: the complement); equal keys order by the row index (the reference's
// scans keep the last of equal scores).  A swap moves a row between two classes, so its two keys are computed once.
//
// NaN scores follow the reference's front-to-back scan: the scan's first row of a class holds the
// pick until a row compares better, and nothing compares better than NaN, so a class whose
// lowest-index row has a NaN score picks that row; a NaN score anywhere else is never picked.
constexpr int kMaskThreads = 512;         // 98 blocks score the 1568 rows of a small layer; 49 of 1024 threads left SMs idle
constexpr int kMaskWarps = kMaskThreads / 32;
constexpr int kSwapMaxIter = 32;          // longest list
constexpr int kGroups = 32;               // groups of rows whose best keys bound the lists
constexpr int kTopSlots = kMaskThreads / 2;   // rows of a class above the bound that are ranked in shared memory
constexpr uint32_t kNoRow = 0xFFFFFFFFu;

template <typename T>
__device__ __forceinline__ T swap_score(T nom, int csum) {
  return (T)((double)nom / (1.0 + (double)csum));
}

// Order-preserving keys: a < b  <=>  key(a) < key(b) for non-NaN scores (-0 counts as +0).
// Key 0 is never produced by a score and marks an empty slot, also after complementing.
template <typename T>
struct ScoreKey;
template <>
struct ScoreKey<float> {
  typedef uint32_t type;
  static __device__ __forceinline__ type make(float v) {
    const uint32_t u = __float_as_uint(v == 0.f ? 0.f : v);
    return (u >> 31) ? ~u : (u | 0x80000000u);
  }
  static __device__ __forceinline__ float value(type k) {
    return __uint_as_float((k >> 31) ? (k ^ 0x80000000u) : ~k);
  }
  static __device__ __forceinline__ type warp_max(type k) { return __reduce_max_sync(0xffffffffu, k); }
};
template <>
struct ScoreKey<double> {
  typedef unsigned long long type;
  static __device__ __forceinline__ type make(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v == 0.0 ? 0.0 : v);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
  }
  static __device__ __forceinline__ double value(type k) {
    return __longlong_as_double((long long)((k >> 63) ? (k ^ 0x8000000000000000ull) : ~k));
  }
  static __device__ __forceinline__ type warp_max(type k) {
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0u);
    return ((type)hi << 32) | lo;
  }
};
// The top 32 bits of a key (never 0).
__device__ __forceinline__ uint32_t filter_key(uint32_t k) { return k; }
__device__ __forceinline__ uint32_t filter_key(unsigned long long k) { return (uint32_t)(k >> 32); }
// Class key: maximum = first in the class order.  cls 0 (silent): highest score; cls 1 (active): lowest.
template <typename T>
__device__ __forceinline__ typename ScoreKey<T>::type class_key(int cls, T v) {
  const typename ScoreKey<T>::type k = ScoreKey<T>::make(v);
  return cls == 0 ? k : ~k;
}
template <typename T>
__device__ __forceinline__ T class_key_value(int cls, typename ScoreKey<T>::type k) {
  return ScoreKey<T>::value(cls == 0 ? k : ~k);
}


__host__ __device__ static inline size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

// Scratch layout: [header][score N x T][active count N x int][filter key N x uint32][old mask column N bytes]
// [best filter keys of both classes per block of rows].
// The header sits first so that it stays in place when layers of several sizes share one work area: it is zero
// between launches.
struct MaskHeader {
  int ticket, nan;
  unsigned long long best[2][kGroups];   // per class: best filter key of every group of rows
};
static constexpr size_t kMaskHeaderBytes = (sizeof(MaskHeader) + 255) & ~(size_t)255;
size_t mask_scratch_bytes(long N, size_t elem) {
  return kMaskHeaderBytes + align256((size_t)N * elem) + 2 * align256((size_t)N * sizeof(int)) + align256((size_t)N) +
         (size_t)((N + kMaskWarps - 1) / kMaskWarps) * sizeof(uint2);
}
cudaError_t mask_scratch_init(void *scratch, cudaStream_t st) { return cudaMemsetAsync(scratch, 0, kMaskHeaderBytes, st); }

template <typename T>
struct MaskScratch {
  MaskHeader *header;
  T *score;
  int *csum;
  uint32_t *filter;
  uint8_t *old_col;
  uint2 *block_best;
  __host__ __device__ MaskScratch(void *scratch, long N) {
    unsigned char *p = static_cast<unsigned char *>(scratch);
    header = reinterpret_cast<MaskHeader *>(p);
    p += kMaskHeaderBytes;
    score = reinterpret_cast<T *>(p);
    p += align256((size_t)N * sizeof(T));
    csum = reinterpret_cast<int *>(p);
    p += align256((size_t)N * sizeof(int));
    filter = reinterpret_cast<uint32_t *>(p);
    p += align256((size_t)N * sizeof(uint32_t));
    old_col = p;
    p += align256((size_t)N);
    block_best = reinterpret_cast<uint2 *>(p);
  }
};

template <typename T>
struct MaskArgs {
  uint8_t *wmask;
  const T *weights, *Ci, *Cj, *Cij;
  T *rewrite_w;
  T cthr, cthr4;
  long N, M, H, Mc, h;
  int iterations;
  int width;       // lanes per row
  int block_rows, rows_log2;   // rows per block, a power of two
  MaskScratch<T> ms;
};

template <typename T>
struct TopShared {
  typename ScoreKey<T>::type key[2][kTopSlots];
  T nom[2][kTopSlots];
  uint32_t row[2][kTopSlots];
  int cs[2][kTopSlots], count[2], blocks, block[kTopSlots];
  typename ScoreKey<T>::type bound_key[2];
  uint32_t bound_row[2];
  // the lists: the first `iterations` rows of either class in class order
  T top_nom[2][kSwapMaxIter];
  int top_cs[2][kSwapMaxIter];
  uint32_t top_row[2][kSwapMaxIter];
  typename ScoreKey<T>::type warp_key[2][kMaskWarps];
  uint32_t warp_row[2][kMaskWarps];
};

// (key, row) pairs in class order
template <typename K>
__device__ __forceinline__ bool before(K ka, uint32_t ra, K kb, uint32_t rb) {
  return ka > kb || (ka == kb && ra > rb);
}

// The last block's lists.  While the rows were scored, every group of them left its best row: the least of as many
// groups' best rows as the list is long bounds what can be in it.  What passes, some fifty rows of a class, is ranked by
// counting.  (One maximum per round cost about 600 cycles a round.)
template <typename T>
__device__ __forceinline__ void top_rows(const MaskArgs<T> &a, int groups, TopShared<T> &sh) {
  typedef typename ScoreKey<T>::type K;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // What the selection reads is asked for in as few rounds as there are dependences: each is a trip through L2.
  struct Rows {
    uint32_t f[4];
    uint8_t m[4];
    T nom[4];
    int cs[4];
  } rows;
  auto fetch = [&](const int (&e)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool in = e[u] < (int)a.N;
      rows.f[u] = in ? __ldcg(a.ms.filter + e[u]) : 0u;
      rows.m[u] = in ? __ldcg(a.ms.old_col + e[u]) : 0;
      rows.nom[u] = in ? __ldcg(a.ms.score + e[u]) : (T)0;
      rows.cs[u] = in ? __ldcg(a.ms.csum + e[u]) : 0;
    }
  };
  // all rows where that is a round trip to memory less; the rows of the blocks that have one that passes otherwise
  const bool all = a.N <= 4 * kMaskThreads;
  uint2 block_best[2];
  int e[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) e[u] = (int)threadIdx.x + u * kMaskThreads;
  if (all) {
    fetch(e);
  } else {
#pragma unroll
    for (int u = 0; u < 2; ++u) block_best[u] = e[u] < (int)gridDim.x ? __ldcg(a.ms.block_best + e[u]) : make_uint2(0, 0);
  }
  if (wid < 2) {
    // (exact keys: equal top words of float64 keys do not decide)
    const unsigned long long g = lane < groups ? __ldcg(&a.ms.header->best[wid][lane]) : ~0ull;
    const uint32_t r = (uint32_t)g;   // row + 1
    a.ms.header->best[wid][lane] = 0;
    K k = ~(K)0;
    if (r == 0) k = 0;   // a group without a row: no bound
    else if (sizeof(T) == 4) k = (K)(g >> 32);
    else if (lane < groups) k = class_key<T>(wid, swap_score(__ldcg(a.ms.score + r - 1u), __ldcg(a.ms.csum + r - 1u)));
    const K least = ~ScoreKey<T>::warp_max(~k);
    const uint32_t row = __reduce_min_sync(0xffffffffu, k == least ? r : kNoRow);
    if (lane == 0) {
      sh.count[wid] = 0;
      sh.blocks = 0;
      sh.bound_key[wid] = least;
      sh.bound_row[wid] = row;   // row + 1
    }
  }
  __syncthreads();
  const uint32_t f0 = filter_key(sh.bound_key[0]), f1 = filter_key(sh.bound_key[1]);
  auto consider = [&](int u) {
    const uint32_t f = rows.f[u];
    const int c = rows.m[u];
    if (f == 0 || f < (c == 0 ? f0 : f1)) return;
    const K k = sizeof(T) == 4 ? (K)f : class_key<T>(c, swap_score(rows.nom[u], rows.cs[u]));
    if (f == (c == 0 ? f0 : f1) && before(sh.bound_key[c], sh.bound_row[c], k, (uint32_t)(e[u] + 1))) return;
    const int at = atomicAdd(&sh.count[c], 1);
    if (at >= kTopSlots) return;
    sh.row[c][at] = (uint32_t)e[u];
    sh.key[c][at] = k;
    sh.nom[c][at] = rows.nom[u];
    sh.cs[c][at] = rows.cs[u];
  };
  if (!all) {
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kMaskThreads) {
      const uint2 best = k < kMaskThreads ? block_best[0] : k < 2 * kMaskThreads ? block_best[1] : __ldcg(a.ms.block_best + k);
      if ((best.x == 0 || best.x < f0) && (best.y == 0 || best.y < f1)) continue;
      const int at = atomicAdd(&sh.blocks, 1);
      if (at < kTopSlots) sh.block[at] = k;
    }
    __syncthreads();
  }
  const bool some = !all && sh.blocks <= kTopSlots;
  const int nrows = some ? sh.blocks * a.block_rows : (int)a.N;
#pragma unroll 1
  for (int t0 = threadIdx.x; t0 < nrows; t0 += 4 * kMaskThreads) {
    if (!all) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = t0 + u * kMaskThreads;
        e[u] = t >= nrows ? (int)a.N : some ? sh.block[t >> a.rows_log2] * a.block_rows + (t & (a.block_rows - 1)) : t;
      }
      fetch(e);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (rows.f[u] >= (f0 < f1 ? f0 : f1)) consider(u);
  }
  __syncthreads();
  const int c = threadIdx.x / kTopSlots, i = threadIdx.x % kTopSlots;
  const int n = sh.count[c];
  K k = 0;
  uint32_t row = 0;
  T nom = (T)0;
  int cs = 0;
  if (i < n && n <= kTopSlots) {
    row = sh.row[c][i];
    nom = sh.nom[c][i];
    cs = sh.cs[c][i];
    k = sh.key[c][i];
  }
  if (i < n && n <= kTopSlots) {
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < n; ++j) rank += before(sh.key[c][j], sh.row[c][j], k, row);
    if (rank < a.iterations) {
      sh.top_row[c][rank] = row;
      sh.top_nom[c][rank] = nom;
      sh.top_cs[c][rank] = cs;
    }
  } else if (i < a.iterations) {
    sh.top_row[c][i] = kNoRow;
  }
  if (sh.count[0] <= kTopSlots && sh.count[1] <= kTopSlots) return;
  // more rows pass than there are slots (many equal scores): one maximum per round
  __syncthreads();
#pragma unroll 1
  for (int round = 0; round < 2 * a.iterations; ++round) {
    const int cc = round & 1, at = round >> 1;
    if (sh.count[cc] <= kTopSlots) continue;
    K pk = ~(K)0, bk = 0;
    uint32_t pr = 0, br = 0;   // row + 1
    if (at > 0) {
      pr = sh.top_row[cc][at - 1] + 1u;   // (0: nothing was left)
      pk = pr != 0 ? class_key<T>(cc, swap_score(sh.top_nom[cc][at - 1], sh.top_cs[cc][at - 1])) : (K)0;
    }
    for (int e = threadIdx.x; e < (int)a.N; e += kMaskThreads) {
      if (__ldcg(a.ms.filter + e) == 0 || __ldcg(a.ms.old_col + e) != cc) continue;
      const K ke = class_key<T>(cc, swap_score(__ldcg(a.ms.score + e), __ldcg(a.ms.csum + e)));
      if (before(pk, pr, ke, (uint32_t)(e + 1)) && before(ke, (uint32_t)(e + 1), bk, br)) {
        bk = ke;
        br = (uint32_t)(e + 1);
      }
    }
    const K wk = ScoreKey<T>::warp_max(bk);
    const uint32_t wr = __reduce_max_sync(0xffffffffu, wk != 0 && bk == wk ? br : 0u);
    if (lane == 0) {
      sh.warp_key[0][wid] = wk;
      sh.warp_row[0][wid] = wr;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      K gk = 0;
      uint32_t gr = 0;
      for (int w = 0; w < kMaskWarps; ++w)
        if (before(sh.warp_key[0][w], sh.warp_row[0][w], gk, gr)) {
          gk = sh.warp_key[0][w];
          gr = sh.warp_row[0][w];
        }
      sh.top_row[cc][at] = gr - 1u;
      if (gr != 0) {
        sh.top_nom[cc][at] = __ldcg(a.ms.score + gr - 1u);
        sh.top_cs[cc][at] = __ldcg(a.ms.csum + gr - 1u);
      }
    }
    __syncthreads();
  }
}

// Key of a row as a member of class c; `cs` is its active count as a member of class `from`: a silent row that becomes
// active has one more connection, an active one that becomes silent one fewer.
template <typename T>
__device__ __forceinline__ typename ScoreKey<T>::type moved_key(T nom, int cs, int from, int c) {
  const T sc = swap_score(nom, cs + c - from);
  return sc == sc ? class_key<T>(c, sc) : 0;
}

// The keys of a lane's candidate rows as silent and as active rows; 0: no row, or its score is NaN.
template <typename T, int NS>
__device__ __forceinline__ void candidate_keys(const uint32_t (&row)[NS], const int (&cls)[NS], const T (&nom)[NS],
                                               const int (&cs)[NS], typename ScoreKey<T>::type (&key)[NS][2]) {
#pragma unroll
  for (int k = 0; k < NS; ++k)
#pragma unroll
    for (int c = 0; c < 2; ++c) key[k][c] = row[k] != kNoRow ? moved_key<T>(nom[k], cs[k], cls[k], c) : 0;
}

// The plainest case of the swaps, decided at once by one warp: lane t holds the t-th row of both lists, swap t exchanges
// exactly these two as long as no row moved by an earlier swap comes before either of them in its new class, and the
// swaps end at the first t whose silent row scores below its active one.  Returns the number of swaps, -1 when a moved
// row interferes.
template <typename T>
__device__ __forceinline__ int swaps_in_order(const typename ScoreKey<T>::type (&key)[2][2], int iterations) {
  typedef typename ScoreKey<T>::type K;
  const int lane = threadIdx.x & 31;
  const bool ok = key[0][0] != 0 && key[1][1] != 0 && !(class_key_value<T>(0, key[0][0]) < class_key_value<T>(1, key[1][1]));
  const unsigned no = ~__ballot_sync(0xffffffffu, ok);
  int n = no ? __ffs(no) - 1 : 32;
  n = n < iterations ? n : iterations;
  const int last = n < iterations ? n : iterations - 1;
  bool clear = true;
#pragma unroll
  for (int c = 0; c < 2; ++c)
    clear = clear && (n == 0 || ScoreKey<T>::warp_max(lane < n ? key[c][1 - c] : (K)0) < __shfl_sync(0xffffffffu, key[1 - c][1 - c], last));
  return clear ? n : -1;
}

// The swaps one by one, by one warp: NS candidate rows per lane (kNoRow: none; duplicates move together).  Returns with
// every lane's classes after the last swap.  Layers that have settled come here most of the time (the rows that swap score
// almost alike): two candidates per lane without NaN scores, a chain of two warp reductions per swap.  With six always, the
// mask update of a settled 1001 x 481 layer took 22.9 us where one with swaps in order took 10.8.
template <typename T, int NS>
__device__ __forceinline__ void replay_swaps(const uint32_t (&row)[NS], int (&cls)[NS],
                                             const typename ScoreKey<T>::type (&key)[NS][2], int iterations) {
  typedef typename ScoreKey<T>::type K;
  constexpr bool NANS = NS > 2;   // the rows that matter only for their NaN scores are among the candidates
#pragma unroll 1
  for (int it = 0; it < iterations; ++it) {
    K best[2];
    uint32_t pick[2];   // row + 1
    bool pick_nan[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      K mine = 0;
#pragma unroll
      for (int k = 0; k < NS; ++k)
        if (cls[k] == c && key[k][c] > mine) mine = key[k][c];
      best[c] = ScoreKey<T>::warp_max(mine);
      uint32_t r = 0;
#pragma unroll
      for (int k = 0; k < NS; ++k)
        if (cls[k] == c && key[k][c] != 0 && key[k][c] == best[c] && row[k] + 1u > r) r = row[k] + 1u;
      pick[c] = __reduce_max_sync(0xffffffffu, r);
      pick_nan[c] = false;
      if constexpr (NANS) {   // the class's first row in index order, and whether its score is NaN
        uint32_t f = kNoRow;
#pragma unroll
        for (int k = 0; k < NS; ++k)
          if (row[k] != kNoRow && cls[k] == c) {
            const uint32_t v = row[k] << 1 | (key[k][c] == 0);
            f = v < f ? v : f;
          }
        f = __reduce_min_sync(0xffffffffu, f);
        if (f != kNoRow && (f & 1u)) {
          pick_nan[c] = true;
          pick[c] = (f >> 1) + 1u;
        }
      }
    }
    // a class is empty, or the best silent row scores below the worst active one (never true with a NaN on either side)
    if (pick[0] == 0 || pick[1] == 0 ||
        (!pick_nan[0] && !pick_nan[1] && class_key_value<T>(0, best[0]) < class_key_value<T>(1, best[1])))
      break;   // uniform across the warp
#pragma unroll
    for (int k = 0; k < NS; ++k)
      if (row[k] != kNoRow && cls[k] <= 1 && (row[k] + 1u == pick[0] || row[k] + 1u == pick[1])) cls[k] = 1 - cls[k];
  }
}

// SCORE: the scores are computed here (otherwise they, the active counts and the old mask column are in the scratch
// already).
template <typename T, bool SCORE>
__global__ void __launch_bounds__(kMaskThreads, sizeof(T) == 4 ? 2 : 1) mask_update_kernel(const MaskArgs<T> a) {
  __shared__ TopShared<T> sh;
  __shared__ unsigned long long s_best[2][kGroups];
  __shared__ uint32_t low_row[2][64], changed[6 * 32];
  __shared__ int s_last, s_nan, n_changed, low_cnt[2], win_cnt[kMaskWarps][2];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int groups = a.iterations <= kGroups / 2 ? kGroups / 2 : kGroups;   // at least as many as the list is long
  if (threadIdx.x == 0) s_nan = 0;
  if (threadIdx.x < 2 * kGroups) s_best[threadIdx.x / kGroups][threadIdx.x % kGroups] = 0;
  __syncthreads();
  after_previous();   // (no access to global memory before it)
  // what the last block selects by: the filter key of a scored row, and the best one of its group
  auto leave_key = [&](long i, T nom, int cnt, int m) {
    const T sc = swap_score(nom, cnt);
    uint32_t f = 0;
    if (m <= 1) {
      if (sc == sc) {
        f = filter_key(class_key<T>(m, sc));
        // (scattered: neighbouring and complementary-coded inputs score alike)
        const uint32_t group = (gridDim.x >= 4 * kGroups ? blockIdx.x : (uint32_t)i) * 0x9E3779B1u >> 16 & (groups - 1);
        atomicMax(&s_best[m][group], (unsigned long long)f << 32 | (uint32_t)(i + 1));
      } else {
        s_nan = 1;
      }
    }
    a.ms.filter[i] = f;
  };
  if constexpr (SCORE) {
    // ---- scores: the mutual-information numerator over the minicolumns of hypercolumn h (terms in REAL, accumulated
    // in double) and the row's count of active connections; one row per group of W lanes, whose loads are all issued
    // before the arithmetic
    const int W = a.width, sub = lane % W;
    const long row = ((long)blockIdx.x * kMaskWarps + wid) * (32 / W) + lane / W;
    const bool live = row < a.N;
    const long i = live ? row : 0;   // (loads need no branch)
    const T *cj = a.Cj + a.h * a.Mc + sub;
    const T *cij = a.Cij + i * a.M + a.h * a.Mc + sub;
    const T *wt = a.weights ? a.weights + i * a.M + a.h * a.Mc + sub : nullptr;
    const uint8_t *mrow = a.wmask + i * a.H;
    const int left = (int)(a.Mc - sub);   // entry e of this lane exists when e * W < left
    const T pi = a.Ci[i];
    T pj[4], pij[4], wv[4];
    auto fetch = [&](int e0) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = (e0 + u) * W < left;
        pj[u] = in ? cj[(e0 + u) * W] : (T)0;   // (below the threshold: no term)
        pij[u] = in ? cij[(e0 + u) * W] : (T)0;
        wv[u] = in && wt ? wt[(e0 + u) * W] : (T)0;
      }
    };
    fetch(0);
    int cnt = 0;
    for (int k = sub; k < (int)a.H; k += W) cnt += mrow[k];
    const uint8_t bit = mrow[a.h];
    double s = 0.0;
    if (pi >= a.cthr) {
#pragma unroll 1
      for (int e = 0; e * W < left; ++e) {   // (one copy of the logarithms; the entries rotate through slot 0)
        if (pj[0] >= a.cthr) {
          const T w = wt ? wv[0] : log_ratio(pij[0], pi, pj[0], a.cthr4);
          const T x = ((T)1 - pi) * pj[0];
          const T y = (pj[0] - pij[0]) / x;
          s += (double)(pij[0] * w + (pj[0] - pij[0]) * sbb_log(y));
        }
        if ((e & 3) == 3) {
          fetch(e + 1);
        } else {
#pragma unroll
          for (int v = 0; v < 3; ++v) {
            pj[v] = pj[v + 1];
            pij[v] = pij[v + 1];
            wv[v] = wv[v + 1];
          }
        }
      }
    }
    for (int off = W >> 1; off > 0; off >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, off, W);
      cnt += __shfl_xor_sync(0xffffffffu, cnt, off, W);
    }
    if (live && sub == 0) {
      a.ms.score[i] = (T)s;
      a.ms.csum[i] = cnt;
      a.ms.old_col[i] = bit;   // the mask column before the swaps
      leave_key(i, (T)s, cnt, bit);
    }
  } else {
    const long i = (long)blockIdx.x * a.block_rows + threadIdx.x;
    if ((int)threadIdx.x < a.block_rows && i < a.N) leave_key(i, a.ms.score[i], a.ms.csum[i], a.ms.old_col[i]);
  }
  // ---- the block that finishes last goes on (the fence of the thread that counts the block covers what the barrier has put
  // before it)
  __syncthreads();
  if (threadIdx.x < 2 * kGroups) {
    const unsigned long long best = s_best[threadIdx.x / kGroups][threadIdx.x % kGroups];
    if (best != 0) atomicMax(&a.ms.header->best[threadIdx.x / kGroups][threadIdx.x % kGroups], best);
    const uint32_t f = __reduce_max_sync(0xffffffffu, (uint32_t)(best >> 32));
    if (lane == 0) reinterpret_cast<uint32_t *>(a.ms.block_best + blockIdx.x)[wid] = f;
    if (threadIdx.x == 0 && s_nan) atomicOr(&a.ms.header->nan, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(&a.ms.header->ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    s_nan = a.ms.header->nan;
    low_cnt[0] = low_cnt[1] = 0;
    a.ms.header->ticket = 0;
    a.ms.header->nan = 0;
  }
  if (threadIdx.x < 128) low_row[threadIdx.x & 1][threadIdx.x >> 1] = kNoRow;
  top_rows<T>(a, groups, sh);
  __syncthreads();
  const bool nan_rows = s_nan != 0;
  if (nan_rows) {
    // some row scores NaN: it can be picked while it is its class's first, so the lowest iterations + 1 rows of either
    // class (one row leaves a class per swap) are candidates too
    const int want = a.iterations + 1;
    for (long w0 = 0; w0 < a.N; w0 += kMaskThreads) {
      const long j = w0 + threadIdx.x;
      const uint8_t m = j < a.N ? __ldcg(a.ms.old_col + j) : (uint8_t)2;
      unsigned bal[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        bal[c] = __ballot_sync(0xffffffffu, m == c);
        if (lane == 0) win_cnt[wid][c] = __popc(bal[c]);
      }
      __syncthreads();
      if (m <= 1) {
        int pos = low_cnt[m] + __popc(bal[m] & ((1u << lane) - 1u));
        for (int w = 0; w < wid; ++w) pos += win_cnt[w][m];
        if (pos < want) low_row[m][pos] = (uint32_t)j;
      }
      __syncthreads();
      if (threadIdx.x < 2)
        for (int w = 0; w < kMaskWarps; ++w) low_cnt[threadIdx.x] += win_cnt[w][threadIdx.x];
      __syncthreads();
      if (low_cnt[0] >= want && low_cnt[1] >= want) break;   // uniform: read after the barrier
    }
  }
  if (wid != 0 && a.rewrite_w != nullptr) {
    // most rows that will move are on the lists: their traces come to this SM while the swaps are decided
    const int lines = (int)((a.Mc * sizeof(T) + 127) / 128) + 1;   // of a row's traces in hypercolumn h, and its Ci
    for (int t = threadIdx.x - 32; t < 2 * a.iterations * (lines + 1); t += kMaskThreads - 32) {
      const int slot = t / (lines + 1), k = t % (lines + 1);
      const uint32_t r = sh.top_row[slot & 1][slot >> 1];
      if (r == kNoRow) continue;
      const long col = k * (long)(128 / sizeof(T));
      const T *p = k == lines ? a.Ci + r : a.Cij + (long)r * a.M + a.h * a.Mc + (col < a.Mc ? col : a.Mc - 1);
      asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
    }
  }
  if (wid == 0) {
    // the rows of both lists, one per lane and class
    uint32_t row[2];
    int cs[2];
    T nom[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      row[c] = lane < a.iterations ? sh.top_row[c][lane] : kNoRow;
      nom[c] = row[c] != kNoRow ? sh.top_nom[c][lane] : (T)0;
      cs[c] = row[c] != kNoRow ? sh.top_cs[c][lane] : 0;
    }
    int n = 0;
    auto move = [&](bool moved, uint32_t r, int count, int from) {   // (the whole warp calls it)
      if (moved) {
        a.wmask[(long)r * a.H + a.h] = (uint8_t)(1 - from);
        a.ms.csum[r] = count + 1 - 2 * from;
      }
      const unsigned who = __ballot_sync(0xffffffffu, moved);
      if (moved) changed[n + __popc(who & ((1u << lane) - 1u))] = r << 1 | (uint32_t)(1 - from);
      n += __popc(who);
    };
    int cls[2] = {0, 1};
    typename ScoreKey<T>::type key[2][2];
    candidate_keys<T, 2>(row, cls, nom, cs, key);
    int swaps = swaps_in_order<T>(key, a.iterations);
    if (nan_rows && swaps >= 0) {
      // ... and no class is headed by a NaN score now or later: its first row has a number for a score and stays
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint32_t first = low_row[c][0];
        const T nm = first != kNoRow ? __ldcg(a.ms.score + first) : (T)0;
        if (nm != nm || __any_sync(0xffffffffu, lane < swaps && row[c] == first)) swaps = -1;
      }
    }
    if (swaps >= 0) {
      move(lane < swaps, row[0], cs[0], 0);
      move(lane < swaps, row[1], cs[1], 1);
    } else if (!nan_rows) {
      replay_swaps<T, 2>(row, cls, key, a.iterations);
#pragma unroll
      for (int c = 0; c < 2; ++c) move(row[c] != kNoRow && cls[c] != c, row[c], cs[c], c);
    } else {
      constexpr int NS = 6;   // both lists, and the lowest rows of both classes
      uint32_t rows[NS];
      int in[NS], css[NS];
      T noms[NS];
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        rows[k] = k < 2 ? row[k & 1] : low_row[k & 1][lane + 32 * ((k - 2) >> 1)];
        noms[k] = rows[k] != kNoRow ? __ldcg(a.ms.score + rows[k]) : (T)0;
        css[k] = rows[k] != kNoRow ? __ldcg(a.ms.csum + rows[k]) : 0;
        in[k] = k & 1;
      }
      typename ScoreKey<T>::type keys[NS][2];
      candidate_keys<T, NS>(rows, in, noms, css, keys);
      replay_swaps<T, NS>(rows, in, keys, a.iterations);
#pragma unroll
      for (int k = 0; k < NS; ++k) move(rows[k] != kNoRow && in[k] != (k & 1), rows[k], css[k], k & 1);
    }
    if (lane == 0) n_changed = a.rewrite_w != nullptr ? n : 0;
  }
  __syncthreads();
  // the weights of hypercolumn h of the rows whose mask bit changed follow the new bit: a warp per row, the rows that became
  // active (they come first) spread over the warps, four entries per lane in flight
#pragma unroll 1
  for (int q = wid; q < n_changed; q += kMaskWarps) {
    const long row = changed[q] >> 1;
    const T ci = a.Ci[row];
    const T *cj = a.Cj + a.h * a.Mc + lane, *cij = a.Cij + row * a.M + a.h * a.Mc + lane;
    T *w = a.rewrite_w + row * a.M + a.h * a.Mc + lane;
    const int left = (int)a.Mc - lane;   // entry e of this lane exists when 32 * e < left
    if (!(changed[q] & 1u) || ci < a.cthr) {
      for (int e = 0; e < left; e += 32) w[e] = (T)0;
      continue;
    }
#pragma unroll 1
    for (int e0 = 0; e0 < left; e0 += 128) {
      T pj[4], pij[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = e0 + 32 * u < left;
        pj[u] = in ? cj[e0 + 32 * u] : (T)0;
        pij[u] = in ? cij[e0 + 32 * u] : (T)0;
      }
#pragma unroll 1
      for (int e = e0; e < left && e < e0 + 128; e += 32) {
        w[e] = !(pj[0] < a.cthr) ? log_ratio(pij[0], ci, pj[0], a.cthr4) : (T)0;
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          pj[v] = pj[v + 1];
          pij[v] = pij[v + 1];
        }
      }
    }
  }
}

// Mask scores of the rows [row_begin, row_end) this rank owns, written into every rank's work arrays
// (scratch_tab: base of each rank's mask scratch, laid out for N rows).
template <typename T>
__global__ void __launch_bounds__(256)
    mask_score_rows_kernel(const uint8_t *__restrict__ wmask, const T *__restrict__ weights, const T *__restrict__ Ci,
                           const T *__restrict__ Cj, const T *__restrict__ Cij, T cthr, T cthr4, long N, long M, long H, long Mc, long h,
                           long row_begin, long row_end, PeerTable scratch_tab) {
  const int lane = threadIdx.x & 31;
  const long i = row_begin + (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= row_end) return;
  const T pi = Ci[i];
  double s = 0.0;
  if (pi >= cthr) {
    for (long jj = lane; jj < Mc; jj += 32) {
      const long col = h * Mc + jj;
      const T pj = Cj[col];
      if (pj >= cthr) {
        const T pij = Cij[i * M + col];
        const T w = weights ? weights[i * M + col] : log_ratio(pij, pi, pj, cthr4);
        const T x = ((T)1 - pi) * pj;
        const T y = (pj - pij) / x;
        s += (double)(pij * w + (pj - pij) * sbb_log(y));
      }
    }
  }
  int cnt = 0;
  for (long k = lane; k < H; k += 32) cnt += wmask[i * H + k];
  for (int off = 16; off > 0; off >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, off);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, off);
  }
  if (lane == 0) {
    const uint8_t bit = wmask[i * H + h];
    for (int d = 0; d < scratch_tab.n; ++d) {
      MaskScratch<T> ms(scratch_tab.ptr[d], N);
      ms.score[i] = (T)s;
      ms.csum[i] = cnt;
      ms.old_col[i] = bit;
    }
  }
}
template <typename T>
cudaError_t launch_mask_score_rows(const uint8_t *wmask, const T *weights, const T *Ci, const T *Cj, const T *Cij, T cthr, long N, long M,
                                   long H, long Mc, long h, long row_begin, long row_end, const PeerTable &scratch_tab,
                                   cudaStream_t st) {
  if (row_end <= row_begin) return cudaSuccess;
  const T cthr4 = cthr * cthr * cthr * cthr;
  mask_score_rows_kernel<T><<<(unsigned)((row_end - row_begin + 7) / 8), 256, 0, st>>>(
      wmask, weights, Ci, Cj, Cij, cthr, cthr4, N, M, H, Mc, h, row_begin, row_end, scratch_tab);
  return launched();
}
template cudaError_t launch_mask_score_rows<float>(const uint8_t *, const float *, const float *, const float *, const float *, float,
                                                   long, long, long, long, long, long, long, const PeerTable &,
                                                   cudaStream_t);
template cudaError_t launch_mask_score_rows<double>(const uint8_t *, const double *, const double *, const double *, const double *,
                                                    double, long, long, long, long, long, long, long, const PeerTable &,
                                                    cudaStream_t);

// After the swaps: owned rows whose mask bit changed get hypercolumn h's weights recomputed from the owner's
// traces, in every rank's weight matrix.  One warp per owned row.
template <typename T>
__global__ void __launch_bounds__(256)
    mask_rewrite_rows_kernel(const uint8_t *__restrict__ wmask, const uint8_t *__restrict__ old_col,
                             const T *__restrict__ Ci, const T *__restrict__ Cj, const T *__restrict__ Cij, T cthr,
                             T cthr4, long M, long H, long Mc, long h, long row_begin, long row_end, PeerTable wtab) {
  const int lane = threadIdx.x & 31;
  const long i = row_begin + (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= row_end) return;
  const uint8_t now = wmask[i * H + h];
  if (now == old_col[i]) return;
  const T ci = Ci[i];
  for (long jj = lane; jj < Mc; jj += 32) {
    const long col = h * Mc + jj;
    const T cj = Cj[col];
    T v = (T)0;
    if (now != 0 && !(ci < cthr) && !(cj < cthr)) v = log_ratio(Cij[i * M + col], ci, cj, cthr4);
    for (int d = 0; d < wtab.n; ++d) static_cast<T *>(wtab.ptr[d])[i * M + col] = v;
  }
}
template <typename T>
cudaError_t launch_mask_rewrite_rows(const uint8_t *wmask, const void *scratch, const T *Ci, const T *Cj, const T *Cij,
                                     T cthr, long N, long M, long H, long Mc, long h, long row_begin, long row_end,
                                     const PeerTable &wtab, cudaStream_t st) {
  if (row_end <= row_begin) return cudaSuccess;
  MaskScratch<T> ms(const_cast<void *>(scratch), N);
  const T cthr4 = cthr * cthr * cthr * cthr;
  mask_rewrite_rows_kernel<T><<<(unsigned)((row_end - row_begin + 7) / 8), 256, 0, st>>>(
      wmask, ms.old_col, Ci, Cj, Cij, cthr, cthr4, M, H, Mc, h, row_begin, row_end, wtab);
  return launched();
}
template cudaError_t launch_mask_rewrite_rows<float>(const uint8_t *, const void *, const float *, const float *,
                                                     const float *, float, long, long, long, long, long, long, long,
                                                     const PeerTable &, cudaStream_t);
template cudaError_t launch_mask_rewrite_rows<double>(const uint8_t *, const void *, const double *, const double *,
                                                      const double *, double, long, long, long, long, long, long, long,
                                                      const PeerTable &, cudaStream_t);

// The full scan stays for lists longer than kSwapMaxIter.
template <typename T, bool SCORE>
static cudaError_t launch_mask(uint8_t *wmask, const T *weights, const T *Ci, const T *Cj, const T *Cij, T cthr, long N,
                               long M, long H, long Mc, long h, long iterations, void *scratch, cudaStream_t st, T *rewrite_w) {
  if (N == 0) return cudaSuccess;
  MaskArgs<T> a{wmask, weights, Ci, Cj, Cij, rewrite_w, cthr, cthr * cthr * cthr * cthr, N, M, H, Mc, h, (int)iterations, 32,
                0, 0, MaskScratch<T>(scratch, N)};
  if (iterations >= 1 && iterations <= kSwapMaxIter && N < (1l << 30) && Mc < (1l << 22)) {
    // lanes per row: as many as shorten the chain of logarithms, but eight where there are rows enough to fill the chip:
    // then instructions bound it, and what a row costs besides its logarithms is paid once for four rows
    if (N >= 16384) a.width = 8;
    while (a.width > 1 && (a.width >> 1) >= Mc) a.width >>= 1;
    a.block_rows = SCORE ? kMaskThreads / a.width : kMaskThreads / 8;
    while ((1 << a.rows_log2) < a.block_rows) a.rows_log2 += 1;
    const long rows = a.block_rows;
    launch_next(mask_update_kernel<T, SCORE>, (unsigned)((N + rows - 1) / rows), kMaskThreads, 0, st, a);
    return launched();
  }
  if constexpr (SCORE) {
    PeerTable own{};
    own.n = 1;
    own.ptr[0] = scratch;
    cudaError_t e = launch_mask_score_rows<T>(wmask, weights, Ci, Cj, Cij, cthr, N, M, H, Mc, h, 0, N, own, st);
    if (e != cudaSuccess) return e;
  }
  mask_swap_kernel<T><<<1, 1024, 0, st>>>(wmask, a.ms.score, a.ms.csum, N, M, H, Mc, h, iterations, rewrite_w,
                                          a.ms.old_col, Ci, Cj, Cij, cthr, a.cthr4);
  return launched();
}

template <typename T>
cudaError_t launch_mask_update(uint8_t *wmask, const T *weights, const T *Ci, const T *Cj, const T *Cij, T cthr,
                               long N, long M, long H, long Mc, long h, long iterations, void *scratch,
                               cudaStream_t st, T *rewrite_w) {
  return launch_mask<T, true>(wmask, weights, Ci, Cj, Cij, cthr, N, M, H, Mc, h, iterations, scratch, st, rewrite_w);
}
// The swaps alone, from per-row scores, active counts and the old mask column already in `scratch`.
template <typename T>
cudaError_t launch_mask_select(uint8_t *wmask, const T *Ci, const T *Cj, const T *Cij, T cthr, long N, long M, long H,
                               long Mc, long h, long iterations, void *scratch, cudaStream_t st, T *rewrite_w) {
  return launch_mask<T, false>(wmask, nullptr, Ci, Cj, Cij, cthr, N, M, H, Mc, h, iterations, scratch, st, rewrite_w);
}
template cudaError_t launch_mask_select<float>(uint8_t *, const float *, const float *, const float *, float, long, long,
                                               long, long, long, long, void *, cudaStream_t, float *);
template cudaError_t launch_mask_select<double>(uint8_t *, const double *, const double *, const double *, double, long,
                                                long, long, long, long, long, void *, cudaStream_t, double *);
template cudaError_t launch_mask_update<float>(uint8_t *, const float *, const float *, const float *, const float *,
                                               float, long, long, long, long, long, long, void *, cudaStream_t,
                                               float *);
template cudaError_t launch_mask_update<double>(uint8_t *, const double *, const double *, const double *,
                                                const double *, double, long, long, long, long, long, long, void *,
                                                cudaStream_t, double *);

}  // namespace sbb
