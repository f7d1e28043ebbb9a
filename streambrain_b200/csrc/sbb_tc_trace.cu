// The fused trace step on the 5th-generation tensor cores.
//
//   D[i, j] = sum_b x[b, i] * y[b, j],   Cij = max(0, (1 - tau) Cij + tau / B * D),   W = log(Cij / (Ci Cj)) under the mask
//
// float32 operands as split TF32 products (hi*hi + hi*lo + lo*hi, see sbb_tc_kernels.cu): A's parts go to tensor memory,
// B's low part beside the raw tile in shared memory.  A cluster of two CTAs works on 256 rows x 192 columns
// (tcgen05.mma.cta_group::2); each CTA stages and splits its own 128 rows of A and half of the columns of B.  (!PAIR, what
// SBB_TC_PAIR=0 selects: one CTA works on 128 rows x 192 columns by itself and stages all columns of B, which leaves room
// for three stages; the products, chains and sums are the same.  It is there to compare with and for
// devices that cannot place pairs.  Train step without a mask update: 1568 -> 30 x 100 at batch 128 20.0 us in pairs, 20.5
// without; 55296 -> 30 x 100 at 256 539 and 656 us; 1568 -> 100 x 300 at 1024 487 and 632.)
// Roles in a CTA (672 threads, one CTA per SM, tiles walked persistently):
//   warps 0-11   epilogue: accumulator, old trace (by TMA, the whole tile's blocks one tile ahead), arithmetic; new traces
//                and weights leave by TMA
//   warps 12-15  A converters (one tile row, that is one tensor-memory lane, per thread)
//   warp 16      TMA producer (one lane)
//   warp 17      MMA issuer (one lane of the pair's leader) and owner of the tensor-memory allocation
//   warp 18      row and column data of the next tile (reciprocals, mask bits) into shared memory: loaded by the epilogue
//                warps themselves these were a round trip to memory per tile that all of them sat out together
//   warps 19-20  B converters
// Accumulation chains: the tensor core truncates every accumulate, so no chain is longer than 256 samples (96 MMAs).  The
// epilogue adds the later chains of a long batch to the running sum in float32, which stays where the old trace landed in
// shared memory; it went through the trace matrix in L2 before (8 bytes per element and chain).
// Every wait is bounded (sbb_tc_ptx.cuh).
#include "sbb_tc.cuh"
#include "sbb_tc_ptx.cuh"

#include <atomic>

#include "sbb_launch.cuh"
#include "sbb_math.cuh"

namespace sbb {

void count_launches(int n);   // sbb_kernels.cu

namespace {

constexpr int kEpi = 12, kConv = 12, kTma = 16, kMma = 17, kVec = 18, kConvB = 19, kBWarps = 2;
constexpr int kThreads = (kConvB + kBWarps) * 32;
constexpr int kBN = 192, kBK = 16;
constexpr int kChainKb = 16;                     // k-blocks per accumulation chain
constexpr int kGroups = kBN / (kEpi / 4) / 32;   // 32-column groups per epilogue warp
constexpr int kABytes = 128 * kBK * 4;
constexpr int kTmemA = 2 * kBN;                  // two accumulators, then per stage kBK columns of A hi and as many of A lo
constexpr int kSlab = 32 * 32 * 4;               // a 32 x 32 block of the trace matrix
constexpr int kHalf = kSlab / 2;                 // 32 rows x 16 columns of weights
struct TileVectors {
  float rci[128], rcj[kBN];     // reciprocals of Ci and Cj, 0 below the threshold
  uint32_t bits[128];           // per row: bit k = mask of hypercolumn (the tile's first) + k
};
template <bool PAIR>
struct Layout {
  static constexpr int BNH = PAIR ? kBN / 2 : kBN;   // columns of B a CTA stages
  static constexpr int STAGES = PAIR ? 5 : 3;        // stages in shared memory
  static constexpr int SLOTS = PAIR ? 4 : 3;         // k-blocks whose A parts tensor memory holds
  static constexpr int B_BYTES = BNH * kBK * 4;
  static constexpr int TX = kABytes + B_BYTES, STAGE = TX + B_BYTES;   // [A | B | B lo]
  static_assert(SLOTS <= STAGES && kTmemA + SLOTS * 2 * kBK <= 512, "tensor memory budget");
  static_assert(STAGE % 1024 == 0 && kABytes % 1024 == 0 && TX % 1024 == 0, "swizzle alignment");
  static constexpr int SLAB_OFFSET = STAGES * STAGE;
  static constexpr int W_OFFSET = SLAB_OFFSET + kEpi * kGroups * kSlab;   // weights on their way out
  static constexpr int VEC_OFFSET = W_OFFSET + kEpi * kHalf;
  static constexpr int BAR_OFFSET = VEC_OFFSET + 2 * (int)sizeof(TileVectors);
  // full, converted, empty per stage; acc_full[2], acc_empty[2], drain, vec_full[2], vec_empty[2]; one per block of the tile
  static constexpr int BARS = 3 * STAGES + 9 + kEpi * kGroups;
  static constexpr int SMEM = BAR_OFFSET + BARS * 8 + 24 + 1024;
  static_assert(BAR_OFFSET % 8 == 0 && SMEM <= 232448, "shared memory budget");
};

struct Trace {
  int m_units, n_tiles, kblocks, m_fastest;   // m_units: row tiles, or pairs of them
  int a_box3, b_box3_tiles;   // A, and column tiles below the limit of B, come in one 3-D box per stage
  int lose_arrive;            // test hook: converter thread 0 of CTA 0 skips its arrival for the first stage
  long long wait_limit;
  int rows, cols;             // N, M
  const float *rci, *rcj;
  const uint8_t *wmask;
  uint32_t hc_magic;          // ceil(2^32 / Mc) where that divides every column exactly, else 0
  int H, Mc;
  int normal;                 // cthr^4 is a normal float: every logarithm's argument is
  float one_minus, cthr4, ema_scale;
};

template <bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
    trace_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmA3, const __grid_constant__ CUtensorMap tmB3,
                 const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmW, const Trace g, int *status) {
  using L = Layout<PAIR>;
  constexpr int kStages = L::STAGES, kStage = L::STAGE, kBNH = L::BNH, kBBytes = L::B_BYTES, kTx = L::TX;
  constexpr int kSlots = L::SLOTS, kSlabOffset = L::SLAB_OFFSET, kVecOffset = L::VEC_OFFSET;
  extern __shared__ uint8_t smem_dyn[];
  const uint32_t dyn_base = smem_u32(smem_dyn);
  const uint32_t base = (dyn_base + 1023u) & ~1023u;   // swizzle atoms need 1024-byte alignment
  uint8_t *smem = smem_dyn + (base - dyn_base);
  const uint32_t bars = base + L::BAR_OFFSET;
  auto bar_full = [&](int s) { return bars + 8u * s; };
  auto bar_conv = [&](int s) { return bars + 8u * (kStages + s); };
  auto bar_empty = [&](int s) { return bars + 8u * (2 * kStages + s); };
  auto bar_acc_full = [&](int b) { return bars + 8u * (3 * kStages + b); };
  auto bar_acc_empty = [&](int b) { return bars + 8u * (3 * kStages + 2 + b); };
  const uint32_t bar_drain = bars + 8u * (3 * kStages + 4);
  auto bar_vec_full = [&](int b) { return bars + 8u * (3 * kStages + 5 + b); };
  auto bar_vec_empty = [&](int b) { return bars + 8u * (3 * kStages + 7 + b); };
  auto leader_arrive = [&](uint32_t bar) {   // (PAIR: the leader's barrier counts both CTAs' threads)
    if constexpr (PAIR) mbar_arrive_rank(bar, 0);
    else mbar_arrive(bar);
  };
  auto commit = [&](uint32_t bar) {   // (PAIR: to both CTAs' barriers)
    if constexpr (PAIR) mma_commit_pair(bar);
    else mma_commit(bar);
  };
  auto bar_slab = [&](int e, int gr) { return bars + 8u * (3 * kStages + 9 + kGroups * e + gr); };
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + L::BAR_OFFSET + L::BARS * 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform)
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_conv(s), (PAIR ? 2 : 1) * (4 + kBWarps) * 32);   // the leader's counts both CTAs' converters
      mbar_init(bar_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full(b), 1);
      mbar_init(bar_acc_empty(b), (PAIR ? 2 : 1) * kEpi);
      mbar_init(bar_vec_full(b), 32);
      mbar_init(bar_vec_empty(b), kEpi);
    }
    mbar_init(bar_drain, 1);
    for (int e = 0; e < kEpi * kGroups; ++e) mbar_init(bar_slab(e / kGroups, e % kGroups), 1);
    *abort_flag = 0;
    *reinterpret_cast<volatile long long *>(abort_flag + 1) = g.wait_limit;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMma) {
    if constexpr (PAIR) {
      tmem_alloc_pair(smem_u32(tmem_slot), 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_slot), 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // the peer's barriers exist before anything arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Only the warp that reads what the kernel before this one in the stream computed (column_vectors_kernel: the reciprocals)
  // waits for its end, and the epilogue, which writes, waits for that warp.  x, y and the old traces come by TMA and were
  // complete before that kernel let any of these blocks start: every kernel does so only after its own predecessors.
  // Train step without a mask update, 1568 -> 30 x 100 at batch 128: 23.3 -> 20.0 us.

  // The clusters walk the tiles side by side, columns fastest (rows fastest where the columns are the longer side): at any
  // time they share the operands of a few row tiles.
  const uint32_t total = (uint32_t)g.m_units * (uint32_t)g.n_tiles;
  const uint32_t w_first = PAIR ? blockIdx.x >> 1 : blockIdx.x, w_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  auto decode = [&](uint32_t w, int &mt, int &nt) {
    const uint32_t fast = g.m_fastest ? g.m_units : g.n_tiles, slow_at = w / fast, fast_at = w - slow_at * fast;
    mt = (int)(g.m_fastest ? fast_at : slow_at);
    nt = (int)(g.m_fastest ? slow_at : fast_at);
    if (PAIR) mt = 2 * mt + (int)rank;   // may be one past the last row tile: such a CTA stages zeros and stores nothing
  };
  auto hc_of = [&](int n) -> int { return (int)(g.hc_magic ? __umulhi((uint32_t)n, g.hc_magic) : (uint32_t)n / (uint32_t)g.Mc); };
  auto first_hc = [&](int nt) -> int { return g.wmask ? hc_of(nt * kBN) : 0; };
  auto last_hc = [&](int nt) -> int { return g.wmask ? hc_of(min(nt * kBN + kBN, g.cols) - 1) : 0; };

  if (warp == kTma) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t w = w_first; w < total && ok; w += w_step) {
        int mt, nt;
        decode(w, mt, nt);
        for (int kb = 0; kb < g.kblocks; ++kb, ++it) {
          const int s = it % kStages, k0 = kb * kBK;
          if (!mbar_wait(bar_empty(s), ((it / kStages) & 1u) ^ 1u, abort_flag, status, kWaitEmpty)) { ok = false; break; }
          mbar_arrive_expect_tx(bar_full(s), kTx);
          const uint32_t a_dst = base + s * kStage, b_dst = a_dst + kABytes;
          if (g.a_box3) {
            tma_load_3d(a_dst, &tmA3, 0, k0, mt * 4, bar_full(s));
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) tma_load_2d(a_dst + c * (kBK * 128), &tmA, mt * 128 + 32 * c, k0, bar_full(s));
          }
          if (nt < g.b_box3_tiles) {
            tma_load_3d(b_dst, &tmB3, 0, k0, nt * (kBN / 32) + (int)rank * (kBNH / 32), bar_full(s));
          } else {
#pragma unroll
            for (int c = 0; c < kBNH / 32; ++c)
              tma_load_2d(b_dst + c * (kBK * 128), &tmB, nt * kBN + (int)rank * kBNH + 32 * c, k0, bar_full(s));
          }
        }
      }
      if (!ok) {   // loads already issued still land here: give them a bounded moment before the CTA retires
        const long long t0 = clock64();
        while (clock64() - t0 < 400000ll) {
        }
      }
    }
  } else if (warp == kMma) {
    // ------------------------------------------------------------ MMA issuer
    if (rank == 0 && elect_one()) {
      // D float32, A (tensor memory) and B (shared memory, MN-major) TF32; 256 rows over the pair (or 128), kBN columns
      constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 16) | ((uint32_t)(kBN >> 3) << 17) |
                                 ((uint32_t)((PAIR ? 256 : 128) >> 4) << 24);
      auto mma = [&](uint32_t d, uint32_t ta, uint64_t db, uint32_t accumulate) {
        if constexpr (PAIR) mma_tf32_ts_pair(d, ta, db, idesc, accumulate);
        else mma_tf32_ts(d, ta, db, idesc, accumulate);
      };
      uint32_t it = 0, chain = 0;
      bool ok = true;
      for (uint32_t w = w_first; w < total && ok; w += w_step) {
        for (int kb = 0; kb < g.kblocks && ok;) {
          const uint32_t buf = chain & 1u;
          if (!mbar_wait(bar_acc_empty(buf), ((chain >> 1) & 1u) ^ 1u, abort_flag, status, kWaitAccEmpty)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + buf * kBN;
          const int kb_end = kb + kChainKb < g.kblocks ? kb + kChainKb : g.kblocks;
          for (bool first = true; kb < kb_end; ++kb, ++it) {
            const int s = it % kStages;
            if (!mbar_wait(bar_conv(s), (it / kStages) & 1u, abort_flag, status, kWaitConv)) { ok = false; break; }
            tc_fence_after();
            const uint32_t b_hi = base + s * kStage + kABytes, b_lo = base + s * kStage + kTx;
            const uint32_t ta = tmem_base + kTmemA + (it % kSlots) * (2 * kBK);
#pragma unroll
            for (int kk = 0; kk < kBK / 8; ++kk) {   // eight 128-byte rows (two 4-row swizzle atoms) of B per instruction
              const uint64_t db_hi = smem_desc_mn(b_hi + kk * 1024, kBK * 128), db_lo = smem_desc_mn(b_lo + kk * 1024, kBK * 128);
              mma(d_tmem, ta + kBK + kk * 8, db_hi, first && kk == 0 ? 0u : 1u);
              mma(d_tmem, ta + kk * 8, db_lo, 1u);
              mma(d_tmem, ta + kk * 8, db_hi, 1u);
            }
            first = false;
            commit(bar_empty(s));   // the stage may be refilled, in both CTAs, once these MMAs have read it
          }
          if (ok) {
            commit(bar_acc_full(buf));
            ++chain;
          }
        }
      }
      // nothing may still be running in the tensor pipe when its memory is freed (bounded by time alone)
      commit(bar_drain);
      if (!mbar_try_wait(bar_drain, 0)) mbar_wait_slow(bar_drain, 0, abort_flag, status, kWaitDrain, false);
    }
  } else if (warp >= kConv && warp < kConv + 4) {
    // ------------------------------------------------------------ A hi / lo parts into tensor memory
    uint32_t it = 0;
    bool ok = true;
    const int cw = warp - kConv;   // tensor-memory lane quarter (kConv is a multiple of four)
    for (uint32_t w = w_first; w < total && ok; w += w_step)
      for (int kb = 0; kb < g.kblocks; ++kb, ++it) {
        const int s = it % kStages;
        if (!mbar_wait_warp(bar_full(s), (it / kStages) & 1u, abort_flag, status, kWaitFull)) { ok = false; break; }
        // MN-major tile [32-row chunk][k][32 rows]: element (k, m) of chunk m / 32 sits in the 128-byte line k at 32-byte
        // piece ((m % 32) / 8) ^ (k % 4); a warp reads one line per k
        const uint8_t *acol = smem + s * kStage + cw * (kBK * 128) + ((lane & 7) << 2);
        uint32_t r[kBK];
#pragma unroll
        for (int k = 0; k < kBK; ++k)
          r[k] = *reinterpret_cast<const uint32_t *>(acol + k * 128 + (((lane >> 3) ^ (k & 3)) << 5));
        if constexpr (kSlots < kStages) {   // the k-block whose place in tensor memory this one takes has been multiplied
          if (it >= kSlots) {
            const uint32_t old = it - kSlots;
            if (!mbar_wait_warp(bar_empty(old % kStages), (old / kStages) & 1u, abort_flag, status, kWaitEmpty)) { ok = false; break; }
            tc_fence_after();
          }
        }
        const uint32_t ta = tmem_base + kTmemA + (it % kSlots) * (2 * kBK) + ((uint32_t)(cw * 32) << 16);
        tmem_st_32x32b<kBK>(ta, r);
#pragma unroll
        for (int k = 0; k < kBK; ++k) r[k] = __float_as_uint(tf32_lo(__uint_as_float(r[k])));
        tmem_st_32x32b<kBK>(ta + kBK, r);
        tmem_wait_st();
        tc_fence_before();
        if (!(g.lose_arrive && it == 0 && threadIdx.x == kConv * 32 && blockIdx.x == 0)) leader_arrive(bar_conv(s));
      }
  } else if (warp >= kConvB) {
    // ------------------------------------------------------------ B's low part beside the raw tile
    uint32_t it = 0;
    bool ok = true;
    const int t = threadIdx.x - kConvB * 32;
    for (uint32_t w = w_first; w < total && ok; w += w_step)
      for (int kb = 0; kb < g.kblocks; ++kb, ++it) {
        const int s = it % kStages;
        if (!mbar_wait_warp(bar_full(s), (it / kStages) & 1u, abort_flag, status, kWaitFull)) { ok = false; break; }
        const float4 *raw = reinterpret_cast<const float4 *>(smem + s * kStage + kABytes);
        float4 *low = reinterpret_cast<float4 *>(smem + s * kStage + kTx);
        constexpr int kPieces = kBBytes / 16 / (kBWarps * 32);
        static_assert(kBBytes % (16 * kBWarps * 32) == 0, "a whole number of 16-byte pieces per thread");
        constexpr int kAhead = 6;   // loads issued before the first store: all of a pair's share
        static_assert(kPieces % kAhead == 0, "whole groups of pieces");
#pragma unroll
        for (int i0 = 0; i0 < kPieces; i0 += kAhead) {
          float4 v[kAhead];
#pragma unroll
          for (int i = 0; i < kAhead; ++i) v[i] = raw[t + (i0 + i) * (kBWarps * 32)];
#pragma unroll
          for (int i = 0; i < kAhead; ++i)
            low[t + (i0 + i) * (kBWarps * 32)] = make_float4(tf32_lo(v[i].x), tf32_lo(v[i].y), tf32_lo(v[i].z), tf32_lo(v[i].w));
        }
        fence_async_smem();   // make the generic-proxy writes visible to the tensor pipe
        leader_arrive(bar_conv(s));
      }
  } else if (warp == kVec) {
    // ------------------------------------------------------------ row and column data, one tile ahead
    uint32_t t = 0;
    after_previous();
    for (uint32_t w = w_first; w < total; w += w_step, ++t) {
      int mt, nt;
      decode(w, mt, nt);
      const uint32_t b = t & 1u;
      TileVectors *v = reinterpret_cast<TileVectors *>(smem + kVecOffset) + b;
      const long n0 = (long)nt * kBN, i0 = (long)mt * 128;
      const int hc0 = first_hc(nt), nhc = g.wmask ? last_hc(nt) - hc0 + 1 : 0;
      float rci[4], rcj[kBN / 32];
      uint32_t bits[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const long i = i0 + lane + 32 * k;
        rci[k] = i < g.rows ? __ldg(g.rci + i) : 0.f;
        bits[k] = g.wmask ? 0u : 0xFFFFFFFFu;
      }
#pragma unroll
      for (int k = 0; k < kBN / 32; ++k) {
        const long n = n0 + lane + 32 * k;
        rcj[k] = n < g.cols ? __ldg(g.rcj + n) : 0.f;
      }
      if (nhc <= 32)
        for (int h = 0; h < nhc; ++h)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const long i = i0 + lane + 32 * k;
            if (i < g.rows && __ldg(g.wmask + i * g.H + hc0 + h) != 0) bits[k] |= 1u << h;
          }
      if (!mbar_wait(bar_vec_empty(b), ((t >> 1) & 1u) ^ 1u, abort_flag, status, kWaitSlab)) break;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v->rci[lane + 32 * k] = rci[k];
        v->bits[lane + 32 * k] = bits[k];
      }
#pragma unroll
      for (int k = 0; k < kBN / 32; ++k) v->rcj[lane + 32 * k] = rcj[k];
      mbar_arrive(bar_vec_full(b));
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // A thread owns one row of the tile and 16 of its columns at a time: what belongs to the row (reciprocal, mask bits) is
    // one register, what belongs to a column the same word for all lanes, and the trace block is read and written back in
    // 16-byte pieces of the thread's own row; the arithmetic is two-wide.  New traces leave from where the old ones landed,
    // weights from a buffer of the warp's own, both by TMA.  With four rows and eight scattered column pairs to a thread it
    // was 37 instructions an element and 5 million store requests of eight bytes a lane at 55296 x 3000; a tile took longer
    // here than in the tensor core.  Train step without a mask update, before and now: 1568 -> 30 x 100 at batch 128 30.8
    // and 23.3 us, 1568 -> 100 x 300 at 1024 541 and 494; 55296 -> 30 x 100 at 256 546 both (there it is memory, and the
    // fetches that wait for it).
    const int q = warp & 3, ch = warp >> 2;     // lane quarter, third of the tile's columns
    const int nchains = (g.kblocks + kChainKb - 1) / kChainKb;
    const uint32_t slabs = base + kSlabOffset + warp * kGroups * kSlab, wbuf = base + L::W_OFFSET + warp * kHalf;
    uint8_t *slab_row = smem + kSlabOffset + warp * kGroups * kSlab + lane * 128;
    uint8_t *w_row = smem + L::W_OFFSET + warp * kHalf + lane * 64;
    const uint64_t scale2 = pair_of(g.ema_scale, g.ema_scale), ln2 = pair_of(kLn2, kLn2);
    uint32_t chain = 0, tile = 0;
    bool ok = true;
    // this warp's block of the old trace: column group gr of tile w
    auto issue_slab = [&](uint32_t w, int gr) {
      int mt, nt;
      decode(w, mt, nt);
      mbar_arrive_expect_tx(bar_slab(warp, gr), kSlab);
      tma_load_2d(slabs + gr * kSlab, &tmC, nt * kBN + (ch * kGroups + gr) * 32, mt * 128 + 32 * q, bar_slab(warp, gr));
    };
    if (w_first < total && elect_one()) {
#pragma unroll
      for (int gr = 0; gr < kGroups; ++gr) issue_slab(w_first, gr);
    }
    for (uint32_t w = w_first; w < total && ok; w += w_step, ++tile) {
      int mt, nt;
      decode(w, mt, nt);
      const bool more = total - w > w_step;
      const int hc_first = first_hc(nt);
      const bool bits_ok = last_hc(nt) - hc_first < 32;
      const int row0 = mt * 128 + 32 * q;
      const TileVectors *v = reinterpret_cast<const TileVectors *>(smem + kVecOffset) + (tile & 1u);
      if (!mbar_wait_warp(bar_vec_full(tile & 1u), (tile >> 1) & 1u, abort_flag, status, kWaitSlab)) { ok = false; break; }
      const float r = v->rci[32 * q + lane];
      const uint64_t r2 = pair_of(r, r);
      for (int cc = 0; cc < nchains && ok; ++cc, ++chain) {
        const uint32_t buf = chain & 1u;
        if (!mbar_wait_warp(bar_acc_full(buf), (chain >> 1) & 1u, abort_flag, status, kWaitAccFull)) { ok = false; break; }
        __syncwarp();
        tc_fence_after();
        const uint32_t tacc = tmem_base + buf * kBN + ch * (kGroups * 32) + ((uint32_t)(32 * q) << 16);
        const bool last_chain = cc == nchains - 1;
        const float decay = cc == 0 ? g.one_minus : 1.f;   // the old trace decays once
        const uint64_t decay2 = pair_of(decay, decay);
#pragma unroll 1
        for (int gr = 0; gr < kGroups; ++gr) {
          if (cc == 0 && !mbar_wait_warp(bar_slab(warp, gr), tile & 1u, abort_flag, status, kWaitSlab)) { ok = false; break; }
          const int vc = (ch * kGroups + gr) * 32;           // first column of the group, in the tile
          const int gs = nt * kBN + vc;
          const bool inside = row0 < g.rows && gs < g.cols;   // (what lies past the edges of a block is clipped by TMA)
          uint32_t word = 0;   // bit k: the element in column k of the group keeps its weight
          if (last_chain && inside) {
            word = 0xFFFFFFFFu;
            if (g.wmask != nullptr) {
              word = 0;
              const uint32_t mb = v->bits[32 * q + lane];
              const int h1 = hc_of(min(gs + 32, g.cols) - 1);
              for (int h = hc_of(gs); h <= h1; ++h) {
                const int from = h * g.Mc - gs, to = from + g.Mc;   // the hypercolumn's columns in the group
                const uint32_t seg = (to < 32 ? (1u << to) - 1u : 0xFFFFFFFFu) & ~(from > 0 ? (1u << from) - 1u : 0u);
                const bool on = bits_ok ? (mb >> (h - hc_first)) & 1u
                                        : row0 + lane < g.rows && __ldg(g.wmask + (long)(row0 + lane) * g.H + h) != 0;
                if (on) word |= seg;
              }
            }
            const uint32_t live = __ballot_sync(0xFFFFFFFFu, v->rcj[vc + lane] != 0.f);   // columns at or above the threshold
            word = r != 0.f ? word & live : 0u;
          }
          uint8_t *sl = slab_row + gr * kSlab;
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            float a[16];
            __syncwarp();   // tcgen05.ld is warp-collective
            tmem_ld_32x32b_x16(tacc + gr * 32 + half * 16, a);
            uint64_t c[8];   // pairs of neighbouring columns
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const ulonglong2 old = *reinterpret_cast<const ulonglong2 *>(sl + (((half * 4 + k) ^ (lane & 7)) << 4));
              c[2 * k] = fma_pair(old.x, decay2, mul_pair(pair_of(a[4 * k], a[4 * k + 1]), scale2));
              c[2 * k + 1] = fma_pair(old.y, decay2, mul_pair(pair_of(a[4 * k + 2], a[4 * k + 3]), scale2));
            }
            if (!last_chain) {   // the running sum stays in shared memory
#pragma unroll
              for (int k = 0; k < 4; ++k)
                *reinterpret_cast<ulonglong2 *>(sl + (((half * 4 + k) ^ (lane & 7)) << 4)) = make_ulonglong2(c[2 * k], c[2 * k + 1]);
              continue;
            }
            const uint32_t sel = word >> (16 * half);
            float wv[16];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              float2 t = halves(c[k]);
              t.x = fmaxf(t.x, 0.f);
              t.y = fmaxf(t.y, 0.f);
              c[k] = pair_of(t.x, t.y);
              const uint64_t rc = mul_pair(r2, *reinterpret_cast<const uint64_t *>(v->rcj + vc + half * 16 + 2 * k));
              const float2 arg = halves(mul_pair(pair_of(fmaxf(t.x, g.cthr4), fmaxf(t.y, g.cthr4)), rc));
              float2 l;
              if (g.normal) {
                l = halves(mul_pair(pair_of(lg2_ftz(arg.x), lg2_ftz(arg.y)), ln2));
              } else {
                l = make_float2(__logf(arg.x), __logf(arg.y));
              }
              wv[2 * k] = sel & (1u << (2 * k)) ? l.x : 0.f;
              wv[2 * k + 1] = sel & (2u << (2 * k)) ? l.y : 0.f;
            }
            if (elect_one()) {   // the weights before these have left their buffer, and the traces the block before this one
              bulk_wait_read_0();
              if (half == 0 && gr > 0 && more) issue_slab(w + w_step, gr - 1);
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              *reinterpret_cast<ulonglong2 *>(sl + (((half * 4 + k) ^ (lane & 7)) << 4)) = make_ulonglong2(c[2 * k], c[2 * k + 1]);
              *reinterpret_cast<float4 *>(w_row + ((k ^ (lane >> 1 & 3)) << 4)) =
                  make_float4(wv[4 * k], wv[4 * k + 1], wv[4 * k + 2], wv[4 * k + 3]);
            }
            // every lane's accesses must have been performed, not merely issued, before TMA reads or overwrites the blocks
            fence_async_smem();
            __syncwarp();
            if (inside && elect_one()) {
              tma_store_2d(&tmW, wbuf, gs + half * 16, row0);
              if (half == 1) tma_store_2d(&tmC, slabs + gr * kSlab, gs, row0);
              bulk_commit();
            }
          }
        }
        if (!ok) break;
        // the accumulator may be overwritten (the leader's MMA warp waits for both CTAs' epilogue warps)
        tc_fence_before();
        __syncwarp();
        if (elect_one()) {
          leader_arrive(bar_acc_empty(buf));
          if (last_chain) {
            mbar_arrive(bar_vec_empty(tile & 1u));
            if (more) {
              bulk_wait_read_0();
              issue_slab(w + w_step, kGroups - 1);
            }
          }
        }
      }
    }
    if (elect_one()) bulk_wait_all();   // what this warp has sent by TMA has landed before the CTA retires
  }

  // ------------------------------------------------------------ tear-down
  __syncwarp();
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // neither CTA retires while the other may still signal it or read its operands
  else __syncthreads();
  if (warp == kMma) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

// Multiplier for n / d by multiply-high, or 0 if it is not exact for every n < limit.
uint32_t exact_division_magic(long d, long limit) {
  if (d <= 1 || d >= (1L << 31) || limit >= (1L << 31)) return 0;
  static thread_local long known_d = -1, known_limit = -1;   // verified once per layer shape and host thread
  static thread_local uint32_t known = 0;
  if (known_d == d && known_limit == limit) return known;
  const uint64_t magic = ((1ull << 32) + (uint64_t)d - 1) / (uint64_t)d;
  uint32_t m = (magic >> 32) ? 0 : (uint32_t)magic;
  for (long n = 0; n < limit && m != 0; ++n)
    if ((long)(((uint64_t)n * magic) >> 32) != n / d) m = 0;
  known_d = d;
  known_limit = limit;
  known = m;
  return m;
}

}  // namespace

cudaError_t launch_trace_update_tc(const float *x, long ldx, const float *y, long B, long N, long M, long H, const float *rci,
                                   const float *rcj, float *Cij, float *w, const uint8_t *wmask, TraceParams<float> p,
                                   cudaStream_t st) {
  if (!tc_available() || !tc_shape_ok(x, y, N, M) || ldx % 4 != 0 || !tc_shape_ok(Cij, w, N, M))
    return cudaErrorNotSupported;
  TcHost host;
  if (!tc_host(&host)) return cudaErrorMemoryAllocation;
  CUtensorMap ma, mb, ma3, mb3, mc, mw;
  if (!tc_map_2d(&ma, x, N, B, ldx, 32, kBK, kMapMnMajor) || !tc_map_2d(&mb, y, M, B, M, 32, kBK, kMapMnMajor) ||
      !tc_map_2d(&mc, Cij, M, N, M, 32, 32, kMapRows) || !tc_map_2d(&mw, w, M, N, M, 16, 32, kMapRows64))
    return cudaErrorInvalidValue;
  const bool a3 = N % 32 == 0 && tc_map_chunks(&ma3, x, N, B, ldx, kBK, 4), b3 = tc_map_chunks(&mb3, y, M, B, M, kBK, (host.pairs ? Layout<true>::BNH : Layout<false>::BNH) / 32);
  if (!a3) ma3 = ma;
  if (!b3) mb3 = mb;
  Trace g{};
  g.m_units = (int)(host.pairs ? (N + 255) / 256 : (N + 127) / 128);
  g.n_tiles = (int)((M + kBN - 1) / kBN);
  g.kblocks = (int)((B + kBK - 1) / kBK);
  g.m_fastest = M > N ? 1 : 0;   // consecutive tiles re-use the larger operand
  g.a_box3 = a3;
  g.b_box3_tiles = b3 ? (int)(M / 32 * 32 / kBN) : 0;
  g.lose_arrive = host.lose_arrive;
  g.wait_limit = host.wait_limit;
  g.rows = (int)N;
  g.cols = (int)M;
  g.rci = rci;
  g.rcj = rcj;
  g.wmask = wmask;
  g.H = (int)H;
  g.Mc = (int)(H > 0 ? M / H : M);
  g.hc_magic = wmask ? exact_division_magic(g.Mc, M + 2) : 0;
  g.normal = p.cthr4 >= 1e-30f;
  g.one_minus = p.one_minus;
  g.cthr4 = p.cthr4;
  g.ema_scale = p.taupdt / p.batch;

  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  const long units = (long)g.m_units * g.n_tiles;
  if (!host.pairs) {
    using L = Layout<false>;
    static std::atomic<bool> configured[64];
    if (!configured[dev].load()) {
      const cudaError_t e = cudaFuncSetAttribute(trace_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
      if (e != cudaSuccess) return e;
      configured[dev].store(true);
    }
    const cudaError_t e = launch_next(trace_kernel<false>, (unsigned)(units < host.sms ? units : host.sms), kThreads, L::SMEM, st,
                                      ma, mb, ma3, mb3, mc, mw, g, host.status);
    if (e == cudaSuccess) count_launches(1);
    return e;
  }
  using L = Layout<true>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = L::SMEM;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  static std::atomic<int> max_clusters[64];   // resident pairs (one CTA per SM; pairs must share a GPC's SMs)
  if (max_clusters[dev].load() == 0) {
    cudaError_t e = cudaFuncSetAttribute(trace_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (e != cudaSuccess) return e;
    cfg.gridDim = dim3((unsigned)(host.sms / 2 * 2), 1, 1);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, trace_kernel<true>, &cfg) != cudaSuccess || n <= 0 || n > host.sms / 2) n = host.sms / 2;
    max_clusters[dev].store(n);
  }
  const long clusters = units < max_clusters[dev].load() ? units : max_clusters[dev].load();
  cfg.gridDim = dim3((unsigned)(2 * clusters), 1, 1);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as launch_next
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, trace_kernel<true>, ma, mb, ma3, mb3, mc, mw, g, host.status);
  if (e == cudaSuccess) {
    count_launches(1);
    tc_count_pair_launch();
  }
  return e;
}

}  // namespace sbb
