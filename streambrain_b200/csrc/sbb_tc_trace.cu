// The fused trace step on the 5th-generation tensor cores.
//
//   D[i, j] = sum_b x[b, i] * y[b, j],   Cij = max(0, (1 - tau) Cij + tau / B * D),   W = log(Cij / (Ci Cj)) under the mask
//
// float32 operands as split TF32 products (hi*hi + hi*lo + lo*hi, see sbb_tc_kernels.cu): A's parts go to tensor memory,
// B's low part beside the raw tile in shared memory.  A cluster of two CTAs works on 256 rows x 192 columns
// (tcgen05.mma.cta_group::2); each CTA stages and splits its own 128 rows of A and half of the columns of B.  (!PAIR, what
// SBB_TC_PAIR=0 selects: one CTA works on 128 rows x 192 columns by itself and stages all columns of B, which leaves room
// for three stages; the products, chains and sums are the same.  It is there to compare with and for
// devices that cannot place pairs.  Train step without a mask update: 1568 -> 30 x 100 at batch 128 32.1 us in pairs, 33.2
// without; 55296 -> 30 x 100 at 256 565 and 686 us.)
// Roles in a CTA (672 threads, one CTA per SM, tiles walked persistently):
//   warps 0-11   epilogue: accumulator, old trace (by TMA, the whole tile's blocks one tile ahead), arithmetic, stores
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
struct TileVectors {
  float rci[128], rcj[kBN];     // reciprocals of Ci and Cj, 0 below the threshold
  uint32_t bits[128];           // per row: bit k = mask of hypercolumn (the tile's first) + k
};
template <bool PAIR>
struct Layout {
  static constexpr int BNH = PAIR ? kBN / 2 : kBN;   // columns of B a CTA stages
  static constexpr int STAGES = PAIR ? 4 : 3;        // (tensor memory holds the A parts of four stages)
  static constexpr int B_BYTES = BNH * kBK * 4;
  static constexpr int TX = kABytes + B_BYTES, STAGE = TX + B_BYTES;   // [A | B | B lo]
  static_assert(kTmemA + STAGES * 2 * kBK <= 512, "tensor memory budget");
  static_assert(STAGE % 1024 == 0 && kABytes % 1024 == 0 && TX % 1024 == 0, "swizzle alignment");
  static constexpr int SLAB_OFFSET = STAGES * STAGE;
  static constexpr int VEC_OFFSET = SLAB_OFFSET + kEpi * kGroups * kSlab;
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
  long rows, cols;            // N, M
  const float *rci, *rcj;
  float *Cij, *W;
  const uint8_t *wmask;
  uint32_t hc_magic;          // ceil(2^32 / Mc) where that divides every column exactly, else 0
  long H, Mc;
  int fast_ok;                // select words usable: Mc >= 32 (or no mask) and cthr^4 a normal float
  float one_minus, cthr4, ema_scale;
};

template <bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
    trace_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmA3, const __grid_constant__ CUtensorMap tmB3,
                 const __grid_constant__ CUtensorMap tmC, const Trace g, int *status) {
  using L = Layout<PAIR>;
  constexpr int kStages = L::STAGES, kStage = L::STAGE, kBNH = L::BNH, kBBytes = L::B_BYTES, kTx = L::TX;
  constexpr int kSlabOffset = L::SLAB_OFFSET, kVecOffset = L::VEC_OFFSET;
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
  after_previous();   // (barriers and tensor memory are set up while the kernel before ends)

  // The clusters walk the tiles side by side, columns fastest (rows fastest where the columns are the longer side): at any
  // time they share the operands of a few row tiles.
  const long total = (long)g.m_units * g.n_tiles;
  const long w_first = PAIR ? blockIdx.x >> 1 : blockIdx.x, w_step = PAIR ? gridDim.x >> 1 : gridDim.x;
  auto decode = [&](long w, int &mt, int &nt) {
    if (g.m_fastest) {
      mt = (int)(w % g.m_units);
      nt = (int)(w / g.m_units);
    } else {
      nt = (int)(w % g.n_tiles);
      mt = (int)(w / g.n_tiles);
    }
    if (PAIR) mt = 2 * mt + (int)rank;   // may be one past the last row tile: such a CTA stages zeros and stores nothing
  };
  auto hc_of = [&](long n) -> int { return g.hc_magic ? (int)__umulhi((uint32_t)n, g.hc_magic) : (int)(n / g.Mc); };
  auto first_hc = [&](int nt) -> int { return g.wmask ? hc_of((long)nt * kBN) : 0; };
  auto last_hc = [&](int nt) -> int {
    const long n = (long)nt * kBN + kBN - 1;
    return g.wmask ? hc_of(n < g.cols ? n : g.cols - 1) : 0;
  };

  if (warp == kTma) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (long w = w_first; w < total && ok; w += w_step) {
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
      for (long w = w_first; w < total && ok; w += w_step) {
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
            const uint32_t ta = tmem_base + kTmemA + s * (2 * kBK);
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
    for (long w = w_first; w < total && ok; w += w_step)
      for (int kb = 0; kb < g.kblocks; ++kb, ++it) {
        const int s = it % kStages;
        if (!mbar_wait(bar_full(s), (it / kStages) & 1u, abort_flag, status, kWaitFull)) { ok = false; break; }
        // MN-major tile [32-row chunk][k][32 rows]: element (k, m) of chunk m / 32 sits in the 128-byte line k at 32-byte
        // piece ((m % 32) / 8) ^ (k % 4); a warp reads one line per k
        const uint8_t *acol = smem + s * kStage + cw * (kBK * 128) + ((lane & 7) << 2);
        uint32_t r[kBK];
#pragma unroll
        for (int k = 0; k < kBK; ++k)
          r[k] = *reinterpret_cast<const uint32_t *>(acol + k * 128 + (((lane >> 3) ^ (k & 3)) << 5));
        const uint32_t ta = tmem_base + kTmemA + s * (2 * kBK) + ((uint32_t)(cw * 32) << 16);
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
    for (long w = w_first; w < total && ok; w += w_step)
      for (int kb = 0; kb < g.kblocks; ++kb, ++it) {
        const int s = it % kStages;
        if (!mbar_wait(bar_full(s), (it / kStages) & 1u, abort_flag, status, kWaitFull)) { ok = false; break; }
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
    for (long w = w_first; w < total; w += w_step, ++t) {
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
    // Thread (lane) owns four tile rows (16*hh + lane/4 + 8*rr) of its warp's TMEM lane quarter and, per 32-column group,
    // the column pairs 8*rep + 2*(lane%4) + {0,1}: four lanes cover 32 contiguous bytes of a row.
    const int q = warp & 3, ch = warp >> 2;     // lane quarter, third of the tile's columns
    const int lr = lane >> 2, lc = (lane & 3) * 2;
    uint32_t swz[4];                            // byte offset of column pair `rep` inside a swizzled 128-byte row
#pragma unroll
    for (int rep = 0; rep < 4; ++rep) swz[rep] = ((uint32_t)((2 * rep + (lc >> 2)) ^ lr) << 4) + (uint32_t)(lc & 3) * 4u;
    const long w_minus_c = g.W - g.Cij;         // the weight of an element sits this far from its trace
    const int nchains = (g.kblocks + kChainKb - 1) / kChainKb;
    const bool has_mask = g.wmask != nullptr;
    uint32_t chain = 0, tile = 0;
    bool ok = true;
    // this warp's block of the old trace: column group gr of tile (mt, nt)
    auto issue_slab = [&](int mt, int nt, int gr) {
      mbar_arrive_expect_tx(bar_slab(warp, gr), kSlab);
      tma_load_2d(base + kSlabOffset + (warp * kGroups + gr) * kSlab, &tmC, nt * kBN + (ch * kGroups + gr) * 32, mt * 128 + 32 * q,
                  bar_slab(warp, gr));
    };
    if (lane == 0 && w_first < total) {
      int mt, nt;
      decode(w_first, mt, nt);
#pragma unroll
      for (int gr = 0; gr < kGroups; ++gr) issue_slab(mt, nt, gr);
    }
    for (long w = w_first; w < total && ok; w += w_step, ++tile) {
      int mt, nt, mt_next = 0, nt_next = 0;
      decode(w, mt, nt);
      if (w + w_step < total) decode(w + w_step, mt_next, nt_next);
      const int hc_first = first_hc(nt);
      const bool bits_ok = last_hc(nt) - hc_first < 32;
      const bool tile_fast = g.fast_ok && (long)mt * 128 + 128 <= g.rows;
      const TileVectors *v = reinterpret_cast<const TileVectors *>(smem + kVecOffset) + (tile & 1u);
      if (!mbar_wait(bar_vec_full(tile & 1u), (tile >> 1) & 1u, abort_flag, status, kWaitSlab)) { ok = false; break; }
      for (int cc = 0; cc < nchains && ok; ++cc, ++chain) {
        const uint32_t buf = chain & 1u;
        if (!mbar_wait(bar_acc_full(buf), (chain >> 1) & 1u, abort_flag, status, kWaitAccFull)) { ok = false; break; }
        __syncwarp();
        tc_fence_after();
        const uint32_t tacc = tmem_base + buf * kBN + ch * (kGroups * 32) + ((uint32_t)(32 * q) << 16);
        const bool last_chain = cc == nchains - 1;
        const float decay = cc == 0 ? g.one_minus : 1.f;   // the old trace decays once
#pragma unroll 1
        for (int gr = 0; gr < kGroups; ++gr) {
          if (cc == 0 && !mbar_wait(bar_slab(warp, gr), tile & 1u, abort_flag, status, kWaitSlab)) { ok = false; break; }
          uint8_t *sl = smem + kSlabOffset + (warp * kGroups + gr) * kSlab + lr * 128;
          const int vc = (ch * kGroups + gr) * 32;           // first column of the group, in the tile
          const long gs = (long)nt * kBN + vc;
          // whole blocks with at most two hypercolumns: one select word per row, bit 8*rep + e = "element e of column
          // pair rep keeps its weight"
          const bool g_fast = tile_fast && gs + 32 <= g.cols;
          uint32_t live32 = 0, first32 = 0xFFFFFFFFu;   // columns at or above the threshold; of the first hypercolumn
          int k0 = 0;
          if (last_chain && g_fast) {
            live32 = __ballot_sync(0xFFFFFFFFu, v->rcj[vc + lane] != 0.f);
            if (has_mask) {
              const int hc0 = hc_of(gs);
              const long bnd = (long)(hc0 + 1) * g.Mc - gs;
              if (bnd < 32) first32 = (1u << bnd) - 1u;
              k0 = hc0 - hc_first;
            }
          }
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            float a[16];
            __syncwarp();   // tcgen05.ld is warp-collective
            tmem_ld_16x256b_x4(tacc + gr * 32 + ((uint32_t)(16 * hh) << 16), a);
            float2 c[2][4];
#pragma unroll
            for (int rr = 0; rr < 2; ++rr)
#pragma unroll
              for (int rep = 0; rep < 4; ++rep) {
                float2 c2 = *reinterpret_cast<const float2 *>(sl + (16 * hh + 8 * rr) * 128 + swz[rep]);
                c2.x = fmaf(c2.x, decay, a[rep * 4 + rr * 2 + 0] * g.ema_scale);
                c2.y = fmaf(c2.y, decay, a[rep * 4 + rr * 2 + 1] * g.ema_scale);
                c[rr][rep] = c2;
              }
            if (!last_chain) {   // the running sum stays in shared memory
#pragma unroll
              for (int rr = 0; rr < 2; ++rr)
#pragma unroll
                for (int rep = 0; rep < 4; ++rep)
                  *reinterpret_cast<float2 *>(sl + (16 * hh + 8 * rr) * 128 + swz[rep]) = c[rr][rep];
              continue;
            }
            if (hh == 1) {
              // the block is about to be overwritten by TMA: every lane's accesses must have been performed, not merely issued
              fence_async_smem();
              __syncwarp();
              if (lane == 0 && w + w_step < total) issue_slab(mt_next, nt_next, gr);
            }
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
              const int vr = 32 * q + 16 * hh + 8 * rr + lr;
              const long i = (long)mt * 128 + vr;
              float *cp = g.Cij + i * g.cols + gs + lc;
              const float r = v->rci[vr];
              const uint32_t mb = v->bits[vr];
              if (g_fast) {
                const uint32_t m0 = 0u - ((mb >> k0) & 1u), m1 = 0u - ((mb >> (k0 + 1)) & 1u);
                const uint32_t word = ((m0 & first32) | (m1 & ~first32)) & live32;
                const uint32_t sel = r != 0.f ? (word >> lc) & 0x03030303u : 0u;
#pragma unroll
                for (int rep = 0; rep < 4; ++rep) {
                  const float2 rcj = *reinterpret_cast<const float2 *>(v->rcj + vc + lc + rep * 8);
                  float2 c2 = c[rr][rep];
                  c2.x = fmaxf(c2.x, 0.f);
                  c2.y = fmaxf(c2.y, 0.f);
                  const float wx = lg2_ftz(fmaxf(c2.x, g.cthr4) * (r * rcj.x)) * kLn2;
                  const float wy = lg2_ftz(fmaxf(c2.y, g.cthr4) * (r * rcj.y)) * kLn2;
                  __stcs(reinterpret_cast<float2 *>(cp + rep * 8), c2);
                  __stcs(reinterpret_cast<float2 *>(cp + w_minus_c + rep * 8),
                         make_float2((sel & (1u << (8 * rep))) ? wx : 0.f, (sel & (2u << (8 * rep))) ? wy : 0.f));
                }
              } else if (i < g.rows) {   // edges, narrow hypercolumns: every element checked
#pragma unroll
                for (int rep = 0; rep < 4; ++rep) {
                  const long n = gs + lc + rep * 8;
                  if (!(n < g.cols)) continue;   // cols is even: n + 1 is in range too
                  const float2 rcj = *reinterpret_cast<const float2 *>(v->rcj + vc + lc + rep * 8);
                  float2 c2 = c[rr][rep];
                  c2.x = fmaxf(c2.x, 0.f);
                  c2.y = fmaxf(c2.y, 0.f);
                  bool on0 = r != 0.f && rcj.x != 0.f, on1 = r != 0.f && rcj.y != 0.f;
                  if (has_mask) {
                    const uint8_t *mr = g.wmask + i * g.H;
                    const int h0 = hc_of(n), h1 = hc_of(n + 1);
                    on0 = on0 && (bits_ok ? (mb >> (h0 - hc_first)) & 1u : (uint32_t)__ldg(mr + h0)) != 0;
                    on1 = on1 && (bits_ok ? (mb >> (h1 - hc_first)) & 1u : (uint32_t)__ldg(mr + h1)) != 0;
                  }
                  const float wx = __logf(fmaxf(c2.x, g.cthr4) * (r * rcj.x));
                  const float wy = __logf(fmaxf(c2.y, g.cthr4) * (r * rcj.y));
                  __stcs(reinterpret_cast<float2 *>(cp + rep * 8), c2);
                  __stcs(reinterpret_cast<float2 *>(cp + w_minus_c + rep * 8), make_float2(on0 ? wx : 0.f, on1 ? wy : 0.f));
                }
              }
            }
          }
        }
        if (!ok) break;
        // the accumulator may be overwritten (the leader's MMA warp waits for both CTAs' epilogue warps)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          leader_arrive(bar_acc_empty(buf));
          if (last_chain) mbar_arrive(bar_vec_empty(tile & 1u));
        }
      }
    }
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

cudaError_t launch_trace_update_tc(const float *x, const float *y, long B, long N, long M, long H, const float *rci,
                                   const float *rcj, float *Cij, float *w, const uint8_t *wmask, TraceParams<float> p,
                                   cudaStream_t st) {
  if (!tc_available() || !tc_shape_ok(x, y, N, M) || !tc_shape_ok(Cij, Cij, N, M) || (reinterpret_cast<uintptr_t>(w) & 7u))
    return cudaErrorNotSupported;
  TcHost host;
  if (!tc_host(&host)) return cudaErrorMemoryAllocation;
  CUtensorMap ma, mb, ma3, mb3, mc;
  if (!tc_map_2d(&ma, x, N, B, 32, kBK, true) || !tc_map_2d(&mb, y, M, B, 32, kBK, true) ||
      !tc_map_2d(&mc, Cij, M, N, 32, 32, false))
    return cudaErrorInvalidValue;
  const bool a3 = N % 32 == 0 && tc_map_chunks(&ma3, x, N, B, kBK, 4), b3 = tc_map_chunks(&mb3, y, M, B, kBK, (host.pairs ? Layout<true>::BNH : Layout<false>::BNH) / 32);
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
  g.rows = N;
  g.cols = M;
  g.rci = rci;
  g.rcj = rcj;
  g.Cij = Cij;
  g.W = w;
  g.wmask = wmask;
  g.H = H;
  g.Mc = H > 0 ? M / H : M;
  g.hc_magic = wmask ? exact_division_magic(g.Mc, M + 2) : 0;
  g.fast_ok = (wmask == nullptr || g.Mc >= 32) && p.cthr4 >= 1e-30f;
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
                                      ma, mb, ma3, mb3, mc, g, host.status);
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
  const cudaError_t e = cudaLaunchKernelEx(&cfg, trace_kernel<true>, ma, mb, ma3, mb3, mc, g, host.status);
  if (e == cudaSuccess) {
    count_launches(1);
    tc_count_pair_launch();
  }
  return e;
}

}  // namespace sbb
