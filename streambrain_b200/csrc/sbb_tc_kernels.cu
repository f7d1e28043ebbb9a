// tcgen05 / TMEM / TMA contraction kernels for sm_100a.
//
// One persistent, warp-specialised kernel template serves the forward product and the raw batch product of the
// data-parallel step (the fused trace step of one device: sbb_tc_trace.cu):
//
//   raw product    D[i, j] = sum_b x[b, i] * y[b, j]   A = x  (MN-major), B = y (MN-major), K = batch
//   forward        D[b, j] = sum_k x[b, k] * w[k, j]   A = x  (K-major),  B = w (MN-major), K = in_features
//
// float32 accuracy on TF32 tensor cores: every operand value v is used as
// hi = v truncated to TF32 (what the tensor core reads of the raw float32) and
// lo = tf32(v - hi), and each k-step issues three MMAs  hi*hi + hi*lo + lo*hi
// into one float32 accumulator in tensor memory (the dropped lo*lo term is
// below 2^-20 relative).  A's hi and lo parts are staged in tensor memory, B's
// lo parts beside the raw tile in shared memory: the tensor core fetches only B
// from shared memory.
//
// Roles inside a CTA (512 threads, one CTA per SM, tiles walked persistently):
//   warps 0-3   A converters: wait for a TMA stage, write A's hi / lo parts to tensor
//               memory (one tile row per thread)
//               and (raw products) B's lo parts to shared memory
//   warps 14-15 B converters (forward product): B's lo parts to shared memory
//   warps 4-11  epilogue: tcgen05.ld the accumulator (16x256b shape, so that four
//               lanes cover 32 contiguous bytes of a row), add up the chains and store
//   warp 12     TMA producer (one lane): cp.async.bulk.tensor loads, no multicast
//   warp 13     MMA issuer (one lane) and owner of the TMEM allocation
// CTA pairs (PAIR; the forward product): the kernel is launched in clusters of
// two CTAs that work on two vertically adjacent row tiles with one 256-row tcgen05.mma.cta_group::2 per k-step,
// issued by the leader CTA.  Each CTA stages and converts its own 128 rows of A into its own tensor memory and
// half of the tile's columns of B into its own shared memory; the converters and the epilogue warps of both
// CTAs report to the leader's mbarriers (mapa + remote arrive), tcgen05.commit with a cluster multicast reports
// back to both.  No TMA load uses multicast: every CTA loads into its own shared memory only.
// Hand-offs use mbarriers; every wait is bounded by a count of SM clock cycles:
// a wait that gives up records a code in a global status word, raises the CTA's
// abort flag, and every role falls through to the common tear-down (drain the
// tensor pipe, free TMEM) instead of spinning.
#include "sbb_tc.cuh"
#include "sbb_tc_ptx.cuh"

#include <atomic>
#include <cstdlib>
#include <mutex>

#include "sbb_launch.cuh"
#include "sbb_math.cuh"

namespace sbb {
namespace {

constexpr int kConvWarps = 4;
constexpr int kEpiWarps = 8;
constexpr int kTmaWarp = kConvWarps + kEpiWarps;
constexpr int kMmaWarp = kTmaWarp + 1;
constexpr int kBConvWarps = 2;                 // warps kMmaWarp + 1 ..: the low parts of B
constexpr int kThreads = (kMmaWarp + 1 + kBConvWarps) * 32;  // 512: with 128 registers each, the whole register file
struct TcWork {
  int m_tiles, n_tiles, splits;
  int k_total;      // extent of the reduction dimension
  int k_per_split;  // multiple of the stage depth
  int m_fastest;    // tile order: row tiles fastest (1) or column tiles fastest (0)
  int a_row0;       // offset added to the A row coordinate (first output row of this launch)
  int a_box3;       // A stage fetched by one 3-D box (MN-major A whose row length is a multiple of 32)
  int b_box3_tiles; // column tiles [0, b_box3_tiles) fetch their B stage by one 3-D box
  int b_prefetch;   // B k-blocks requested into L2 ahead of the load into shared memory (0 = none)
  long long wait_limit;  // SM clock cycles after which a wait on an mbarrier gives up
  int lose_arrive;  // test hook: converter thread 0 of CTA 0 skips its arrival for the first stage
};

struct TcEpilogue {
  // raw store: out[(split*rows + m)*ld + n]
  float *out;
  long rows, cols, ld;
  // raw store of an MN-major product: the tile leaves through shared memory and TMA stores of 32 x 32 blocks
  // (tmC = the output, row 0 = first row of this launch) instead of register stores: whole 128-byte rows per
  // request, which is what a destination in another GPU's memory needs to be written at link speed
  int tma_store;
};

// Optional timeline (compile with -DSBB_TC_TRACE): CTA 0 stamps clock64() at the hand-offs of its first
// 64 tiles -- event numbers: 0 / 8 first / last TMA issue, 5 / 9 first / last conversion, 7 accumulator
// free, 1 first MMA, 2 accumulator committed, 3 epilogue start, 10 epilogue data ready, 13-15 column
// groups done, 4 epilogue end -- and sbb_tc_trace_read copies the 64 x 16 stamps out.  Compiled out otherwise.
#ifdef SBB_TC_TRACE
__device__ unsigned long long g_tc_trace[64 * 16];
#define TC_TRACE(tile, ev) do { if (blockIdx.x == 0 && (tile) < 64) g_tc_trace[(tile) * 16 + (ev)] = (unsigned long long)clock64(); } while (0)
#else
#define TC_TRACE(tile, ev)
#endif

// ------------------------------------------------------------------ the kernel
constexpr int kSlabBytes = 32 * 32 * 4;  // one epilogue warp's 32-row x 32-column block of the output

// The A operand's hi / lo parts live in tensor memory (written by the converters), so only B
// has a "lo" copy in shared memory and the tensor core fetches only B from there.
// PRESPLIT: the low parts of both operands come from memory (written by the column-sum kernels that run just
// before), so a stage is four TMA landing zones [A | B | B lo | A lo], nothing is converted inside the kernel
// and the tensor core takes both operands from shared memory.
// PAIR: two CTAs share one 256-row MMA; each stages its own 128 rows of A and BN / 2 columns of B.
template <int BN, int BK, int STAGES, bool SLABS, bool PRESPLIT = false, bool PAIR = false>
struct TcSmem {
  static constexpr int A_BYTES = 128 * BK * 4;
  static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * BK * 4;
  static constexpr int RAW_BYTES = A_BYTES + B_BYTES;  // TMA landing zone: the raw values serve as "hi"
  static constexpr int STAGE_BYTES = PRESPLIT ? 2 * RAW_BYTES : RAW_BYTES + B_BYTES;   // + B's lo parts (+ A's)
  static constexpr int TX_BYTES = PRESPLIT ? 2 * RAW_BYTES : RAW_BYTES;                // bytes TMA lands per stage
  // tensor memory: two accumulators, then (not PRESPLIT) per stage BK columns of A hi and BK of A lo
  static constexpr int TMEM_A_COL = 2 * BN;
  static constexpr int TMEM_COLS = 512;
  // A's parts of this many k-blocks fit beside the accumulators; shared memory may hold more stages than that
  static constexpr int SLOTS = (TMEM_COLS - 2 * BN) / (2 * BK) < STAGES ? (TMEM_COLS - 2 * BN) / (2 * BK) : STAGES;
  static_assert(PRESPLIT || SLOTS >= 2, "tensor memory budget");
  static_assert(STAGE_BYTES % 1024 == 0, "stages keep the 1024-byte swizzle alignment");
  static constexpr int SLAB_OFFSET = STAGES * STAGE_BYTES;
  // two 32 x 32 block buffers per epilogue warp: staging for the TMA stores of the raw product
  static constexpr int SLAB_TOTAL = SLABS ? kEpiWarps * 2 * kSlabBytes : 0;
  static constexpr int BAR_OFFSET = SLAB_OFFSET + SLAB_TOTAL;
  // full, conv, empty per stage; acc_full[2], acc_empty[2], drain; slab[warp][2]
  static constexpr int NUM_BARS = 3 * STAGES + 5 + 2 * kEpiWarps;
  static constexpr int TOTAL = BAR_OFFSET + NUM_BARS * 8 + 16 + 1024;  // + tmem ptr, abort flag, alignment slack
  static_assert(TOTAL <= 232448, "shared memory budget");
};

// CHAIN = number of k-blocks accumulated in tensor memory before the running sum
// is taken over by float32 registers (0 = the whole k-range in tensor memory).
// The tensor core adds each MMA into its accumulator with less than IEEE
// rounding, so the error of a chain grows with its length; long reductions
// (the forward pass sums over in_features) are cut into short chains whose
// results the epilogue warps add in full float32.
template <bool A_KMAJOR, int BN, int BK, int STAGES, int CHAIN, bool PRESPLIT = false, bool PAIR = false>
// (16 warps of 128 registers per thread: the whole register file, one CTA per SM)
__global__ void __launch_bounds__(kThreads, 1)
    tc_contraction_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ CUtensorMap tmA3, const __grid_constant__ CUtensorMap tmB3,
                          const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmAlo,
                          const __grid_constant__ CUtensorMap tmBlo, const __grid_constant__ CUtensorMap tmA3lo,
                          const __grid_constant__ CUtensorMap tmB3lo, TcWork wk, TcEpilogue ep, int *status) {
  using SM = TcSmem<BN, BK, STAGES, !A_KMAJOR, PRESPLIT, PAIR>;
  static_assert(!(PRESPLIT && A_KMAJOR), "pre-split operands are the two MN-major ones of the batch contractions");
  static_assert(!PAIR || (!PRESPLIT && BN % 64 == 0), "CTA pairs convert their operands themselves");
  // In a pair, CTA `rank` of the cluster works on row tile 2 * (pair's tile) + rank; the leader (rank 0) issues the MMAs.
  // B's low parts by the two extra warps (see their role below): forward product
  constexpr bool BWARPS = A_KMAJOR;
  const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
  constexpr int BNH = PAIR ? BN / 2 : BN;   // columns of B this CTA stages
  static_assert(!A_KMAJOR || BK == 32, "a K-major operand is loaded as one 128-byte-wide box");
  static_assert(BN % 64 == 0 && BN <= 256 && BK % 8 == 0 && BK <= 32, "tile shape");
  static_assert(CHAIN == 0 || BN <= 128, "register-resident running sums are sized for 128 columns");
  extern __shared__ uint8_t smem_dyn[];
  const uint32_t dyn_base = smem_u32(smem_dyn);
  const uint32_t base = (dyn_base + 1023u) & ~1023u;  // swizzle atoms need 1024-byte alignment
  uint8_t *smem = smem_dyn + (base - dyn_base);
  const uint32_t bars = base + SM::BAR_OFFSET;
  auto bar_full = [&](int s) { return bars + 8u * s; };
  auto bar_conv = [&](int s) { return bars + 8u * (STAGES + s); };
  auto bar_empty = [&](int s) { return bars + 8u * (2 * STAGES + s); };
  auto bar_acc_full = [&](int b) { return bars + 8u * (3 * STAGES + b); };
  auto bar_acc_empty = [&](int b) { return bars + 8u * (3 * STAGES + 2 + b); };
  const uint32_t bar_drain = bars + 8u * (3 * STAGES + 4);
  auto bar_slab = [&](int e, int b) { return bars + 8u * (3 * STAGES + 5 + 2 * e + b); };
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + SM::BAR_OFFSET + SM::NUM_BARS * 8);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform)

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_conv(s), (PAIR ? 2 : 1) * (kConvWarps + (BWARPS ? kBConvWarps : 0)) * 32);   // the leader's counts both CTAs' converters
      mbar_init(bar_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full(b), 1);
      mbar_init(bar_acc_empty(b), (PAIR ? 2 : 1) * kEpiWarps * 32);
    }
    mbar_init(bar_drain, 1);
    for (int e = 0; e < kEpiWarps; ++e) {
      mbar_init(bar_slab(e, 0), 1);
      mbar_init(bar_slab(e, 1), 1);
    }
    *abort_flag = 0;
    *reinterpret_cast<volatile long long *>(abort_flag + 1) = wk.wait_limit;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    if constexpr (PAIR) {
      tmem_alloc_pair(smem_u32(tmem_slot), SM::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_slot), SM::TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // the peer's barriers exist before anything arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  after_previous();   // (barriers and tensor memory are set up while the kernel before ends)

  // PAIR: the work items are pairs of row tiles, and the two CTAs of a cluster walk them together
  const int m_units = PAIR ? (wk.m_tiles + 1) / 2 : wk.m_tiles;
  const long total = (long)m_units * wk.n_tiles * wk.splits;
  const long w_first = PAIR ? (long)(blockIdx.x >> 1) : (long)blockIdx.x;
  const long w_step = PAIR ? (long)(gridDim.x >> 1) : (long)gridDim.x;
  // Decode a work index into (m_tile, n_tile, split) and its k-block range.
  auto decode = [&](long w, int &mt, int &nt, int &sp, int &kbeg, int &nkb) {
    if (wk.m_fastest) {
      mt = (int)(w % m_units);
      const long r = w / m_units;
      nt = (int)(r % wk.n_tiles);
      sp = (int)(r / wk.n_tiles);
    } else {
      nt = (int)(w % wk.n_tiles);
      const long r = w / wk.n_tiles;
      mt = (int)(r % m_units);
      sp = (int)(r / m_units);
    }
    if (PAIR) mt = 2 * mt + (int)rank;   // may be one past the last row tile: such a CTA stages zeros and stores nothing
    kbeg = sp * wk.k_per_split;
    const int kend = min(wk.k_total, kbeg + wk.k_per_split);
    nkb = (kend - kbeg + BK - 1) / BK;
  };

  if (warp == kTmaWarp) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (long w = w_first; w < total && ok; w += w_step) {
        int mt, nt, sp, kbeg, nkb;
        decode(w, mt, nt, sp, kbeg, nkb);
        auto prefetch_b = [&](int kb) {   // k-block kb of this unit's B operand -> L2
          const int k0 = kbeg + kb * BK;
          if (nt < wk.b_box3_tiles) {
            tma_prefetch_3d(&tmB3, 0, k0, nt * (BN / 32));
          } else {
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) tma_prefetch_2d(&tmB, nt * BN + 32 * c, k0);
          }
        };
        for (int kb = 0; kb < wk.b_prefetch && kb < nkb; ++kb) prefetch_b(kb);
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1u;
          if (wk.b_prefetch > 0 && kb + wk.b_prefetch < nkb) prefetch_b(kb + wk.b_prefetch);
          if (!mbar_wait(bar_empty(s), ph ^ 1u, abort_flag, status, kWaitEmpty)) { ok = false; break; }
          if (kb == 0) TC_TRACE((w - w_first) / w_step, 0);
          if (kb == nkb - 1) TC_TRACE((w - w_first) / w_step, 8);
          mbar_arrive_expect_tx(bar_full(s), SM::TX_BYTES);
          const uint32_t a_dst = base + s * SM::STAGE_BYTES;
          const uint32_t b_dst = a_dst + SM::A_BYTES;
          const int k0 = kbeg + kb * BK;
          if constexpr (PRESPLIT) {   // the low parts, same boxes from the low-part planes
            const uint32_t blo_dst = a_dst + SM::RAW_BYTES, alo_dst = blo_dst + SM::B_BYTES;
            if (wk.a_box3) {
              tma_load_3d(alo_dst, &tmA3lo, 0, k0, (wk.a_row0 + mt * 128) / 32, bar_full(s));
            } else {
#pragma unroll
              for (int c = 0; c < 4; ++c)
                tma_load_2d(alo_dst + c * (BK * 128), &tmAlo, wk.a_row0 + mt * 128 + 32 * c, k0, bar_full(s));
            }
            if (nt < wk.b_box3_tiles) {
              tma_load_3d(blo_dst, &tmB3lo, 0, k0, nt * (BN / 32), bar_full(s));
            } else {
#pragma unroll
              for (int c = 0; c < BN / 32; ++c)
                tma_load_2d(blo_dst + c * (BK * 128), &tmBlo, nt * BN + 32 * c, k0, bar_full(s));
            }
          }
          if (A_KMAJOR) {
            tma_load_2d(a_dst, &tmA, k0, wk.a_row0 + mt * 128, bar_full(s));
          } else if (wk.a_box3) {
            tma_load_3d(a_dst, &tmA3, 0, k0, (wk.a_row0 + mt * 128) / 32, bar_full(s));
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              tma_load_2d(a_dst + c * (BK * 128), &tmA, wk.a_row0 + mt * 128 + 32 * c, k0, bar_full(s));
          }
          // (PAIR: this CTA's half of the tile's columns; the 3-D map's box is BNH / 32 chunks deep)
          if (nt < wk.b_box3_tiles) {
            tma_load_3d(b_dst, &tmB3, 0, k0, nt * (BN / 32) + (int)rank * (BNH / 32), bar_full(s));
          } else {
#pragma unroll
            for (int c = 0; c < BNH / 32; ++c)
              tma_load_2d(b_dst + c * (BK * 128), &tmB, nt * BN + (int)rank * BNH + 32 * c, k0, bar_full(s));
          }
        }
      }
      if (!ok) {
        // Loads already issued still land in this CTA's shared memory: give them
        // a bounded moment before the CTA retires.
        const long long t0 = clock64();
        while (clock64() - t0 < 400000ll) {
        }
      }
    }
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    if (rank == 0 && elect_one()) {
      // D float32, A and B TF32; A (tensor memory) K-major, B (shared memory) MN-major
      // (PRESPLIT: A from shared memory too, MN-major like B; PAIR: 256 rows over the two CTAs)
      constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((PRESPLIT ? 1u : 0u) << 15) | (1u << 16) |
                                 ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((PAIR ? 256 : 128) >> 4) << 24);
      uint32_t it = 0, chain = 0;
      bool ok = true;
      for (long w = w_first; w < total && ok; w += w_step) {
        int mt, nt, sp, kbeg, nkb;
        decode(w, mt, nt, sp, kbeg, nkb);
        int kb = 0;
        while (kb < nkb && ok) {
          const uint32_t buf = chain & 1u, aph = (chain >> 1) & 1u;
          if (!mbar_wait(bar_acc_empty(buf), aph ^ 1u, abort_flag, status, kWaitAccEmpty)) { ok = false; break; }
          TC_TRACE(chain, 7);
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + buf * BN;
          const int kb_end = CHAIN > 0 ? min(nkb, kb + CHAIN) : nkb;
          for (bool first = true; kb < kb_end; ++kb, ++it) {
            const int s = it % STAGES;
            const uint32_t ph = (it / STAGES) & 1u;
            // the stage is ready when the converters have split it, or (PRESPLIT) as soon as TMA has landed it
            if (!mbar_wait(PRESPLIT ? bar_full(s) : bar_conv(s), ph, abort_flag, status, kWaitConv)) { ok = false; break; }
            if (first) TC_TRACE(chain, 1);
            tc_fence_after();
            const uint32_t b_hi = base + s * SM::STAGE_BYTES + SM::A_BYTES;
            const uint32_t b_lo = base + s * SM::STAGE_BYTES + SM::RAW_BYTES;
            const uint32_t ta_hi = tmem_base + SM::TMEM_A_COL + (it % SM::SLOTS) * (2 * BK);
#pragma unroll
            for (int kk = 0; kk < BK / 8; ++kk) {
              // One MMA consumes 8 k-values: 8 columns of A in tensor memory, eight 128-byte rows
              // (two 4-row swizzle atoms) of the MN-major B in shared memory.
              const uint64_t db_hi = smem_desc_mn(b_hi + kk * 1024, BK * 128);
              const uint64_t db_lo = smem_desc_mn(b_lo + kk * 1024, BK * 128);
              if constexpr (PRESPLIT) {
                const uint32_t a_hi = base + s * SM::STAGE_BYTES, a_lo = b_lo + SM::B_BYTES;
                const uint64_t da_hi = smem_desc_mn(a_hi + kk * 1024, BK * 128);
                const uint64_t da_lo = smem_desc_mn(a_lo + kk * 1024, BK * 128);
                mma_tf32_ss(d_tmem, da_lo, db_hi, idesc, (first && kk == 0) ? 0u : 1u);
                mma_tf32_ss(d_tmem, da_hi, db_lo, idesc, 1u);
                mma_tf32_ss(d_tmem, da_hi, db_hi, idesc, 1u);
              } else if constexpr (PAIR) {
                mma_tf32_ts_pair(d_tmem, ta_hi + BK + kk * 8, db_hi, idesc, (first && kk == 0) ? 0u : 1u);
                mma_tf32_ts_pair(d_tmem, ta_hi + kk * 8, db_lo, idesc, 1u);
                mma_tf32_ts_pair(d_tmem, ta_hi + kk * 8, db_hi, idesc, 1u);
              } else {
                mma_tf32_ts(d_tmem, ta_hi + BK + kk * 8, db_hi, idesc, (first && kk == 0) ? 0u : 1u);
                mma_tf32_ts(d_tmem, ta_hi + kk * 8, db_lo, idesc, 1u);
                mma_tf32_ts(d_tmem, ta_hi + kk * 8, db_hi, idesc, 1u);
              }
            }
            first = false;
            // the stage may be refilled once these MMAs have read it (PAIR: in both CTAs)
            if constexpr (PAIR) mma_commit_pair(bar_empty(s));
            else mma_commit(bar_empty(s));
          }
          if (ok) {
            TC_TRACE(chain, 2);
            if constexpr (PAIR) mma_commit_pair(bar_acc_full(buf));
            else mma_commit(bar_acc_full(buf));
            ++chain;
          }
        }
      }
      // Drain: nothing of this CTA may still be running in the tensor pipe when TMEM is freed.
      // (bounded by time alone: also a CTA that is giving up lets its MMAs in flight finish before TMEM goes)
      if constexpr (PAIR) mma_commit_pair(bar_drain);   // (the peer's copy of this barrier is not waited on)
      else mma_commit(bar_drain);
      if (!mbar_try_wait(bar_drain, 0)) mbar_wait_slow(bar_drain, 0, abort_flag, status, kWaitDrain, false);
    }
  } else if (warp < kConvWarps) {
    // ------------------------------------------------------------ hi / lo converters (idle when PRESPLIT)
    uint32_t it = 0;
    bool ok = true;
    for (long w = w_first; !PRESPLIT && w < total && ok; w += w_step) {
      int mt, nt, sp, kbeg, nkb;
      decode(w, mt, nt, sp, kbeg, nkb);
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1u;
        if (!mbar_wait_warp(bar_full(s), ph, abort_flag, status, kWaitFull)) { ok = false; break; }
        if (threadIdx.x == 0 && kb == 0) TC_TRACE((w - w_first) / w_step, 5);
        if (threadIdx.x == 0 && kb == nkb - 1) TC_TRACE((w - w_first) / w_step, 9);
        static_assert(kConvWarps == 4, "one A row (tensor-memory lane) per converter thread");
        // A: this thread's row of the tile goes to its lane of tensor memory, hi (the raw bits) in BK
        // columns and lo in the next BK.
        uint32_t r[BK];
        if constexpr (A_KMAJOR) {
          // K-major tile, 128-byte rows: 16-byte chunk c of row m sits at chunk c ^ (m % 8)
          static_assert(BK == 32, "a K-major row is one 128-byte swizzle span");
          const uint8_t *arow = smem + s * SM::STAGE_BYTES + threadIdx.x * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint4 q4 = *reinterpret_cast<const uint4 *>(arow + ((c ^ (threadIdx.x & 7)) << 4));
            r[4 * c + 0] = q4.x; r[4 * c + 1] = q4.y; r[4 * c + 2] = q4.z; r[4 * c + 3] = q4.w;
          }
        } else {
          // MN-major tile [32-row chunk][k][32 rows]: element (k, m) of chunk m / 32 sits in the
          // 128-byte line k at 32-byte piece ((m % 32) / 8) ^ (k % 4); a warp reads one line per k.
          const uint8_t *acol = smem + s * SM::STAGE_BYTES + warp * (BK * 128) + ((lane & 7) << 2);
#pragma unroll
          for (int k = 0; k < BK; ++k)
            r[k] = *reinterpret_cast<const uint32_t *>(acol + k * 128 + ((((lane >> 3) ^ (k & 3))) << 5));
        }
        if constexpr (SM::SLOTS < STAGES) {   // the k-block whose place in tensor memory this one takes has been multiplied
          if (it >= SM::SLOTS) {
            const uint32_t old = it - SM::SLOTS;
            if (!mbar_wait_warp(bar_empty(old % STAGES), (old / STAGES) & 1u, abort_flag, status, kWaitEmpty)) { ok = false; break; }
            tc_fence_after();
          }
        }
        const uint32_t ta = tmem_base + SM::TMEM_A_COL + (it % SM::SLOTS) * (2 * BK) + ((uint32_t)(warp * 32) << 16);
        tmem_st_32x32b<BK>(ta, r);
#pragma unroll
        for (int k = 0; k < BK; ++k) r[k] = __float_as_uint(tf32_lo(__uint_as_float(r[k])));
        tmem_st_32x32b<BK>(ta + BK, r);
        if constexpr (!BWARPS) {
          // B: lo parts beside the raw tile in shared memory.  Every load is issued before the first
          // store: the hand-off to the MMA warp costs one shared-memory round trip, not one per piece.
          constexpr int kConvThreads = kConvWarps * 32;
          const float4 *rawb = reinterpret_cast<const float4 *>(smem + s * SM::STAGE_BYTES + SM::A_BYTES);
          float4 *lob = reinterpret_cast<float4 *>(smem + s * SM::STAGE_BYTES + SM::RAW_BYTES);
          constexpr int kPieces = SM::B_BYTES / 16 / kConvThreads;
          static_assert(SM::B_BYTES % (16 * kConvThreads) == 0, "a whole number of 16-byte pieces per thread");
          float4 v[kPieces];
#pragma unroll
          for (int i = 0; i < kPieces; ++i) v[i] = rawb[threadIdx.x + i * kConvThreads];
#pragma unroll
          for (int i = 0; i < kPieces; ++i)
            lob[threadIdx.x + i * kConvThreads] =
                make_float4(tf32_lo(v[i].x), tf32_lo(v[i].y), tf32_lo(v[i].z), tf32_lo(v[i].w));
          fence_async_smem();  // make the generic-proxy writes visible to the tensor pipe
        }
        tmem_wait_st();
        tc_fence_before();
        // (test hook: one lost arrival leaves the MMA warp waiting until its time limit, see tc_debug_lose_arrive)
        if (!(wk.lose_arrive && it == 0 && threadIdx.x == 0 && blockIdx.x == 0)) {
          if constexpr (PAIR) mbar_arrive_rank(bar_conv(s), 0);   // the leader's MMA warp waits for both CTAs
          else mbar_arrive(bar_conv(s));
        }
      }
    }
  } else if (warp > kMmaWarp) {
    // ------------------------------------------------------------ B's lo parts (BWARPS kernels)
    // Two warps of their own: on the A converters' path this work lengthens the chain (wait for the stage, load,
    // split, store, fence, arrive) that every k-block of the MMA stream waits for.  Measured: forward product
    // 0.437 -> 0.396 ms.
    uint32_t it = 0;
    bool ok = true;
    const int t = threadIdx.x - (kMmaWarp + 1) * 32;   // 0 .. 63
    for (long w = w_first; BWARPS && w < total && ok; w += w_step) {
      int mt, nt, sp, kbeg, nkb;
      decode(w, mt, nt, sp, kbeg, nkb);
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1u;
        if (!mbar_wait_warp(bar_full(s), ph, abort_flag, status, kWaitFull)) { ok = false; break; }
        // lo parts beside the raw tile in shared memory; every load is issued before the first store
        constexpr int kBThreads = kBConvWarps * 32;
        const float4 *rawb = reinterpret_cast<const float4 *>(smem + s * SM::STAGE_BYTES + SM::A_BYTES);
        float4 *lob = reinterpret_cast<float4 *>(smem + s * SM::STAGE_BYTES + SM::RAW_BYTES);
        constexpr int kPieces = SM::B_BYTES / 16 / kBThreads;
        static_assert(SM::B_BYTES % (16 * kBThreads) == 0, "a whole number of 16-byte pieces per thread");
        float4 v[kPieces];
#pragma unroll
        for (int i = 0; i < kPieces; ++i) v[i] = rawb[t + i * kBThreads];
#pragma unroll
        for (int i = 0; i < kPieces; ++i)
          lob[t + i * kBThreads] = make_float4(tf32_lo(v[i].x), tf32_lo(v[i].y), tf32_lo(v[i].z), tf32_lo(v[i].w));
        fence_async_smem();  // make the generic-proxy writes visible to the tensor pipe
        if constexpr (PAIR) mbar_arrive_rank(bar_conv(s), 0);
        else mbar_arrive(bar_conv(s));
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Thread (lane) owns four tile rows (16*hh + lane/4 + 8*rr) of its warp's TMEM lane
    // quarter and, per 32-column group, the column pairs 8*rep + 2*(lane%4) + {0,1}:
    // four lanes cover 32 contiguous bytes of a row, so global accesses fill whole sectors.
    const int q = warp & 3;                      // TMEM lane quarter this warp may read
    const int ch = (warp - kConvWarps) >> 2;     // which half of the tile's columns
    const int lr = lane >> 2, lc = (lane & 3) * 2;
    constexpr int NG = BN / 64;                  // 32-column groups per warp
    uint32_t chain = 0;
    bool ok = true;
    const int ew = warp - kConvWarps;            // epilogue warp index
    uint32_t swz[4];                             // byte offset of column pair `rep` inside a swizzled 128-byte row
#pragma unroll
    for (int rep = 0; rep < 4; ++rep) swz[rep] = ((uint32_t)((2 * rep + (lc >> 2)) ^ lr) << 4) + (uint32_t)(lc & 3) * 4u;
    // Raw product leaving by TMA: this warp's 32 x 32 block of column group g (lo: tile rows lr, lr + 8; hi:
    // 16 + lr, 24 + lr; four column pairs each) goes to a staging buffer in the swizzled layout of the
    // tensor map and one lane sends it.  Blocks past the edge of the output are clipped by the TMA unit.
    uint32_t stores = 0;
    auto store_block = [&](const float (&lo)[16], const float (&hi)[16], int mt, int nt, int g) {
      const uint32_t sb = stores & 1u;
      if (lane == 0) bulk_wait_read_1();   // the store that used this buffer two blocks ago has read it
      __syncwarp();
      uint8_t *sl = smem + SM::SLAB_OFFSET + (ew * 2 + sb) * kSlabBytes + lr * 128;
#pragma unroll
      for (int rr = 0; rr < 2; ++rr)
#pragma unroll
        for (int rep = 0; rep < 4; ++rep) {
          *reinterpret_cast<float2 *>(sl + (8 * rr) * 128 + swz[rep]) = make_float2(lo[rep * 4 + rr * 2], lo[rep * 4 + rr * 2 + 1]);
          *reinterpret_cast<float2 *>(sl + (16 + 8 * rr) * 128 + swz[rep]) =
              make_float2(hi[rep * 4 + rr * 2], hi[rep * 4 + rr * 2 + 1]);
        }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmC, base + SM::SLAB_OFFSET + (ew * 2 + sb) * kSlabBytes, nt * BN + ch * (BN / 2) + g * 32,
                     mt * 128 + 32 * q);
        bulk_commit();
      }
      ++stores;
    };
    for (long w = w_first; w < total && ok; w += w_step) {
      int mt, nt, sp, kbeg, nkb;
      decode(w, mt, nt, sp, kbeg, nkb);
      const long m_base = (long)mt * 128 + 32 * q;   // first tile row of this warp's lane quarter
      const long n_base = (long)nt * BN + ch * (BN / 2);
      bool rv[4];
      long grow[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long m = m_base + 16 * (j >> 1) + lr + 8 * (j & 1);
        rv[j] = m < ep.rows;
        grow[j] = m;
      }
      if constexpr (CHAIN > 0) {
        // ---- running sums in registers, one TMEM chain at a time (forward product)
        float sum[NG][2][16];
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
#pragma unroll
            for (int k = 0; k < 16; ++k) sum[g][hh][k] = 0.f;
        const int nchains = (nkb + CHAIN - 1) / CHAIN;
        for (int c = 0; c < nchains && ok; ++c, ++chain) {
          const uint32_t buf = chain & 1u, aph = (chain >> 1) & 1u;
          if (!mbar_wait_warp(bar_acc_full(buf), aph, abort_flag, status, kWaitAccFull)) { ok = false; break; }
          __syncwarp();
          tc_fence_after();
#pragma unroll
          for (int g = 0; g < NG; ++g) {
            float a0[16], a1[16];
            const uint32_t t0 = tmem_base + buf * BN + ch * (BN / 2) + g * 32 + ((uint32_t)(32 * q) << 16);
            tmem_ld_pair(t0, t0 + (16u << 16), a0, a1);
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              sum[g][0][k] += a0[k];
              sum[g][1][k] += a1[k];
            }
          }
          tc_fence_before();
          if constexpr (PAIR) mbar_arrive_rank(bar_acc_empty(buf), 0);
          else mbar_arrive(bar_acc_empty(buf));
        }
        if (ok && !A_KMAJOR && ep.tma_store) {
#pragma unroll
          for (int g = 0; g < NG; ++g) store_block(sum[g][0], sum[g][1], mt, nt, g);
        } else if (ok) {
#pragma unroll
          for (int g = 0; g < NG; ++g)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (!rv[j]) continue;
              float *orow = ep.out + ((long)sp * ep.rows + grow[j]) * ep.ld;
#pragma unroll
              for (int rep = 0; rep < 4; ++rep) {
                const long n = n_base + g * 32 + rep * 8 + lc;
                if (n < ep.cols)
                  __stcs(reinterpret_cast<float2 *>(orow + n),
                         make_float2(sum[g][j >> 1][rep * 4 + (j & 1) * 2], sum[g][j >> 1][rep * 4 + (j & 1) * 2 + 1]));
              }
            }
        }
      } else {
        const uint32_t buf = chain & 1u, aph = (chain >> 1) & 1u;
        if (!mbar_wait_warp(bar_acc_full(buf), aph, abort_flag, status, kWaitAccFull)) { ok = false; break; }
        if (threadIdx.x == kConvWarps * 32) TC_TRACE(chain, 3);
        __syncwarp();
        tc_fence_after();
        // this warp's accumulator block: TMEM lanes 32q.., columns of its half tile
        const uint32_t tacc = tmem_base + buf * BN + ch * (BN / 2) + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
        for (int g = 0; g < NG; ++g) {
          float a0[16], a1[16];
          const uint32_t t0 = tacc + g * 32;
          __syncwarp();  // tcgen05.ld is warp-collective
          tmem_ld_pair(t0, t0 + (16u << 16), a0, a1);
          if (!A_KMAJOR && ep.tma_store) {
            store_block(a0, a1, mt, nt, g);
            continue;
          }
          const long n0 = n_base + g * 32 + lc;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (!rv[j]) continue;
            const float *acc = (j >> 1) ? a1 : a0;
            float *orow = ep.out + ((long)sp * ep.rows + grow[j]) * ep.ld;
#pragma unroll
            for (int rep = 0; rep < 4; ++rep)
              if (n0 + rep * 8 < ep.cols)   // cols is even: n+1 is in range too
                __stcs(reinterpret_cast<float2 *>(orow + n0 + rep * 8),
                       make_float2(acc[rep * 4 + (j & 1) * 2], acc[rep * 4 + (j & 1) * 2 + 1]));
          }
        }
        if (threadIdx.x == kConvWarps * 32) TC_TRACE(chain, 4);
        tc_fence_before();
        // the accumulator buffer may be overwritten (PAIR: the leader's MMA warp waits for both CTAs' epilogues)
        if constexpr (PAIR) mbar_arrive_rank(bar_acc_empty(buf), 0);
        else mbar_arrive(bar_acc_empty(buf));
        ++chain;
      }
    }
  }

  // stores this thread sent by TMA must have left shared memory (and landed) before the CTA retires
  if (!A_KMAJOR && warp >= kConvWarps && warp < kTmaWarp && lane == 0) bulk_wait_all();
  // ------------------------------------------------------------ tear-down
  __syncwarp();
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // neither CTA retires while the other may still signal it or read its operands
  else __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, SM::TMEM_COLS);
    else tmem_dealloc(tmem_base, SM::TMEM_COLS);
  }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

std::mutex g_mutex;
EncodeTiledFn g_encode = nullptr;
int g_available = -1;           // -1 unknown, 0 no, 1 yes
int *g_status[64] = {nullptr};  // per-device status word, in mapped host memory: read without a copy
int g_sm_count_tc[64] = {0};
std::atomic<int> g_reserved_sms{-1};   // -1: not set yet (the environment decides on first use)
std::atomic<long long> g_wait_limit{kWaitLimitCycles};
std::atomic<int> g_lose_arrive{0};     // launches that still have to lose one arrival (test hook)
std::atomic<unsigned long long> g_pair_launches{0};
long long wait_limit_now() { return g_wait_limit.load(); }
int take_lose_arrive() {
  int n = g_lose_arrive.load();
  while (n > 0 && !g_lose_arrive.compare_exchange_weak(n, n - 1)) {
  }
  return n > 0 ? 1 : 0;
}

int current_device() {
  int dev = 0;
  cudaGetDevice(&dev);
  return dev < 0 || dev >= 64 ? 0 : dev;
}

bool init_once() {
  static std::atomic<bool> ready{false};   // the steady state takes no lock
  if (ready.load(std::memory_order_acquire)) return true;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (g_available < 0) {
    g_available = 0;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess && fn != nullptr) {
      g_encode = reinterpret_cast<EncodeTiledFn>(fn);
      g_available = 1;
    } else {
      (void)cudaGetLastError();
    }
  }
  ready.store(g_available == 1, std::memory_order_release);
  return g_available == 1;
}

int *status_word() {
  const int dev = current_device();
  static std::atomic<int *> known[64];
  if (int *p = known[dev].load(std::memory_order_acquire)) return p;
  std::lock_guard<std::mutex> lock(g_mutex);
  if (g_status[dev] == nullptr) {
    int *p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess) return nullptr;
    *p = 0;
    g_status[dev] = p;
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    g_sm_count_tc[dev] = n > 0 ? n : 148;
  }
  known[dev].store(g_status[dev], std::memory_order_release);
  return g_status[dev];
}

// Encoded tensor maps are kept per host thread, keyed by everything that goes into them: a layer's step
// re-encodes the same handful of maps (same buffers, same shapes) every call, and the driver's encoder
// costs about a microsecond each, which is a tenth of the step of a small layer.
struct MapKey {
  const void *base;
  long inner, outer, pitch;
  int box_a, box_b, kind;
  bool operator==(const MapKey &o) const {
    return base == o.base && inner == o.inner && outer == o.outer && pitch == o.pitch && box_a == o.box_a && box_b == o.box_b && kind == o.kind;
  }
};
struct MapCache {
  static constexpr int kSlots = 128;
  MapKey key[kSlots];
  CUtensorMap map[kSlots];
  bool used[kSlots] = {false};
  static unsigned slot(const MapKey &k) {
    uint64_t h = reinterpret_cast<uintptr_t>(k.base) * 0x9E3779B97F4A7C15ull;
    h ^= (uint64_t)k.inner * 0xC2B2AE3D27D4EB4Full + (uint64_t)(k.outer ^ k.pitch << 20) * 0x165667B19E3779F9ull +
         (uint64_t)(k.box_a * 131 + k.box_b * 17 + k.kind);
    return (unsigned)(h >> 40) % kSlots;
  }
  bool find(const MapKey &k, CUtensorMap *out) const {
    const unsigned s = slot(k);
    if (!used[s] || !(key[s] == k)) return false;
    *out = map[s];
    return true;
  }
  void put(const MapKey &k, const CUtensorMap &m) {
    const unsigned s = slot(k);
    key[s] = k;
    map[s] = m;
    used[s] = true;
  }
};
thread_local MapCache g_map_cache;

bool make_map_uncached(CUtensorMap *map, const MapKey &k) {
  cuuint64_t dims[2] = {(cuuint64_t)k.inner, (cuuint64_t)k.outer};
  cuuint64_t strides[1] = {(cuuint64_t)k.pitch * sizeof(float)};
  cuuint32_t box[2] = {(cuuint32_t)k.box_a, (cuuint32_t)k.box_b};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(k.base), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              k.kind == kMapMnMajor ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B
                              : k.kind == kMapRows64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                     : CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// 3-D view {32, rows, cols/32} of a row-major [rows, cols] float32 matrix (element (i, r, c) = m[r][32c + i]);
// a box {32, box_rows, box_chunks} lands in shared memory as [chunk][row][32], the MN-major stage layout.
bool make_map_chunks_uncached(CUtensorMap *map, const MapKey &k) {
  if (k.inner < 32) return false;
  cuuint64_t dims[3] = {32, (cuuint64_t)k.outer, (cuuint64_t)(k.inner / 32)};
  cuuint64_t strides[2] = {(cuuint64_t)k.pitch * sizeof(float), 128};
  cuuint32_t box[3] = {32, (cuuint32_t)k.box_a, (cuuint32_t)k.box_b};
  cuuint32_t estr[3] = {1, 1, 1};
  return g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void *>(k.base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2-D float32 tensor map over a row-major [outer, inner] matrix with rows `pitch` elements apart, zero fill.
bool make_map(CUtensorMap *map, const float *base, long inner, long outer, long pitch, int box_inner, int box_outer, int layout) {
  const MapKey k{base, inner, outer, pitch, box_inner, box_outer, layout};
  if (g_map_cache.find(k, map)) return true;
  if (!make_map_uncached(map, k)) return false;
  g_map_cache.put(k, *map);
  return true;
}
bool make_map(CUtensorMap *map, const float *base, long inner, long outer, int box_inner, int box_outer, int layout) {
  return make_map(map, base, inner, outer, inner, box_inner, box_outer, layout);
}
bool make_map_chunks(CUtensorMap *map, const float *base, long cols, long rows, long pitch, int box_rows, int box_chunks) {
  const MapKey k{base, cols, rows, pitch, box_rows, box_chunks, -1};
  if (g_map_cache.find(k, map)) return true;
  if (!make_map_chunks_uncached(map, k)) return false;
  g_map_cache.put(k, *map);
  return true;
}
bool make_map_chunks(CUtensorMap *map, const float *base, long cols, long rows, int box_rows, int box_chunks) {
  return make_map_chunks(map, base, cols, rows, cols, box_rows, box_chunks);
}

// Column tiles of width bn whose every 32-column group lies inside the matrix.
int full_chunk_tiles(long cols, int bn) { return (int)(((cols / 32) * 32) / bn); }

struct TcMaps {
  CUtensorMap a, b, a3, b3, c;
  CUtensorMap alo, blo, a3lo, b3lo;   // the operands' low-part planes (pre-split kernels)
};

template <bool A_KMAJOR, int BN, int BK, int STAGES, int CHAIN, bool PRESPLIT = false>
cudaError_t launch_tc(const TcMaps &tm, const TcWork &wk, const TcEpilogue &ep, cudaStream_t st,
                      bool leave_reserved_sms = false) {
  using SM = TcSmem<BN, BK, STAGES, !A_KMAJOR, PRESPLIT>;
  int *status = status_word();
  if (status == nullptr) return cudaErrorMemoryAllocation;
  auto kernel = tc_contraction_kernel<A_KMAJOR, BN, BK, STAGES, CHAIN, PRESPLIT>;
  static std::atomic<bool> configured[64];   // per device; setting the attribute twice is harmless
  const int dev = current_device();
  if (!configured[dev].load()) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL);
    if (e != cudaSuccess) return e;
    configured[dev].store(true);
  }
  const long total = (long)wk.m_tiles * wk.n_tiles * wk.splits;
  if (total <= 0) return cudaSuccess;
  int sms = g_sm_count_tc[dev] - (leave_reserved_sms ? tc_get_reserved_sms() : 0);
  if (sms < 1) sms = 1;
  const unsigned grid = (unsigned)(total < sms ? total : sms);
  return launch_next(kernel, grid, kThreads, SM::TOTAL, st, tm.a, tm.b, tm.a3, tm.b3, tm.c, tm.alo, tm.blo, tm.a3lo, tm.b3lo,
                     wk, ep, status);
}

// SBB_TC_PAIR=0 keeps one CTA per tile, in the forward product and in the trace update (read once).
bool pairs_enabled() {
  static const bool on = [] {
    const char *e = getenv("SBB_TC_PAIR");
    return !(e != nullptr && e[0] == '0');
  }();
  return on;
}

// The CTA-pair form of a kernel: clusters of two CTAs, one 256 x BN tile per pair.
template <bool A_KMAJOR, int BN, int BK, int STAGES, int CHAIN>
cudaError_t launch_tc_pair(const TcMaps &tm, const TcWork &wk, const TcEpilogue &ep, cudaStream_t st) {
  using SM = TcSmem<BN, BK, STAGES, !A_KMAJOR, false, true>;
  int *status = status_word();
  if (status == nullptr) return cudaErrorMemoryAllocation;
  auto kernel = tc_contraction_kernel<A_KMAJOR, BN, BK, STAGES, CHAIN, false, true>;
  static std::atomic<bool> configured[64];
  const int dev = current_device();
  if (!configured[dev].load()) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL);
    if (e != cudaSuccess) return e;
    configured[dev].store(true);
  }
  const long pairs = (long)((wk.m_tiles + 1) / 2) * wk.n_tiles * wk.splits;
  if (pairs <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = SM::TOTAL;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // as many pairs as can be resident at once (one CTA per SM; pairs must share a GPC's SMs)
  static int max_clusters[64] = {0};
  if (max_clusters[dev] == 0) {
    cfg.gridDim = dim3((unsigned)(g_sm_count_tc[dev] / 2 * 2), 1, 1);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) n = g_sm_count_tc[dev] / 2;
    max_clusters[dev] = n;
  }
  long clusters = max_clusters[dev] < g_sm_count_tc[dev] / 2 ? max_clusters[dev] : g_sm_count_tc[dev] / 2;
  if (clusters > pairs) clusters = pairs;
  cfg.gridDim = dim3((unsigned)(2 * clusters), 1, 1);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // as launch_next
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tm.a, tm.b, tm.a3, tm.b3, tm.c, tm.alo, tm.blo, tm.a3lo, tm.b3lo, wk,
                                           ep, status);
  if (e == cudaSuccess) tc_count_pair_launch();
  return e;
}

}  // namespace

void tc_count_pair_launch() { g_pair_launches += 1; }
unsigned long long tc_pair_launches() { return g_pair_launches.load(); }

bool tc_host(TcHost *out) {
  out->status = status_word();
  out->sms = g_sm_count_tc[current_device()];
  out->wait_limit = wait_limit_now();
  out->lose_arrive = out->status != nullptr ? take_lose_arrive() : 0;
  out->pairs = pairs_enabled();
  return out->status != nullptr && init_once();
}
bool tc_map_2d(void *map, const float *base, long inner, long outer, long pitch, int box_inner, int box_outer, int layout) {
  return make_map(static_cast<CUtensorMap *>(map), base, inner, outer, pitch, box_inner, box_outer, layout);
}
bool tc_map_chunks(void *map, const float *base, long cols, long rows, long pitch, int box_rows, int box_chunks) {
  return make_map_chunks(static_cast<CUtensorMap *>(map), base, cols, rows, pitch, box_rows, box_chunks);
}

// Launch counter shared with the general-shape kernels (defined in sbb_kernels.cu).
void count_launches(int n);

bool tc_available() {
  if (!init_once()) return false;
  int dev = 0, major = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  static std::atomic<int> known[64];   // compute capability of the devices asked about
  if (dev >= 0 && dev < 64 && (major = known[dev].load()) != 0) return major == 10;
  if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) return false;
  if (dev >= 0 && dev < 64) known[dev].store(major);
  return major == 10;
}

bool tc_shape_ok(const void *x, const void *y_or_w, long N, long M) {
  return N % 4 == 0 && M % 4 == 0 && N >= 4 && M >= 4 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(y_or_w) & 15u) == 0 && N < 2147483136L && M < 2147483136L;   // (tile coordinates in 32 bits)
}

namespace {
// A stage of a pair is 32 KB and its MMAs take 0.39 us: six of them cover the 2 us from asking for a k-block until its place is
// free again (fetch, split, multiply), four did not; tensor memory has room for the split rows of four.  Forward pass with four
// and with six: 55296 -> 30 x 100 at batch 256 356 and 338 us, 1568 -> 100 x 300 at 1024 418 and 386.
constexpr int kFwdBN = 128, kFwdBK = 32, kFwdStages = 4, kFwdPairStages = 6;
constexpr int kFwdPrefetch = 0;  // k-blocks of W requested into L2 ahead of the shared-memory pipeline (measured: no gain at 4-16)
constexpr int kFwdChain = 4;  // 4 k-blocks of 32 = 128 k-values (48 MMAs) per tensor-memory accumulation chain
constexpr int kTrBN = 192, kTrBK = 16, kTrStages = 4;
// k-blocks per accumulation chain of the batch contractions: 16 x 16 = 256 samples (96 MMAs), after which the
// epilogue takes the partial sum over in float32.  Measured on B200: the tensor-memory accumulate truncates,
// so a chain's sum is low by about 1e-8 x (samples in the chain) relative; 256 keeps that below 4e-6.
constexpr int kTrChainKb = 16;
constexpr int kLongBN = 128, kLongStages = 5;   // tiles of the row-block product when the batch spans several chains

// k-blocks per split and the number of (non-empty) splits for the forward product: the split count
// that minimises (waves of CTAs) x (k-blocks per unit), plus the cost of writing and re-reading
// one more partial result.  A unit count just above a multiple of the SM count would otherwise
// run a nearly empty last wave (192 units on 148 SMs take as long as 296).
void forward_split_plan(long B, long N, long M, int &splits, int &k_per_split) {
  // (a step asks three times for the same shape, and trying every split count costs microseconds)
  struct Plan {
    long B, N, M;
    int splits, k_per_split, dev;
  };
  static thread_local Plan last{-1, -1, -1, 0, 0, -1};
  if (last.B == B && last.N == N && last.M == M && last.dev == current_device()) {
    splits = last.splits;
    k_per_split = last.k_per_split;
    return;
  }
  const long tiles = ((B + 127) / 128) * ((M + kFwdBN - 1) / kFwdBN);
  const long kblocks = (N + kFwdBK - 1) / kFwdBK;
  const int dev = current_device();
  const long sms = g_sm_count_tc[dev] > 0 ? g_sm_count_tc[dev] : 148;
  long max_splits = kblocks / 8 > 0 ? kblocks / 8 : 1;   // at least 8 k-blocks per split
  if (max_splits > 64) max_splits = 64;
  // one partial result costs B*M*8 bytes of traffic; in units of one k-block of one CTA (about 0.8 us
  // at 6.5 TB/s, spread over the SMs)
  const double partial_cost = (double)B * (double)M * 8.0 / 6.5e12 / 0.8e-6;
  double best_cost = 0.0;
  long best_per = kblocks;
  for (long want = 1; want <= max_splits; ++want) {
    const long per = (kblocks + want - 1) / want;
    const long actual = (kblocks + per - 1) / per;
    const long waves = (tiles * actual + sms - 1) / sms;
    const double cost = (double)waves * (double)per + (double)actual * partial_cost;
    if (want == 1 || cost < best_cost) {
      best_cost = cost;
      best_per = per;
    }
  }
  splits = (int)((kblocks + best_per - 1) / best_per);
  k_per_split = (int)best_per * kFwdBK;
  last = Plan{B, N, M, splits, k_per_split, dev};
}
}  // namespace

int forward_splits_tc(long B, long N, long M) {
  status_word();  // fills the SM count
  int s, k;
  forward_split_plan(B, N, M, s, k);
  return s;
}

cudaError_t launch_forward_product_tc(const float *x, const float *w, float *partial, long B, long N, long M,
                                      int splits, cudaStream_t st) {
  if (!tc_available() || !tc_shape_ok(x, w, N, M) || (reinterpret_cast<uintptr_t>(partial) & 7u)) return cudaErrorNotSupported;
  int plan_splits, k_per_split;
  status_word();
  forward_split_plan(B, N, M, plan_splits, k_per_split);
  if (plan_splits != splits) return cudaErrorInvalidValue;
  TcMaps tm;
  if (!make_map(&tm.a, x, N, B, 32, 128, kMapRows) || !make_map(&tm.b, w, M, N, 32, kFwdBK, kMapMnMajor)) return cudaErrorInvalidValue;
  tm.a3 = tm.a;
  tm.c = tm.a;
  // CTA pairs when the row tiles pair up: the two CTAs that need the same tile of W each fetch half of it
  const bool pair = pairs_enabled() && ((B + 127) / 128) % 2 == 0;
  const bool b3 = make_map_chunks(&tm.b3, w, M, N, kFwdBK, (pair ? kFwdBN / 2 : kFwdBN) / 32);
  if (!b3) tm.b3 = tm.b;
  tm.alo = tm.blo = tm.a3lo = tm.b3lo = tm.a;
  TcWork wk{(int)((B + 127) / 128), (int)((M + kFwdBN - 1) / kFwdBN), splits, (int)N, k_per_split, 1, 0, 0,
            b3 ? full_chunk_tiles(M, kFwdBN) : 0, kFwdPrefetch, wait_limit_now(), take_lose_arrive()};
#ifdef SBB_TC_TRACE
  if (const char *e = getenv("SBB_FWD_PREFETCH")) wk.b_prefetch = atoi(e);   // timeline builds may vary the distance
#endif
  TcEpilogue ep{};
  ep.out = partial;
  ep.rows = B;
  ep.cols = M;
  ep.ld = M;
  cudaError_t e = pair ? launch_tc_pair<true, kFwdBN, kFwdBK, kFwdPairStages, kFwdChain>(tm, wk, ep, st)
                       : launch_tc<true, kFwdBN, kFwdBK, kFwdStages, kFwdChain>(tm, wk, ep, st);
  if (e == cudaSuccess) count_launches(1);
  return e;
}

namespace {
// Tensor maps of the two MN-major operands x[B, N] and y[B, M] of a batch contraction with `bn`-column tiles, and
// (pre != 0) of their low-part planes.  a3 / b3 report whether the one-box 3-D forms exist.
bool batch_operand_maps(TcMaps &tm, const float *x, const float *y, const float *x_lo, const float *y_lo, bool pre,
                        long B, long N, long M, int bn, bool &a3, bool &b3) {
  if (!make_map(&tm.a, x, N, B, 32, kTrBK, kMapMnMajor) || !make_map(&tm.b, y, M, B, 32, kTrBK, kMapMnMajor)) return false;
  a3 = N % 32 == 0 && make_map_chunks(&tm.a3, x, N, B, kTrBK, 4);
  if (!a3) tm.a3 = tm.a;
  b3 = make_map_chunks(&tm.b3, y, M, B, kTrBK, bn / 32);
  if (!b3) tm.b3 = tm.b;
  tm.alo = tm.a;
  tm.blo = tm.b;
  tm.a3lo = tm.a3;
  tm.b3lo = tm.b3;
  if (pre) {
    if (!make_map(&tm.alo, x_lo, N, B, 32, kTrBK, kMapMnMajor) || !make_map(&tm.blo, y_lo, M, B, 32, kTrBK, kMapMnMajor)) return false;
    if (a3 && !make_map_chunks(&tm.a3lo, x_lo, N, B, kTrBK, 4)) return false;
    if (b3 && !make_map_chunks(&tm.b3lo, y_lo, M, B, kTrBK, bn / 32)) return false;
  }
  return true;
}
bool lo_planes_usable(const float *x_lo, const float *y_lo) {
  return x_lo != nullptr && y_lo != nullptr && (reinterpret_cast<uintptr_t>(x_lo) & 15u) == 0 &&
         (reinterpret_cast<uintptr_t>(y_lo) & 15u) == 0;
}
}  // namespace

cudaError_t launch_outer_product_tc(const float *x, const float *y, long B, long N, long M, float *delta,
                                    long row_begin, long row_end, cudaStream_t st, const float *x_lo,
                                    const float *y_lo) {
  if (!tc_available() || !tc_shape_ok(x, y, N, M) || row_begin % 128 != 0 ||
      (reinterpret_cast<uintptr_t>(delta) & 7u))
    return cudaErrorNotSupported;
  if (row_end <= row_begin) return cudaSuccess;
  TcMaps tm;
  const bool pre = lo_planes_usable(x_lo, y_lo);
  const bool longb = B > (long)kTrChainKb * kTrBK;
  bool a3 = false, b3 = false;
  if (!batch_operand_maps(tm, x, y, x_lo, y_lo, pre, B, N, M, longb ? kLongBN : kTrBN, a3, b3)) return cudaErrorInvalidValue;
  tm.c = tm.a;
  const long rows = row_end - row_begin;
  const int kper = (int)((B + kTrBK - 1) / kTrBK) * kTrBK;
  if (longb) {
    // More than one accumulation chain: 128-column tiles whose running sums stay in the epilogue warps'
    // registers (as in the forward product), so no partial sum travels through memory.
    const bool b3n = b3;
    TcWork wk{(int)((rows + 127) / 128), (int)((M + kLongBN - 1) / kLongBN), 1, (int)B, kper, M > N ? 1 : 0,
              (int)row_begin, a3 ? 1 : 0, b3n ? full_chunk_tiles(M, kLongBN) : 0, 0, wait_limit_now(), 0};
    TcEpilogue ep{};
    ep.out = delta + row_begin * M;
    ep.rows = rows;
    ep.cols = M;
    ep.ld = M;
    ep.tma_store = (reinterpret_cast<uintptr_t>(ep.out) & 15u) == 0 && make_map(&tm.c, ep.out, M, rows, 32, 32, kMapRows);
    if (!ep.tma_store) tm.c = tm.a;
    cudaError_t e = pre ? launch_tc<false, kLongBN, kTrBK, kLongStages, kTrChainKb, true>(tm, wk, ep, st, true)
                        : launch_tc<false, kLongBN, kTrBK, kLongStages, kTrChainKb>(tm, wk, ep, st, true);
    if (e == cudaSuccess) count_launches(1);
    return e;
  }
  // tiles are walked so that the larger operand is the one re-used by consecutive tiles: column tiles
  // fastest when x (B x N) is the larger, row tiles fastest when y (B x M) is
  TcWork wk{(int)((rows + 127) / 128), (int)((M + kTrBN - 1) / kTrBN), 1, (int)B, kper, M > N ? 1 : 0, (int)row_begin,
            a3 ? 1 : 0, b3 ? full_chunk_tiles(M, kTrBN) : 0, 0, wait_limit_now(), take_lose_arrive()};
  TcEpilogue ep{};
  ep.out = delta + row_begin * M;
  ep.rows = rows;
  ep.cols = M;
  ep.ld = M;
  ep.tma_store = (reinterpret_cast<uintptr_t>(ep.out) & 15u) == 0 && make_map(&tm.c, ep.out, M, rows, 32, 32, kMapRows);
  if (!ep.tma_store) tm.c = tm.a;
  // the one contraction that runs beside a collective (the reduction of the previous row block)
  cudaError_t e = pre ? launch_tc<false, kTrBN, kTrBK, kTrStages, 0, true>(tm, wk, ep, st, true)
                      : launch_tc<false, kTrBN, kTrBK, kTrStages, 0>(tm, wk, ep, st, true);
  if (e == cudaSuccess) count_launches(1);
  return e;
}

// Parts the batch of a trace step is cut into (1: the fused kernel), as trace_splits: both kernels take about 0.42 us per
// k-block of 16 samples, in rounds of 74 pairs of SMs with 256 x 192 outputs or of 148 SMs with 128 x 128.  Measured (column
// vectors included, fused -> best of 2 to 48 parts -> the rule's): 88 x 528 at batch 5851 165 -> 31 -> 31 us, 256 x 256 at 2048 63 ->
// 19 -> 21, 512 x 1024 at 4096 116 -> 46 -> 46, 664 x 16 at 5453 153 -> 30 -> 30, 128 x 96 at 512 22 -> 13 -> 13; 2048 x 1024 at 2048 (48
// pairs) 64 -> 74 with two parts, 20000 x 64 at 1024 (79 pairs) 69 -> 66.
namespace {
// k-blocks of a part.  Parts of more than 1024 samples in all are whole accumulation chains, so that their sums are those of the
// fused kernel's chains to the bit; cut elsewhere, the chains' truncation differs from its by up to 4e-6 of the sum, of which a
// layer with a large taupdt and its own activations for outputs makes 1e-5 in two steps (1024 -> 128 at batch 8192).
long part_kblocks(long kblocks, long splits) {
  const long unit = kblocks > 64 ? kTrChainKb : 1, units = (kblocks + unit - 1) / unit;
  return (units + splits - 1) / splits * unit;
}
}  // namespace

int trace_splits_tc(long B, long N, long M) {
  const long kblocks = (B + kTrBK - 1) / kTrBK, pairs = ((N + 255) / 256) * ((M + kTrBN - 1) / kTrBN);
  const long tiles = ((N + 127) / 128) * ((M + kLongBN - 1) / kLongBN);
  if (kblocks < 16 || N > 4096) return 1;   // (many inputs: they keep the order of their sums, as few_plan's)
  status_word();   // fills the SM count
  const long sms = g_sm_count_tc[current_device()];
  auto ceil_div = [](long a, long b) { return (a + b - 1) / b; };
  int best = 1;
  double least = 0.85 * (double)(ceil_div(pairs, sms / 2 > 0 ? sms / 2 : 1) * kblocks) * 0.42;
  for (long s = 2; s <= 48 && kblocks / s >= 4; ++s) {
    if (s * N * M > (1l << 26)) break;
    const long per = part_kblocks(kblocks, s), parts = ceil_div(kblocks, per);
    const double c = (double)(ceil_div(tiles * parts, sms) * per) * 0.42 + 5.0 + (double)(parts * N * M) * 8.0 / 3e6;
    if (c < least) least = c, best = (int)s;
  }
  return (int)ceil_div(kblocks, part_kblocks(kblocks, best));   // no empty part
}

cudaError_t launch_split_product_tc(const float *x, const float *y, long B, long N, long M, int splits, float *partial,
                                    cudaStream_t st) {
  if (!tc_available() || !tc_shape_ok(x, y, N, M) || (reinterpret_cast<uintptr_t>(partial) & 7u)) return cudaErrorNotSupported;
  TcMaps tm;
  bool a3 = false, b3 = false;
  if (!batch_operand_maps(tm, x, y, nullptr, nullptr, false, B, N, M, kLongBN, a3, b3)) return cudaErrorInvalidValue;
  tm.c = tm.a;
  const long kblocks = (B + kTrBK - 1) / kTrBK;
  TcWork wk{(int)((N + 127) / 128), (int)((M + kLongBN - 1) / kLongBN), splits, (int)B, (int)part_kblocks(kblocks, splits) * kTrBK,
            M > N ? 1 : 0, 0, a3 ? 1 : 0, b3 ? full_chunk_tiles(M, kLongBN) : 0, 0, wait_limit_now(), take_lose_arrive()};
  TcEpilogue ep{};
  ep.out = partial;
  ep.rows = N;
  ep.cols = M;
  ep.ld = M;
  const cudaError_t e = launch_tc<false, kLongBN, kTrBK, kLongStages, kTrChainKb>(tm, wk, ep, st);
  if (e == cudaSuccess) count_launches(1);
  return e;
}

#ifdef SBB_TC_TRACE
extern "C" int sbb_tc_trace_read(unsigned long long *out) {
  cudaDeviceSynchronize();
  return (int)cudaMemcpyFromSymbol(out, g_tc_trace, sizeof(unsigned long long) * 64 * 16);
}
#endif

void tc_set_wait_limit(long long cycles) { g_wait_limit.store(cycles > 0 ? cycles : kWaitLimitCycles); }
long long tc_get_wait_limit() { return g_wait_limit.load(); }
void tc_debug_lose_arrive(int launches) { g_lose_arrive.store(launches > 0 ? launches : 0); }

void tc_set_reserved_sms(int sms) { g_reserved_sms.store(sms < 0 ? 0 : sms); }
int tc_get_reserved_sms() {
  int v = g_reserved_sms.load();
  if (v < 0) {
    const char *e = getenv("SBB_COMM_SMS");
    v = e ? atoi(e) : 0;
    if (v < 0) v = 0;
    g_reserved_sms.store(v);
  }
  return v;
}

static volatile int *status_if_any() {
  const int dev = current_device();
  std::lock_guard<std::mutex> lock(g_mutex);
  return g_status[dev];
}

// The status word without synchronising the device: meaningful for work the caller has already waited for.
cudaError_t tc_peek_status(int *status) {
  volatile int *p = status_if_any();
  *status = p ? *p : 0;
  return cudaSuccess;
}

cudaError_t tc_clear_status() {
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return e;
  if (volatile int *p = status_if_any()) *p = 0;
  return cudaSuccess;
}

cudaError_t tc_read_status(int *status) {
  *status = 0;
  const cudaError_t e = cudaDeviceSynchronize();
  return e != cudaSuccess ? e : tc_peek_status(status);
}

}  // namespace sbb
