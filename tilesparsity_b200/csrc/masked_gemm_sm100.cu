// Persistent grouped masked GEMM for tile-wise sparse weights (sm_100a: tcgen05 + TMEM + TMA).
//
// Replaces the reference's per-tile CUTLASS launches (one stream per column tile,
// StreamMaskedGEMM/perf/basic_nn.cu:378-445; kernel StreamMaskedGEMM/cutlass/gemm/gemm.h:45-61 with
// the masked A loads of cutlass/tile_iterator.h:786-816 and the masked stores of :1262-1292) by ONE
// launch over a work list.  Data layout is the reference's (column-major everywhere,
// basic_nn.cu:412-426):
//
//   At : activations, stored [K][lda] with the batch dimension M contiguous (column-major M x K);
//        the kernel only sees where each kept row starts (16-byte segment numbers in the block records),
//        which is how a convolution's shifted input planes stand in for an im2col matrix
//   Wp : packed weights, stored [rows][ldw] with K contiguous; tile t owns rows w_row0 .. +n_count,
//        entry (j, i) = W[kept_k[i], kept_n[j]]   (gen_masked_stream_weight, basic_nn.cu:757-769)
//   Ct : output, stored [N][ldc] with M contiguous; kept column j of a tile lands in row c_row(j)
//
// and the product computed per tile is  Ct[c_row(j), m] = alpha * sum_i Wp[j, i] * At[kept_k[i], m]
// (+ beta * Ct), accumulated in fp32.
//
// Mapping onto the tensor core: the tile's kept columns are the MMA's M dimension (128 TMEM lanes),
// the batch is its N dimension (MT = 128 or 256 columns per instruction), the kept rows are K.  The
// packed weights are the K-major A operand, fetched by TMA with 128-byte swizzle; the gathered
// activation rows are the MN-major B operand, fetched with 16-byte cp.async into the same swizzle
// pattern (one kept row is one contiguous 2*MT-byte global segment).
//
// Pipeline: four stages of 64 kept rows (six for 128-row units).  Two groups of four gather warps take turns on the
// blocks, a quarter of a block's rows each; all a warp needs to know about a block is one record (descriptor + 64
// resolved row numbers) that a bulk copy brought to shared memory kAhead blocks before its weights.  Each lane hands its
// copies to the stage's mbarrier with cp.async.mbarrier.arrive, so a stage is released to the MMA warp the moment its
// bytes have landed.  Accumulators live in TMEM, double buffered: the epilogue of one work unit overlaps the main loop
// of the next.  Eight epilogue warps (two per TMEM lane quarter; each half of them takes every other 64-column group of
// the unit) convert their 32 rows of a group to 16 bit in a 128-byte-swizzled 4 KiB staging buffer per warp.  When the
// tile's kept columns are consecutive rows of Ct (no column pruning) a warp's rows leave with one TMA store; otherwise
// with 16-byte coalesced stores through the kept-column list.
//
// Warp roles (576 threads): warp 0 = weights by TMA and block records, warp 1 = TMEM allocation + MMA issue, warps
// 2-9 = activation gather, warps 10-17 = epilogue.  18 warps leave 96 registers per thread, which the epilogue keeps to
// by holding 32 accumulators at a time.
#include <cstddef>
#include <type_traits>

#include "ts_common.cuh"
#include "ts_kernels.h"

namespace ts {

namespace {

constexpr int kNT = 128;                 // columns per tile (MMA M, TMEM lanes)
constexpr int kKB = 64;                  // kept rows per pipeline stage
constexpr int kWBytes = kNT * kKB * 2;   // 16 KiB of packed weights per stage
constexpr int kEpiWarps = 8;
constexpr uint32_t kASbo = 1024;         // bytes between 8-row K groups of the gathered operand
constexpr uint32_t kALbo = kKB * 128;    // bytes between its 64-column batch groups
constexpr uint32_t kWSbo = 1024;         // bytes between 8-row groups of the weight operand
constexpr int kMaxStages = 6;
// Gather warps: two groups of four that take turns on the K blocks; the warps of a group fill a block
// together, 16 rows each, which is one K step of the MMA.  The copies alone need only four warps to keep the
// L2-to-SM path full (470 cycles per 32 KiB on B200 with every SM copying, the same with 8 and 16), but a warp
// spends 600 cycles on a block whatever its width (record, stage wait, burst, hand-over): narrow units and
// short chains are bound by that (encoder layer at 32 rows 16.2 -> 15.6 us with the second group).
constexpr int kWarpsPerBlock = 4;
constexpr int kWarpGroups = 2;
constexpr int kGW = kWarpGroups * kWarpsPerBlock;
constexpr int kRowsPerWarp = kKB / kWarpsPerBlock;
constexpr int kGatherWarp0 = 2;          // warps 0 and 1: weights, MMA
constexpr int kEpiWarp0 = kGatherWarp0 + kGW;       // first epilogue warp
constexpr int kThreads = 32 * (kEpiWarp0 + kEpiWarps);
constexpr int kMetaInts = kBlockMetaInts;  // one block record: {m0, meta, 0, 0} + 64 row numbers
constexpr int kAhead = 4;                // records are requested this many blocks ahead of the weights
constexpr int kMaxRecs = kMaxStages + kAhead;
constexpr int kEpiWarpBytes = 4096;      // staging of one epilogue warp: 32 rows x 64 batch columns

struct Barriers {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t rec_full[kMaxRecs];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) int rec[kMaxRecs][kMetaInts];   // ring of block records, slot = block % Cfg::kRecs
};

// Compile-time shape of one kernel variant: MT batch rows per work unit.
template <int MT>
struct Cfg {
  // as many stages as fit beside the staging buffers in 227 KiB
  static constexpr int kStages = MT == 256 ? 4 : 6;
  static constexpr int kRecs = kStages + kAhead;
  static_assert(kStages <= kMaxStages && kRecs <= kMaxRecs, "stage count");
  static constexpr int kABytes = kKB * MT * 2;
  static constexpr int kStageBytes = kWBytes + kABytes;
  static constexpr int kEpiBytes = kEpiWarps * kEpiWarpBytes;
  static constexpr int kTmemCols = 2 * MT;          // two accumulators of MT fp32 columns
  static constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + static_cast<int>(sizeof(Barriers));
  static_assert(kSmemBytes <= 232448, "stages, staging and barriers exceed the shared memory of one CTA");
  static constexpr int kLanesPerRow = MT / 8;       // 16-byte chunks in one gathered row
  static constexpr int kRowsPerInstr = 32 / kLanesPerRow;
  static constexpr int kGroups = MT / 128;          // 64-column groups of a unit per epilogue warp
};

__device__ __forceinline__ WorkItem load_item(const WorkItem* p) {
  const int4* q = reinterpret_cast<const int4*>(p);
  union {
    int4 v[3];
    WorkItem w;
  } u;
  u.v[0] = ld_coherent(q);
  u.v[1] = ld_coherent(q + 1);
  u.v[2] = ld_coherent(q + 2);
  return u.w;
}

// Work item of CTA `cta` in round r, or an empty item past the end of the schedule.
__device__ __forceinline__ WorkItem fetch_item(const WorkItem* sched, int rounds, int grid, int cta,
                                               int r) {
  if (r < rounds) return load_item(sched + static_cast<size_t>(r) * grid + cta);
  WorkItem w;
  w.k_list = nullptr;
  w.n_list = nullptr;
  w.k_count = w.n_count = w.w_row0 = w.c_row0 = w.flags = w.m_begin = w.m_len = 0;
  w.tile = -1;
  return w;
}

// What the epilogue reads of a work item that the warp holds one word per lane.
constexpr int kItemWords = sizeof(WorkItem) / 4;
constexpr int kItemWordTile = 11;
static_assert(offsetof(WorkItem, n_list) == 8 && offsetof(WorkItem, k_count) == 16 && offsetof(WorkItem, n_count) == 20 &&
                  offsetof(WorkItem, c_row0) == 28 && offsetof(WorkItem, flags) == 32 && offsetof(WorkItem, m_begin) == 36 &&
                  offsetof(WorkItem, m_len) == 40 && offsetof(WorkItem, tile) == 44,
              "word numbers below");
struct EpiItem {
  const int* n_list;
  int n_count, c_row0, flags, m_begin, m_len;
  bool has_rows;
};
__device__ __forceinline__ EpiItem epi_item(int word) {
  constexpr uint32_t kAll = 0xffffffffu;
  EpiItem w;
  const uint32_t lo = __shfl_sync(kAll, word, 2), hi = __shfl_sync(kAll, word, 3);
  w.n_list = reinterpret_cast<const int*>((static_cast<uint64_t>(hi) << 32) | lo);
  w.has_rows = __shfl_sync(kAll, word, 4) > 0;
  w.n_count = __shfl_sync(kAll, word, 5);
  w.c_row0 = __shfl_sync(kAll, word, 7);
  w.flags = __shfl_sync(kAll, word, 8);
  w.m_begin = __shfl_sync(kAll, word, 9);
  w.m_len = __shfl_sync(kAll, word, 10);
  return w;
}

__device__ __forceinline__ int k_blocks(const WorkItem& w) { return (w.k_count + kKB - 1) / kKB; }

// Ct row (global column of W) of tile column j of a work item.
__device__ __forceinline__ long long c_row_of(const EpiItem& w, int j) {
  return w.c_row0 + (w.n_list ? ld_coherent(w.n_list + j) + ((w.flags & kItemRelative) ? j : 0) : j);
}

// gelu(x) = x * 0.5 * (1 + tanh(u)), u = sqrt(2/pi) * (x + 0.044715 x^3)  (Pruning/BERT/utils/modeling.py:264-277),
// for two values, written as x / (1 + exp(-2u)): the same function without the cancellation of 1 + tanh for
// negative u.  The special-function unit bounds it (16 results per cycle and SM), so the two share one
// reciprocal, 1 / (a b): three special-function instructions a pair.  exp's argument is cut at 2^60, so that the
// product stays finite, and the factor is 0 from there on (it is below 1e-18): a large negative x gives -0 and
// -inf a NaN, as the tanh form does.
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// -2u * log2(e) = x * (-2 sqrt(2/pi) log2(e)) * (1 + 0.044715 x^2)
__device__ __forceinline__ float gelu_exponent(float x) { return x * fmaf(x * x, -0.10294324f, -2.3022082f); }
constexpr float kGeluCut = 60.0f;
__device__ __forceinline__ void gelu2(float& x0, float& x1) {
  const float t0 = gelu_exponent(x0), t1 = gelu_exponent(x1);
  const float a = 1.0f + ex2_approx(fminf(t0, kGeluCut)), b = 1.0f + ex2_approx(fminf(t1, kGeluCut));
  const float r = rcp_approx(a * b);
  x0 *= t0 < kGeluCut ? r * b : 0.0f;
  x1 *= t1 < kGeluCut ? r * a : 0.0f;
}

__device__ __forceinline__ float apply_act(float x, int act) {
  if (act == kActRelu) return fmaxf(x, 0.0f);
  if (act == kActGelu) return x * rcp_approx(1.0f + ex2_approx(gelu_exponent(x)));
  return x;
}

// MODE selects what the epilogue can do: kModeLean act(alpha * acc + bias) through TMA tile stores only (the
// host picks it when beta == 0 and every scheduled tile keeps 128 consecutive columns), kModePlain every
// epilogue form and the list-driven stores, kModeSplit in addition the fp32 partial sums of split-K parts,
// kModePeers the copies for the other GPUs of a tile-sharded layer; kModeRows is kModeLean with a row-major
// output (batch row m of C contiguous over the columns of W), kModeNhwc the same for a convolution, without
// the scratch pixels of the padded space.  Code a call cannot reach stays out of
// the variant it runs: the hot loops share one instruction cache.
constexpr int kModePlain = 0, kModeSplit = 1, kModePeers = 2, kModeLean = 3, kModeRows = 4, kModeNhwc = 5;
constexpr int kFlagTmaStore = 1, kFlagWaitFirst = 2;
template <int DT, int MT, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
masked_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w,
                   const __grid_constant__ CUtensorMap tmap_c, int flags,
                   const WorkItem* __restrict__ sched, int rounds,
                   const int* __restrict__ block_meta, int blk_stride,
                   const uint16_t* __restrict__ At, long long lda,
                   uint16_t* __restrict__ Ct, long long ldc, int M, const __grid_constant__ EpilogueArgs ep,
                   int* __restrict__ status) {
  const float alpha = ep.alpha, beta = ep.beta;
  const int act = ep.act;
  const bool use_tma_store = (flags & kFlagTmaStore) != 0;
  // the schedule, the records or the weights come from the kernel before this one
  if (flags & kFlagWaitFirst) {
    grid_dependency_wait();
    fence_proxy_async();      // the records and the weights are fetched by bulk copies
  }
  constexpr bool SPLIT = MODE == kModeSplit, PEERS = MODE == kModePeers, NHWC = MODE == kModeNhwc, ROWS = MODE == kModeRows || NHWC;
  constexpr bool LEAN = MODE == kModeLean || ROWS;
  using C = Cfg<MT>;
  constexpr int kStages = C::kStages;
  // 1024-byte alignment: the swizzle pattern is a function of the shared-memory address bits.  The declaration asks for
  // it, so no byte is set aside to reach it.
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* epi = smem + kStages * C::kStageBytes;
  Barriers* bars = reinterpret_cast<Barriers*>(epi + C::kEpiBytes);
  volatile int* abort_flag = &bars->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int grid = gridDim.x;
  const int cta = blockIdx.x;

  // First work item: requested before the set-up below so its latency overlaps it.  The schedule is
  // static data.
  WorkItem w = fetch_item(sched, rounds, grid, cta, 0);
  const int* recs = block_meta + static_cast<size_t>(cta) * blk_stride * kMetaInts;

  if (warp == 0 && elect_one()) {
    for (int s = 0; s < kStages; ++s) {
      // weight TMA thread + the cp.async lanes of the gather warps
      mbar_init(smem_u32(&bars->full[s]), 1 + 32 * kWarpsPerBlock);
      mbar_init(smem_u32(&bars->empty[s]), 1);       // one tcgen05.commit
    }
    for (int s = 0; s < C::kRecs; ++s) mbar_init(smem_u32(&bars->rec_full[s]), 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bars->acc_full[a]), 1);
      mbar_init(smem_u32(&bars->acc_empty[a]), kEpiWarps);
    }
    bars->abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async_smem();
    // The records of the first blocks: their latency is the head of the chain record -> rows -> MMA.
    for (int i = 0; i < kAhead; ++i) {
      const uint32_t bar = smem_u32(&bars->rec_full[i]);
      mbar_arrive_expect_tx(bar, kMetaInts * 4);
      bulk_load(smem_u32(bars->rec[i]), recs + static_cast<size_t>(i) * kMetaInts, kMetaInts * 4, bar);
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&bars->tmem_base), C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = bars->tmem_base;
  // The next kernel in the stream may begin its own set-up now (it cannot touch this kernel's
  // outputs before its grid_dependency_wait, which returns only when this grid has completed).
  grid_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------------ weights and block records
    // Block `it`: its weights once its stage is free, and the record of block it + kAhead, whose ring slot
    // was last used by block it + kAhead - kRecs = it - kStages, consumed when that stage became free.
    if (elect_one()) {
      tma_prefetch_desc(&tmap_w);
      uint32_t it = 0;
      bool ok = true;
      for (int r = 0; ok && w.tile >= 0; ++r) {
        const WorkItem wn = fetch_item(sched, rounds, grid, cta, r + 1);
        const int nkb = k_blocks(w);
        // (a split-K part starts at K block flags >> 8 of its tile's packed weights)
        const int kb_first = SPLIT ? static_cast<int>(static_cast<uint32_t>(w.flags) >> kItemKb0Shift) : 0;
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const uint32_t s = it % kStages;
          const uint32_t ph = (it / kStages) & 1u;
          ok = mbar_wait(smem_u32(&bars->empty[s]), ph ^ 1u, abort_flag);
          if (!ok) break;
          const uint32_t bar = smem_u32(&bars->full[s]);
          mbar_arrive_expect_tx(bar, kWBytes);
          tma_load_2d(smem_u32(smem + s * C::kStageBytes), &tmap_w, (kb + kb_first) * kKB, w.w_row0, bar);
          const uint32_t slot = (it + kAhead) % C::kRecs;
          const uint32_t rbar = smem_u32(&bars->rec_full[slot]);
          mbar_arrive_expect_tx(rbar, kMetaInts * 4);
          bulk_load(smem_u32(bars->rec[slot]), recs + static_cast<size_t>(it + kAhead) * kMetaInts, kMetaInts * 4, rbar);
        }
        w = wn;
      }
      // the records past the end marker (never read) must have landed before the CTA retires
      for (uint32_t i = it; i < it + kAhead; ++i) {
        mbar_wait(smem_u32(&bars->rec_full[i % C::kRecs]), (i / C::kRecs) & 1u, abort_flag);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // One elected thread runs the whole loop (see elect_one).  The MMA's N dimension is the unit's
    // batch-row count (at most MT).
    constexpr uint32_t idesc0 = umma_idesc_f16(DT == kBF16 ? 1 : 0, /*a_mn=*/0, /*b_mn=*/1, kNT, 0);
    if (elect_one()) {
      uint32_t it = 0, acc_it = 0;
      bool ok = true;
      for (int r = 0; ok && w.tile >= 0; ++r) {
        const WorkItem wn = fetch_item(sched, rounds, grid, cta, r + 1);
        const int nkb = (w.k_count + kKB - 1) / kKB;
        const uint32_t a = acc_it & 1u;
        const uint32_t aph = (acc_it >> 1) & 1u;
        ok = mbar_wait(smem_u32(&bars->acc_empty[a]), aph ^ 1u, abort_flag);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + a * MT;
        // batch rows past the end of the matrix are neither gathered nor multiplied (N in steps of 16)
        const int n_cols = min(w.m_len, (M - w.m_begin + 15) & ~15);
        const uint32_t idesc = idesc0 | (static_cast<uint32_t>(n_cols >> 3) << 17);
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const uint32_t s = it % kStages;
          const uint32_t ph = (it / kStages) & 1u;
          ok = mbar_wait(smem_u32(&bars->full[s]), ph, abort_flag);
          if (!ok) break;
          // The gathered rows were written through the generic proxy; the MMA reads them through
          // the async proxy.
          fence_proxy_async_smem();
          tc_fence_after_sync();
          const int krem = w.k_count - kb * kKB;
          const int nk16 = krem >= kKB ? kKB / 16 : (krem + 15) / 16;
          const uint32_t w_addr = smem_u32(smem + s * C::kStageBytes);
          const uint32_t a_addr = w_addr + kWBytes;
          // weights: K-major, 16 K elements = 32 bytes inside the 128-byte swizzled row; activations:
          // MN-major, 16 K rows = two 8-row groups
          const uint64_t dw = umma_smem_desc_sw128(w_addr, 16, kWSbo);
          const uint64_t da = umma_smem_desc_sw128(a_addr, kALbo, kASbo);
#pragma unroll
          for (int k = 0; k < kKB / 16; ++k) {
            if (k < nk16) {
              umma_f16(tmem_d, dw + static_cast<uint64_t>(k * 32 >> 4), da + static_cast<uint64_t>(k * 2 * kASbo >> 4), idesc,
                       (kb > 0 || k > 0) ? 1u : 0u);
            }
          }
          umma_commit(smem_u32(&bars->empty[s]));
        }
        if (!ok) break;
        if (nkb > 0) {
          umma_commit(smem_u32(&bars->acc_full[a]));
        } else {
          mbar_arrive(smem_u32(&bars->acc_full[a]));  // tile with no kept rows: nothing to wait for
        }
        ++acc_it;
        w = wn;
      }
    }
  } else if (warp < kEpiWarp0) {
    // ------------------------------------------------------------------ activation gather
    // Group p of warps takes the blocks p, p + kWarpGroups, ... (16 rows a warp).  Per block: wait for
    // the stage, issue the warp's rows in one burst of 16-byte copies, hand them to the stage's barrier.
    // The row numbers of the group's next block go from the record ring to registers before that wait, so neither
    // the record nor a shared-memory read sits between a free stage and its copies (a read between two
    // copies would also stall the warp until the load/store unit has taken the copies before it).
    constexpr int kLpr = C::kLanesPerRow, kRpi = C::kRowsPerInstr;
    const int chunk = lane % kLpr, sub = lane / kLpr;
    const int g = chunk >> 3, c = chunk & 7;
    const uint32_t group = (warp - kGatherWarp0) / kWarpsPerBlock;
    const int row_base = ((warp - kGatherWarp0) % kWarpsPerBlock) * kRowsPerWarp;         // first row of the warp's slice
    int rr[kRowsPerWarp], rn[kRowsPerWarp];
    int m0 = 0, m0_next;
    uint32_t meta = kBlockEnd, meta_next;
    auto read_record = [&](uint32_t j, int& m0_out, uint32_t& meta_out, int (&rows)[kRowsPerWarp]) -> bool {
      const uint32_t slot = j % C::kRecs;
      if (!mbar_wait(smem_u32(&bars->rec_full[slot]), (j / C::kRecs) & 1u, abort_flag)) return false;
      const int* rec = bars->rec[slot];
      const int2 head = *reinterpret_cast<const int2*>(rec);
      m0_out = head.x;
      meta_out = static_cast<uint32_t>(head.y);
#pragma unroll
      for (int q4 = 0; q4 < kRowsPerWarp / 4; ++q4) {
        const int4 v = *reinterpret_cast<const int4*>(rec + 4 + row_base + q4 * 4);
        rows[q4 * 4] = v.x;
        rows[q4 * 4 + 1] = v.y;
        rows[q4 * 4 + 2] = v.z;
        rows[q4 * 4 + 3] = v.w;
      }
      return true;
    };
    bool ok = read_record(group, m0, meta, rr);
    // The schedule is static; the activations may be the previous kernel's output: wait for it
    // before the first row is copied.
    grid_dependency_wait();

    for (uint32_t j = group; ok && meta != kBlockEnd; j += kWarpGroups) {
      if (!read_record(j + kWarpGroups, m0_next, meta_next, rn)) break;
      const int nv = static_cast<int>(meta & 0x7fu) - row_base;                 // valid rows of the slice
      const int m_len = (static_cast<int>((meta >> 8) & 3u) + 1) * 64;          // batch rows of the unit
      const int m = m0 + chunk * 8;
      // lanes past the unit or past the batch: their columns are never multiplied into a stored result
      const bool live = chunk * 8 < m_len && m < M;
      const uint16_t* src_col = At + m;
      const uint32_t s = j % kStages;
      const uint32_t ph = (j / kStages) & 1u;
      const uint32_t dst0 = smem_u32(smem + s * C::kStageBytes + kWBytes) + g * kALbo;
      const uint32_t bar = smem_u32(&bars->full[s]);
      if (!mbar_wait(smem_u32(&bars->empty[s]), ph ^ 1u, abort_flag)) break;
      // Two separate bursts: mixing the zero-fill form into the loop of plain copies makes every
      // copy as slow as the zero-fill form.  A slice without valid rows is not multiplied at all.
      if (live && nv >= kRowsPerWarp) {
#pragma unroll
        for (int e = 0; e < kRowsPerWarp / kRpi; ++e) {
          const int row = row_base + e * kRpi + sub;
          int kr;
          if constexpr (kRpi == 1) {
            kr = rr[e];
          } else {
            kr = sub ? rr[e * 2 + 1] : rr[e * 2];
          }
          cp_async_16_full(dst0 + (row >> 3) * kASbo + (row & 7) * 128 + ((c ^ (row & 7)) << 4),
                           src_col + (static_cast<long long>(kr) << 3));
        }
      } else if (live && nv > 0) {
#pragma unroll
        for (int e = 0; e < kRowsPerWarp / kRpi; ++e) {
          const int row = row_base + e * kRpi + sub;
          int kr;
          if constexpr (kRpi == 1) {
            kr = rr[e];
          } else {
            kr = sub ? rr[e * 2 + 1] : rr[e * 2];
          }
          const bool valid = row - row_base < nv;
          cp_async_16(dst0 + (row >> 3) * kASbo + (row & 7) * 128 + ((c ^ (row & 7)) << 4),
                      valid ? src_col + (static_cast<long long>(kr) << 3) : At, valid ? 16u : 0u);
        }
      }
      cp_async_arrive_noinc(bar);
      m0 = m0_next;
      meta = meta_next;
#pragma unroll
      for (int e = 0; e < kRowsPerWarp; ++e) rr[e] = rn[e];
    }
    cp_async_wait_all();  // nothing of this thread is in flight when the CTA retires
  } else {
    // ------------------------------------------------------------------ epilogue
    // Every warp works alone: it owns 32 tile columns (its TMEM lane quarter) and every other 64-column
    // group of the unit's batch, stages a group (32 rows x 128 bytes, 128-byte swizzle) in a buffer of its
    // own and sends it off, as one TMA tile store where its 32 rows are consecutive rows of Ct, else with
    // 16-byte stores through the kept-column list.  No barrier between warps.  What bounds it is the SM's
    // store path (32 bytes per cycle: 2048 cycles for a 256 x 128 unit; 6.4 TB/s over the GPU), whatever
    // the kind of store; direct stores instead of TMA take that time from the gather's load/store queue
    // (2048 x 4096 layer at 6400 rows: 51 thousand cycles per CTA instead of 44).
    const int ew = warp - kEpiWarp0;             // 0..7
    const int half = ew >> 2;                    // takes the 64-column groups half, half+2, ...
    const int q = warp & 3;                      // TMEM lane quarter this warp may read
    const int j = q * 32 + lane;                 // tile column owned by this thread
    const int peer_rot = (PEERS && ep.n_peers > 0) ? cta % ep.n_peers : 0;   // the peer this CTA writes first
    uint8_t* const own_stage = epi + ew * kEpiWarpBytes;
    // Work items are held one word per lane, the next one in flight while this one is worked on: whole
    // copies in every lane cost the registers that two TMEM chunks need.
    const int* const items = reinterpret_cast<const int*>(sched + cta) + lane;
    auto item_word = [&](int r) -> int {
      return r < rounds && lane < kItemWords ? ld_coherent(items + static_cast<size_t>(r) * grid * kItemWords) : -1;
    };
    int word = item_word(0);
    grid_dependency_wait();   // Ct may still be read or written by the previous kernel
    // Tensor maps that live in device memory: an earlier one may have stood at the same address.
    if constexpr (SPLIT) if (lane == 0) fence_tensormap(ep.scratch_map);
    if constexpr (PEERS) if (lane == 0 && ep.peer_maps != nullptr) {
      for (int p = 0; p < ep.n_peers; ++p) fence_tensormap(ep.peer_maps + p);
    }
    for (uint32_t r = 0; __shfl_sync(0xffffffffu, word, kItemWordTile) >= 0; ++r) {
      const int word_next = item_word(r + 1);
      const EpiItem w = epi_item(word);
      const uint32_t a = r & 1u;
      const uint32_t aph = (r >> 1) & 1u;
      const int m0 = w.m_begin;
      const int m_cnt = min(w.m_len, M - m0);
      const bool active = j < w.n_count;
      // TMA store of the local copy: consecutive Ct rows, nothing to read back
      const bool tma_store = LEAN || (use_tma_store && (w.flags & kItemDenseRows) && beta == 0.0f &&
                                      (!PEERS || ep.multicast == nullptr));
      const bool tma_peers = PEERS && tma_store && ep.peer_maps != nullptr;   // the peers' copies leave by TMA too
      // The CTA's last unit: every K block has been consumed, so the pipeline stages are free and
      // each group gets a staging buffer of its own there; none waits for a store before it.
      const bool last_unit = __shfl_sync(0xffffffffu, word_next, kItemWordTile) < 0;
      const int tile_row0 = w.c_row0 + ((tma_store && w.n_list) ? ld_coherent(w.n_list) : 0);
      // (the store-only variants' tiles keep consecutive columns: no list to read, and nothing to wait for without a bias)
      const long long c_row = !active ? 0 : (LEAN ? tile_row0 + j : c_row_of(w, j));
      const int c_row_or_none = active ? static_cast<int>(c_row) : -1;
      const float bias_j = (ep.bias != nullptr && active) ? ld_coherent(ep.bias + c_row) : 0.0f;
      if (!mbar_wait(smem_u32(&bars->acc_full[a]), aph, abort_flag)) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + a * MT + (static_cast<uint32_t>(q * 32) << 16);
      const bool has_acc = w.has_rows;
      // Not unrolled, and 32 accumulators in registers at a time: the hot code stays small enough for the
      // instruction cache it shares with the other roles, and nothing spills (a spilled register waits
      // behind the gather's copies in the load/store queue: with 64 accumulators a unit took 7000 cycles).
#pragma unroll 1
      for (int gi = 0; gi < C::kGroups; ++gi) {
        const int col0 = (gi * 2 + half) * 64;              // first batch column of the group
        const int cols = m_cnt - col0;                      // (uniform over the warp)
        uint8_t* stage = last_unit ? smem + (ew * C::kGroups + gi) * kEpiWarpBytes : own_stage;
#pragma unroll 1
        for (int b = 0; b < 2; ++b) {
          uint32_t v[32];
          if (has_acc && cols > b * 32) {
            tmem_ld_32x32(taddr + col0 + b * 32, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = 0u;
          }
          if (gi + 1 == C::kGroups && b == 1) {
            // every TMEM read of this accumulator by this warp has completed: hand it back to the MMA warp
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->acc_empty[a]));
          }
          if (cols <= b * 32) continue;
          if constexpr (SPLIT) if (w.flags & kItemScratch) {
            // split-K part: alpha * acc leaves as fp32 for the part's scratch rows (32 rows x 128 bytes);
            // bias, beta and the activation are applied by the kernel that adds the parts up.  (Tile
            // columns past n_count carry zero weights, so their rows receive zeros.)
            if (lane == 0) bulk_wait_read_all();
            __syncwarp();
#pragma unroll
            for (int cc = 0; cc < 8; ++cc) {
              *reinterpret_cast<float4*>(own_stage + lane * 128 + ((cc ^ (lane & 7)) << 4)) =
                  make_float4(alpha * __uint_as_float(v[cc * 4]), alpha * __uint_as_float(v[cc * 4 + 1]),
                              alpha * __uint_as_float(v[cc * 4 + 2]), alpha * __uint_as_float(v[cc * 4 + 3]));
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(ep.scratch_map, smem_u32(own_stage), m0 + col0 + b * 32, w.c_row0 + q * 32);
              bulk_commit();
            }
            continue;
          }
          if (b == 0 && !last_unit) {
            if (lane == 0) bulk_wait_read_all();            // the store before this one has read the buffer
            __syncwarp();
          }
          uint8_t* const row_ptr = stage + lane * 128;
          auto convert = [&](auto act_c) {
            constexpr int kAct = decltype(act_c)::value;
#pragma unroll
            for (int p = 0; p < 4; ++p) {                   // eight batch columns, one 16-byte piece
              float y[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) y[e] = fmaf(alpha, __uint_as_float(v[p * 8 + e]), bias_j);
              if constexpr (!LEAN) {
                const int col = b * 32 + p * 8;
                if (beta != 0.0f && active && col < cols) {
                  const uint4 old = *reinterpret_cast<const uint4*>(Ct + c_row * ldc + m0 + col0 + col);
                  const uint32_t ow[4] = {old.x, old.y, old.z, old.w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    y[e * 2] = fmaf(beta, unpack1<DT>(static_cast<uint16_t>(ow[e] & 0xffffu)), y[e * 2]);
                    y[e * 2 + 1] = fmaf(beta, unpack1<DT>(static_cast<uint16_t>(ow[e] >> 16)), y[e * 2 + 1]);
                  }
                }
              }
              if constexpr (kAct == kActRelu) {
#pragma unroll
                for (int e = 0; e < 8; ++e) y[e] = fmaxf(y[e], 0.0f);
              }
              if constexpr (kAct == kActGelu) {
#pragma unroll
                for (int e = 0; e < 4; ++e) gelu2(y[e * 2], y[e * 2 + 1]);
              }
              if constexpr (ROWS) {
                // row-major: two neighbouring lanes (columns n, n + 1) swap halves, so that each holds one
                // batch row of the column pair; staged as [64 batch rows][32 columns], a store instruction
                // covers two rows of 64 bytes
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const uint32_t own = pack2<DT>(y[e * 2], y[e * 2 + 1]);
                  const uint32_t other = __shfl_xor_sync(0xffffffffu, own, 1);
                  const uint32_t pair = (lane & 1) ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
                  *reinterpret_cast<uint32_t*>(stage + (b * 32 + p * 8 + e * 2 + (lane & 1)) * 64 + (lane >> 1) * 4) = pair;
                }
              } else {
                *reinterpret_cast<uint4*>(row_ptr + (((b * 4 + p) ^ (lane & 7)) << 4)) =
                    make_uint4(pack2<DT>(y[0], y[1]), pack2<DT>(y[2], y[3]), pack2<DT>(y[4], y[5]), pack2<DT>(y[6], y[7]));
              }
            }
          };
          if (act == kActNone) convert(std::integral_constant<int, kActNone>{});
          else if (act == kActRelu) convert(std::integral_constant<int, kActRelu>{});
          else convert(std::integral_constant<int, kActGelu>{});
        }
        if (cols <= 0) continue;
        if constexpr (SPLIT) if (w.flags & kItemScratch) continue;
        if constexpr (NHWC) {
          // 64 pixels x 32 channels (64 bytes a pixel): four lanes per pixel, eight pixels of one image row per
          // instruction.  Against a Ct in the padded space and an unpacking kernel this saves both their
          // traffic and a launch: 8 images of 112 x 112, 64 -> 128 channels, 49.4 -> 35.5 us a pass.
          __syncwarp();
          const int piece = lane & 3, sub = lane >> 2;
          const bool ch_ok = q * 32 + piece * 8 < w.n_count;
          uint16_t* const out = Ct + tile_row0 + q * 32 + piece * 8;
          const int n_px8 = min(8, cols >> 3);
          uint4 val[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) val[r] = *reinterpret_cast<const uint4*>(stage + (r * 8 + sub) * 64 + piece * 16);
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const uint32_t g = static_cast<uint32_t>(m0 + col0) / 8 + r;           // group of eight padded pixels
            const int row = ep.nhwc_mul_wp8 ? static_cast<int>(__umulhi(g, ep.nhwc_mul_wp8)) : static_cast<int>(g);
            const int x = (static_cast<int>(g) - row * ep.nhwc_wp8) * 8 + sub;
            const int img = ep.nhwc_mul_hp ? static_cast<int>(__umulhi(static_cast<uint32_t>(row), ep.nhwc_mul_hp)) : row;
            const int y = row - img * ep.nhwc_hp;
            if (r < n_px8 && y < ep.nhwc_h && x < ep.nhwc_w && ch_ok) {
              *reinterpret_cast<uint4*>(out + ((static_cast<long long>(img) * ep.nhwc_h + y) * ep.nhwc_w + x) * ldc) = val[r];
            }
          }
          __syncwarp();
        } else if (tma_store) {
          fence_proxy_async_smem();
          __syncwarp();                          // the whole group is staged
          if (lane == 0 && q * 32 < w.n_count) {
            if constexpr (ROWS) tma_store_2d(&tmap_c, smem_u32(stage), tile_row0 + q * 32, m0 + col0);
            else tma_store_2d(&tmap_c, smem_u32(stage), m0 + col0, tile_row0 + q * 32);
            if constexpr (PEERS) if (tma_peers) {
              for (int p = 0; p < ep.n_peers; ++p) {
                int pp = p + peer_rot;
                if (pp >= ep.n_peers) pp -= ep.n_peers;
                tma_store_2d(ep.peer_maps + pp, smem_u32(stage), m0 + col0, tile_row0 + q * 32);
              }
            }
            bulk_commit();
          }
        }
        if constexpr (!LEAN) {
          if (!tma_store || (PEERS && ep.n_peers > 0 && !tma_peers)) {
            // copy-out through the kept-column list: this warp's own 32 rows, four rows per instruction,
            // 16 bytes per lane; to Ct unless the TMA store took it, and to every peer.  Tile-sharded
            // layers: the peers are the other GPUs' copies of Ct, written over NVLink; CTAs start at
            // different peers so that the GPUs' stores do not converge on one destination at a time.
            __syncwarp();
            const int piece = lane & 7, rsub = lane >> 3;
            const bool m_ok = piece * 8 < cols;
#pragma unroll
            for (int r4 = 0; r4 < 32; r4 += 16) {
              int cr[4];
              uint4 val[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int row = r4 + e * 4 + rsub;              // row inside the warp's quarter
                cr[e] = __shfl_sync(0xffffffffu, c_row_or_none, row);
                val[e] = *reinterpret_cast<const uint4*>(stage + row * 128 + ((piece ^ (row & 7)) << 4));
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                if (cr[e] >= 0 && m_ok) {
                  const long long off = static_cast<long long>(cr[e]) * ldc + m0 + col0 + piece * 8;
                  if constexpr (PEERS) {
                    if (ep.multicast != nullptr) {
                      multimem_st_16(ep.multicast + off, val[e]);     // every GPU's copy, this one included
                      continue;
                    }
                  }
                  if (!tma_store) *reinterpret_cast<uint4*>(Ct + off) = val[e];
                  if constexpr (PEERS) {
                    for (int p = 0; p < ep.n_peers; ++p) {
                      int pp = p + peer_rot;
                      if (pp >= ep.n_peers) pp -= ep.n_peers;
                      *reinterpret_cast<uint4*>(ep.peers[pp] + off) = val[e];
                    }
                  }
                }
              }
            }
            __syncwarp();
          }
        }
      }
      word = word_next;
    }
    // The CTA may retire once its last TMA stores have read the staging buffers; the stores
    // themselves complete before the grid does.
    if (lane == 0) bulk_wait_read_all();
  }

  __syncwarp();   // warps 0 and 1 ran their roles on one elected thread
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, C::kTmemCols);
  if (threadIdx.x == 0 && bars->abort_flag) atomicExch(status, kErrTimeout);
}

// One record per K block of a schedule: {first batch row of the unit, meta word, 0, 0} followed by
// the start of the 64 rows the block gathers (0 past the block's last row), each as a count of
// 16-byte segments from the activation base pointer.  For a matrix At[K][lda] kept row k starts at
// segment k * lda / 8.  For a convolution the "matrix" is never materialised: kept row
// k = (r * kw + j) * cin + c of the im2col matrix (Pruning/VGG/prune_algo.py:16-24 fixes that order)
// is channel c of the copy of the padded input shifted by j pixels, read r image rows further down:
// segment ((j * cin + c) * plane_ld + r * Wp) / 8.  The kept row number itself comes from the tile's
// list, or list position + offset for lists in the reference's relative form.
// Lists that the caller hands over per call (reference-signature entry point): `lists` carries their addresses, the
// descriptors hold the tile's number (stream_list_code) plus the byte offset inside its list instead of an address, and
// the work items get their column lists here.
__device__ __forceinline__ void expand_record(const BlockDesc& d, const int* idx, int r, int* rec, const RowMap& map) {
  int v = 0;
  if (d.meta != kBlockEnd && r < static_cast<int>(d.meta & 0x7fu)) {
    v = ld_coherent(idx + r);
    if (d.meta & 0x80u) v += static_cast<int>(d.meta >> 10) + r;
    if (map.conv_cin > 0) {
      const int c = v % map.conv_cin, rj = v / map.conv_cin;
      const int j = rj % map.conv_kw, rr = rj / map.conv_kw;
      v = static_cast<int>((static_cast<long long>(j) * map.conv_cin + c) * map.ld8 + static_cast<long long>(rr) * map.conv_wp8);
    } else {
      v = static_cast<int>(static_cast<long long>(v) * map.ld8);
    }
  }
  rec[4 + r] = v;
  if (r < 4) rec[r] = r == 0 ? d.m0 : (r == 1 ? static_cast<int>(d.meta) : 0);
}

__global__ void __launch_bounds__(256)
expand_block_meta_kernel(const BlockDesc* __restrict__ blocks, long long n_blocks, int* __restrict__ meta,
                         const RowMap map) {
  const long long b = blockIdx.x * 4LL + (threadIdx.x >> 6);
  if (b >= n_blocks) return;
  const BlockDesc d = blocks[b];
  expand_record(d, d.idx, threadIdx.x & 63, meta + b * kMetaInts, map);
}

__global__ void __launch_bounds__(256)
expand_stream_kernel(const BlockDesc* __restrict__ blocks, int n_blocks, int* __restrict__ meta, WorkItem* __restrict__ items,
                     int n_items, const RowMap map, const __grid_constant__ StreamLists lists) {
  grid_launch_dependents();
  // the GEMM before this kernel may still be reading the records and items of the call before
  grid_dependency_wait();
  const int b = blockIdx.x * 4 + (threadIdx.x >> 6);
  if (b < n_blocks) {
    const BlockDesc d = blocks[b];
    const unsigned long long code = reinterpret_cast<unsigned long long>(d.idx);
    const int* idx = d.meta == kBlockEnd ? nullptr : lists.k[code >> kStreamTileShift] + (code & ((1ull << kStreamTileShift) - 1)) / 4;
    expand_record(d, idx, threadIdx.x & 63, meta + static_cast<long long>(b) * kMetaInts, map);
  }
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n_items && items[i].tile >= 0) items[i].n_list = lists.n[items[i].tile];
}

// Second pass of a split-K schedule: Ct[row][m] = act(sum of the parts' fp32 partial sums + beta * Ct[row][m]
// + bias[row]) for every kept column of every split tile.  grid (ceil(M / 8 / 256), 128, split tiles).
template <int DT>
__global__ void __launch_bounds__(256)
split_reduce_kernel(const SplitTile* __restrict__ tiles, const float* __restrict__ scratch, long long sld,
                    uint16_t* __restrict__ Ct, long long ldc, int M, float beta, const float* __restrict__ bias,
                    int act) {
  const SplitTile t = tiles[blockIdx.z];
  const int j = blockIdx.y;
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (j >= t.n_count || m >= M) return;
  const long long row = t.c_row0 + (t.n_list ? __ldg(t.n_list + j) + (t.relative ? j : 0) : j);
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.0f;
  for (int p = 0; p < t.parts; ++p) {
    const float4* src = reinterpret_cast<const float4*>(scratch + (static_cast<long long>(t.scratch_row0) + p * 128 + j) * sld + m);
    const float4 a = src[0], b = src[1];
    acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
    acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
  }
  uint4* dst = reinterpret_cast<uint4*>(Ct + row * ldc + m);
  uint32_t oldw[4] = {0, 0, 0, 0};
  if (beta != 0.0f) {
    const uint4 o = *dst;
    oldw[0] = o.x; oldw[1] = o.y; oldw[2] = o.z; oldw[3] = o.w;
  }
  const float bj = bias ? __ldg(bias + row) : 0.0f;
  uint32_t out[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float c0 = unpack1<DT>(static_cast<uint16_t>(oldw[e] & 0xffffu));
    const float c1 = unpack1<DT>(static_cast<uint16_t>(oldw[e] >> 16));
    const float y0 = acc[2 * e] + beta * c0 + bj;
    const float y1 = acc[2 * e + 1] + beta * c1 + bj;
    out[e] = pack2<DT>(apply_act(y0, act), apply_act(y1, act));
  }
  *dst = make_uint4(out[0], out[1], out[2], out[3]);
}

template <int DT, int MT, int MODE>
cudaError_t launch_variant(const CUtensorMap& tmap_w, const CUtensorMap& tmap_c, int flags,
                           const WorkItem* sched, int rounds, int grid, const int* block_meta, int blk_stride,
                           const void* At, long long lda, void* Ct, long long ldc, int M,
                           const EpilogueArgs& ep, int* status, cudaStream_t stream) {
  // Programmatic dependent launch lets this kernel's set-up overlap the tail of the kernel before it in
  // the stream; what it may read before that kernel has completed is the caller's choice (kFlagWaitFirst).
  auto kern = masked_gemm_kernel<DT, MT, MODE>;
  // The dynamic shared-memory limit is a per-device, per-kernel attribute: set it once for each.
  static bool attr_set[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !attr_set[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<MT>::kSmemBytes);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Cfg<MT>::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, tmap_w, tmap_c, flags, sched, rounds, block_meta, blk_stride,
                            static_cast<const uint16_t*>(At), lda, static_cast<uint16_t*>(Ct), ldc, M,
                            ep, status);
}

}  // namespace

cudaError_t masked_gemm_launch(int dtype, int unit_rows, const CUtensorMap& tmap_w, const CUtensorMap* tmap_c,
                               const WorkItem* sched, int rounds, int grid, const int* block_meta,
                               int blk_stride, const void* At, long long lda, void* Ct, long long ldc, int M,
                               const EpilogueArgs& ep, int* status, bool early_start, bool lean, OutForm form,
                               cudaStream_t stream) {
#define TS_LAUNCH(DT, MT, MD)                                                                                  \
  launch_variant<DT, MT, MD>(tmap_w, tmap_c ? *tmap_c : tmap_w, flags, sched, rounds, grid, block_meta, \
                             blk_stride, At, lda, Ct, ldc, M, ep, status, stream)
#define TS_LAUNCH_DT(MT, MD) (dtype == kBF16 ? TS_LAUNCH(kBF16, MT, MD) : TS_LAUNCH(kF16, MT, MD))
  const int flags = (tmap_c ? kFlagTmaStore : 0) | (early_start ? 0 : kFlagWaitFirst);
  if (unit_rows != 256 && unit_rows != 128) return cudaErrorInvalidValue;
  if (form != kOutColumns) {
    if (!lean || ep.beta != 0.0f || ep.scratch_map || ep.n_peers > 0 || ep.multicast) return cudaErrorInvalidValue;
    if (form == kOutNhwc) return unit_rows == 256 ? TS_LAUNCH_DT(256, kModeNhwc) : TS_LAUNCH_DT(128, kModeNhwc);
    if (tmap_c == nullptr) return cudaErrorInvalidValue;
    return unit_rows == 256 ? TS_LAUNCH_DT(256, kModeRows) : TS_LAUNCH_DT(128, kModeRows);
  }
  // a schedule with split-K parts never writes peers (the host keeps the two apart)
  if (ep.scratch_map != nullptr) return unit_rows == 256 ? TS_LAUNCH_DT(256, kModeSplit) : TS_LAUNCH_DT(128, kModeSplit);
  if (ep.n_peers > 0 || ep.multicast != nullptr) {
    return unit_rows == 256 ? TS_LAUNCH_DT(256, kModePeers) : TS_LAUNCH_DT(128, kModePeers);
  }
  // lean: the caller has checked that every unit takes the TMA store
  if (lean && tmap_c != nullptr && ep.beta == 0.0f) {
    return unit_rows == 256 ? TS_LAUNCH_DT(256, kModeLean) : TS_LAUNCH_DT(128, kModeLean);
  }
  return unit_rows == 256 ? TS_LAUNCH_DT(256, kModePlain) : TS_LAUNCH_DT(128, kModePlain);
#undef TS_LAUNCH_DT
#undef TS_LAUNCH
  return cudaErrorInvalidValue;
}

cudaError_t split_reduce_launch(int dtype, const SplitTile* tiles, int n_split, const float* scratch, long long sld,
                                void* Ct, long long ldc, int M, float beta, const float* bias, int act,
                                cudaStream_t stream) {
  if (n_split <= 0 || M <= 0) return cudaSuccess;
  dim3 grid(static_cast<unsigned>((M / 8 + 255) / 256), 128, n_split);
  if (dtype == kBF16) {
    split_reduce_kernel<kBF16><<<grid, 256, 0, stream>>>(tiles, scratch, sld, static_cast<uint16_t*>(Ct), ldc, M, beta, bias, act);
  } else {
    split_reduce_kernel<kF16><<<grid, 256, 0, stream>>>(tiles, scratch, sld, static_cast<uint16_t*>(Ct), ldc, M, beta, bias, act);
  }
  return cudaGetLastError();
}

cudaError_t expand_block_meta_launch(const BlockDesc* blocks, long long n_blocks, int* meta, const RowMap& map,
                                     cudaStream_t stream) {
  if (n_blocks <= 0) return cudaSuccess;
  expand_block_meta_kernel<<<static_cast<unsigned>((n_blocks + 3) / 4), 256, 0, stream>>>(blocks, n_blocks, meta, map);
  return cudaGetLastError();
}

cudaError_t expand_stream_launch(const BlockDesc* blocks, int n_blocks, int* meta, WorkItem* items, int n_items,
                                 const RowMap& map, const StreamLists& lists, cudaStream_t stream) {
  const int n = (n_blocks + 3) / 4 > (n_items + 255) / 256 ? (n_blocks + 3) / 4 : (n_items + 255) / 256;
  if (n <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(n));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, expand_stream_kernel, blocks, n_blocks, meta, items, n_items, map, lists);
}

}  // namespace ts
