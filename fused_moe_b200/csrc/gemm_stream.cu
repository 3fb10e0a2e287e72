// Grouped FP8 GEMMs for calls of few tokens (at most kStreamMaxTokens): the weight stream.
//
// With a handful of rows per expert the layer is bound by reading expert weights from HBM (44 MB per active expert), so
// the tile is turned around: the 128 MMA rows (TMEM lanes) are weight rows, the MMA's N is the tile's token rows (16, 32 or
// 64; an expert holds no more rows than the call has tokens).  Arithmetic is the one of gemm.cu (which replaces the
// reference's `moe_blockwise_grouped_mm_v2`, solution/python/moe_gemm.cu:527-654, whose own small-batch configuration also
// swaps A and B, moe_gemm.cu:614-648): raw e4m3 dot product per 128-wide K block, promoted in fp32 registers with the
// fp32 block scales.
//
// What bounds it besides HBM is the number of hand-offs: a wait on an mbarrier, a TMA issue, four MMAs with their commits or a
// read-back of tensor memory each cost their warp a few hundred cycles whatever their size, and 16 KB of weights take ~690
// cycles to arrive at an SM's share of the measured HBM rate.  Therefore
//   * two K blocks travel and are handed over together (one 4D weight box of 32 KB, one accumulator group of two times
//     16 columns, one wait of every role): one K block at a time took 860 cycles per K block, promotion warps and issuer both
//     busy; two take 520 with one MMA issuer and 440 with two;
//   * the (slab, K group) units of the whole call are cut into one contiguous range per SM, so that every SM reads the same
//     number of weight bytes; a slab whose range is cut leaves fp32 partial sums in scratch, the CTA that arrives last
//     adds them in range order and runs the epilogue, so results stay run-to-run identical.
// Whole calls, 32 experts (11 active, 16 tokens) 157 -> 110 us, 5 active (1 token) 81 -> 59; 256 experts, 4 tokens (30 active,
// 1.32 GB of weights) 313 -> 241 us, of which GEMM1 167 at 5.3 TB/s and GEMM2 77 at 5.7 TB/s.
// Measured and dropped: GEMM1 and GEMM2 sharing the SMs so that GEMM2's first weights travel early (three and two stages
// instead of five each: 2 to 4 % slower); three MMA issuers (no change); promotion without its FMAs, boxes without the
// token rows, another L2 promotion (no change: neither bounds it); tiles of up to 128 token rows for larger calls (901 tokens:
// 432 us against 245 with the 128 x 256 tiles of gemm.cu).
//
// Work item = (M tile of the packed rows, slab of 128 weight rows).  GEMM1's slab is 64 gate rows plus the 64 matching
// up rows (one box over the expert's two planes), so lanes 0-63 hold g and lanes 64-127 hold u of the same columns.
// Warps: 0 and the last ones TMA producers (one lane each, groups in turn); 1, 2 MMA issuers (alternate groups); 3 a producer;
// from 4 promotion and epilogue, one warp per TMEM lane quarter (NT = 64: two, taking alternate chunks of 16 token columns).
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.cuh"
#include "stream_plan.cuh"

namespace b200moe {

namespace {

constexpr int kSlabRows = 128;
constexpr int kWBytes = kSlabRows * kBlockK;   // 16 KiB of weights per K block
constexpr int kGroup = kStreamGroup;           // K blocks per hand-off: one stage, one accumulator group, one wait of each role
constexpr int kAccs = 4;                       // accumulator groups in tensor memory
constexpr int kScaleSlots = 16;                // ring of activation scales; see the reuse argument at the producer
constexpr int kMaxKBlocks = 64;                // a lane keeps two of an item's weight scales
constexpr int kTileTable = 32;                 // M tiles one CTA's range may touch (checked by the host)

template <int MODE, int NT> struct SCfg {
  static constexpr int kTokBytes = NT * kBlockK;                      // of one K block
  static constexpr int kStageBytes = kGroup * (kWBytes + kTokBytes);  // [group][128 weight rows], [group][NT token rows]
  static constexpr int kStages = NT <= 16 ? 5 : 4;
  static constexpr int kIssuers = 2;
  static constexpr int kProducers = NT <= 16 ? kStages : 2;   // (12 warps in all: a 13th costs every thread 40 registers; at 168 <1, 64> spills 16 bytes)
  // The roles wait by parity, so nobody may wait for a phase while the one before last is still open.  A producer owns its
  // stages.  The issuers take turns on an odd number of stages; an issuer waits for its accumulators first, i.e. until group
  // it - kAccs has been promoted, and that has to cover the stage's previous use, group it - kStages.
  static_assert(kStages % kProducers == 0 && kAccs <= kStages, "a parity wait could pass a phase early");
  static constexpr int kHalves = NT <= 16 ? 1 : 2;       // promotion warps per TMEM lane quarter
  static constexpr int kPromoWarps = 4 * kHalves;
  static constexpr int kWarps = kIssuers + kProducers + kPromoWarps;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kRingBytes = MODE == 1 ? kScaleSlots * kGroup * NT * 4 : 0;
  static constexpr int kXchBytes = MODE == 1 ? 64 * NT * 4 : 0;   // u values of 64 up rows, [token][row]
  // token rows read where the caller keeps them: each promotion warp's copy of a tile's token scales, [K block][16]
  static constexpr int kPanelBytes = MODE == 1 && NT == 16 ? kMaxKBlocks * 16 * 4 : 0;
  static constexpr int kToksBytes = MODE == 1 && NT == 16 ? kTileTable * 16 * 4 : 0;
  static constexpr int kTmemCols = kAccs * kGroup * NT;
  static constexpr int kSmemBytes = kStages * kStageBytes + kRingBytes + kXchBytes + 4 * kPanelBytes + kToksBytes + 512 +
                                    kTileTable * 8 + 1024;
  static_assert(kScaleSlots >= kStages + kAccs + 1, "activation scales would be overwritten before their last read");
  static_assert(kSmemBytes <= 227 * 1024, "more shared memory than a CTA may have");
  static_assert(kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "tensor memory");
};
static_assert(kGroup == 2, "the promotion loop below reads two K blocks per hand-off");

// 32 lanes x 16 consecutive fp32 columns, and waits that name the loaded registers
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_on(uint32_t (&a)[16], uint32_t (&b)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : B200MOE_RW8(a, 0), B200MOE_RW8(a, 8), B200MOE_RW8(b, 0), B200MOE_RW8(b, 8)
               :
               : "memory");
}
__device__ __forceinline__ void tmem_wait_on(uint32_t (&a)[16], uint32_t (&b)[16], uint32_t (&c)[16], uint32_t (&d)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : B200MOE_RW8(a, 0), B200MOE_RW8(a, 8), B200MOE_RW8(b, 0), B200MOE_RW8(b, 8),
                 B200MOE_RW8(c, 0), B200MOE_RW8(c, 8), B200MOE_RW8(d, 0), B200MOE_RW8(d, 8)
               :
               : "memory");
}

// acc[16] += raw[16] * (sa[16] * sb) (GEMM1; `sa` in shared memory, the same address in all lanes) or raw * sb
template <int MODE>
__device__ __forceinline__ void promote16(float2* acc, const uint32_t (&r)[16], const float4* sa, float sb) {
  const float2 sb2 = make_float2(sb, sb);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    float2 s0 = sb2, s1 = sb2;
    if (MODE == 1) {
      const float4 s = sa[v];
      s0 = __fmul2_rn(make_float2(s.x, s.y), sb2);
      s1 = __fmul2_rn(make_float2(s.z, s.w), sb2);
    }
    acc[2 * v] = __ffma2_rn(make_float2(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1])), s0, acc[2 * v]);
    acc[2 * v + 1] =
        __ffma2_rn(make_float2(__uint_as_float(r[4 * v + 2]), __uint_as_float(r[4 * v + 3])), s1, acc[2 * v + 1]);
  }
}

// Transposes 8 values per lane within groups of 8 lanes: on return v[i] of lane l holds what lane (l & ~7) + i held in
// v[l & 7] (three butterfly rounds of four shuffles).
__device__ __forceinline__ void transpose8(float (&v)[8], int lane) {
#pragma unroll
  for (int d = 1; d < 8; d <<= 1) {
    const bool upper = (lane & d) != 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i & d) continue;
      const float send = upper ? v[i] : v[i | d];
      const float got = __shfl_xor_sync(0xffffffffu, send, d);
      if (upper) v[i] = got;
      else v[i | d] = got;
    }
  }
}

// The token box and the MMA's N for a tile of `rows` real rows: 16, 32 or 64 (log2 - 4 picks the tensor map).
__device__ __forceinline__ int n_class(int rows) { return rows <= 16 ? 0 : rows <= 32 ? 1 : 2; }

// PROF (B200MOE_PROF=1): CTA 0's cycle counters, g.prof[0 .. 8], and a 1 in g.prof[9] (the grouped kernels' differ).
template <int MODE, int NT, bool PROF>
__global__ void __launch_bounds__(SCfg<MODE, NT>::kThreads, 1)
stream_gemm_kernel(const __grid_constant__ StreamParams sp) {
  using Cfg = SCfg<MODE, NT>;
  constexpr int S = Cfg::kStages;
  constexpr uint32_t kProducers = Cfg::kProducers, kIssuers = Cfg::kIssuers;
  constexpr int G = kGroup;
  constexpr int kPromoWarps = Cfg::kPromoWarps;
  constexpr int H = Cfg::kHalves;
  constexpr int CH = NT / (16 * H);   // chunks of 16 token columns per promotion warp
  const GemmParams& p = sp.g;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  const float* ring = reinterpret_cast<const float*>(smem + S * Cfg::kStageBytes);         // [slot][G][NT]
  float* xch = reinterpret_cast<float*>(smem + S * Cfg::kStageBytes + Cfg::kRingBytes);    // [NT][64]
  float* panels = xch + Cfg::kXchBytes / 4;                              // [4 warps][K block][16] (rows in place)
  int* toks = reinterpret_cast<int*>(panels + Cfg::kPanelBytes);         // [M tile of the range][16] (rows in place)
  uint64_t* bars = reinterpret_cast<uint64_t*>(toks + Cfg::kToksBytes / 4);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = bar_full + 8 * S;
  const uint32_t bar_tfull = bar_empty + 8 * S;
  const uint32_t bar_tempty = bar_tfull + 8 * kAccs;
  const uint32_t bar_drain = bar_tempty + 8 * kAccs;   // 2
  const uint32_t bar_xready = bar_drain + 16;          // 4: u of an up warp is in shared memory
  const uint32_t bar_xfree = bar_xready + 32;          // 4: its gate warp has read it
  const uint32_t bar_split = bar_xfree + 32;           // 2: partial sums written; arrival order known
  const uint32_t bar_rq = bar_split + 16;              // 2: the item's activations stored; outcome of the arrival count known
  uint32_t* words = reinterpret_cast<uint32_t*>(bars + 2 * S + 2 * kAccs + 14);
  static_assert((2 * S + 2 * kAccs + 14) * 8 + 20 <= 512, "barrier area");
  uint32_t* tmem_slot = words;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(words + 1);   // [1] is never set: teardown waits ignore an abort
  volatile int* split_flag = reinterpret_cast<volatile int*>(words + 3);
  volatile int* rq_flag = reinterpret_cast<volatile int*>(words + 4);
  int2* table = reinterpret_cast<int2*>(reinterpret_cast<uint8_t*>(bars) + 512);   // (expert, real rows) of the CTA's M tiles

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < kAccs; ++b) {
      mbar_init(bar_tfull + 8 * b, 1);
      mbar_init(bar_tempty + 8 * b, kPromoWarps);
    }
    mbar_init(bar_drain, 1);
    mbar_init(bar_drain + 8, 1);
    for (int i = 0; i < 4; ++i) {
      mbar_init(bar_xready + 8 * i, 1);
      mbar_init(bar_xfree + 8 * i, 1);
    }
    mbar_init(bar_split, kPromoWarps);
    mbar_init(bar_split + 8, 1);
    mbar_init(bar_rq, kPromoWarps);
    mbar_init(bar_rq + 8, 1);
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    fence_mbar_init();
    tma_prefetch_desc(&p.tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), Cfg::kTmemCols);
    tmem_relinquish();
  }
  // Without a gather pass (decode calls that the one-block front kernel routed and placed) that front kernel itself is
  // in front of GEMM1: everything is read behind the wait, the token rows and their scales where the caller keeps them.
  const bool direct = MODE == 1 && NT == 16 && p.direct_a != 0;
  if (direct) {
    chain_wait();
    chain_release();
  }
  // Otherwise the tables of the placement kernels (scan) were complete before this kernel could become resident: the
  // kernel in front of it released its dependents behind its own wait.  So the range of this CTA and its first weight
  // boxes need no wait; everything else is read behind it.
  const int KB = p.kblocks, K = (KB + G - 1) / G;   // K blocks, and the groups that are the units of work
  const int box_kb = min(G, KB);                    // K blocks of a box (past the end of K they are filled with zeros)
  const int units = __ldcg(p.meta) * p.n_tiles * K;
  const int per_cta = stream_range(units, K, (int)gridDim.x);   // units of a CTA (the last ones may get none)
  const int u0 = min(units, (int)blockIdx.x * per_cta);
  const int u1 = min(units, u0 + per_cta);
  const int mt0 = u0 / (K * p.n_tiles);
  if (u0 < u1) {
    const int n_mt = min((u1 - 1) / (K * p.n_tiles) - mt0 + 1, kTileTable);
    if (direct)   // (entries past a tile's rows are -1)
      for (int i = threadIdx.x; i < n_mt * 16; i += Cfg::kThreads)
        toks[i] = __ldcg(p.row_token + (size_t)(mt0 + i / 16) * kTileM + i % 16);
    if ((int)threadIdx.x < n_mt) {
      const int mt = mt0 + threadIdx.x;
      const int e = __ldcg(p.tile_expert + mt);
      const int left = __ldcg(p.expert_count + e) - (mt * kTileM - __ldcg(sp.expert_row0 + e));
      table[threadIdx.x] = make_int2(e, min(left, NT));   // (an expert has no more rows than the call has tokens)
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // warps 1, 2: MMA issuers; 4 .. 3 + kPromoWarps: promotion; the others: producers
  const bool issuer = warp >= 1 && warp <= (int)kIssuers;
  const bool promo = warp >= 4 && warp < 4 + kPromoWarps;
  const uint32_t pme = warp == 0 ? 0u : (uint32_t)(warp < 4 ? warp - (int)kIssuers : warp - (int)kIssuers - kPromoWarps);
  const bool producer = !issuer && !promo;

  auto load_weights = [&](uint32_t s, int kg, int slab, int e) {   // the group's K blocks in one box
    const uint32_t dst = smem_base + s * Cfg::kStageBytes, full = bar_full + 8 * s;
    if (MODE == 1) tma_load_4d(dst, &p.tmap_b, 0, slab * 64, 2 * e, kg * G, full);   // 64 gate rows + 64 up rows
    else tma_load_3d(dst, &p.tmap_b, 0, e * p.n_per_expert + slab * kSlabRows, kg * G, full);
  };
  // bytes of a stage: boxes come whole, scales only for the K blocks that exist
  auto stage_bytes = [&](int n, int kg) {
    return (uint32_t)(box_kb * (kWBytes + n * kBlockK) + (MODE == 1 ? min(G, KB - kg * G) * n * 4 : 0));
  };

  uint32_t early = 0;   // groups of the range whose weight box is on its way before the wait
  if (producer && lane == 0 && u0 < u1 && !direct) {
    const int tile = u0 / K, kb0 = u0 - tile * K;
    const int2 info = table[0];
    const int n = 16 << n_class(info.y);
    early = min(min(K - kb0, u1 - u0), S);
    for (uint32_t j = pme; j < early; j += kProducers) {
      mbar_arrive_expect_tx(bar_full + 8 * j, stage_bytes(n, kb0 + (int)j));
      load_weights(j, kb0 + (int)j, tile % p.n_tiles, info.x);
    }
  }
  if (!direct) {
    chain_wait();
    chain_release();
  }
  if (MODE == 1 && p.zero_tokens > 0) {
    // no gather pass ran: the output rows that GEMM2 adds into are zeroed here, a few stores per CTA
    const int vec_per_row = p.hidden / 8;   // 8 bf16 = 16 bytes
    const long long total = (long long)p.zero_tokens * vec_per_row;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
      const long long t = i / vec_per_row;
      reinterpret_cast<uint4*>(p.out + t * p.out_stride)[i - t * vec_per_row] = make_uint4(0u, 0u, 0u, 0u);
    }
  }

  if (producer) {
    if (lane == 0) {
      // ------------------------------ TMA producers (groups in turn) ------------------------------
      // Activation scales: slot it % 16 is rewritten for group it once the MMAs of group it - S have
      // completed; those started after every promotion warp had released the accumulators of group it - S - 4, i.e.
      // was through with the scales of group it - S - 5.
      uint32_t it = 0;
      bool alive = true;
      long long t_wait = 0, t_issue = 0;
      const long long t_begin = PROF ? clock64() : 0;
      for (int u = u0; u < u1 && alive;) {
        const int tile = u / K, kb0 = u - tile * K;
        const int len = min(K - kb0, u1 - u);
        const int m_tile = tile / p.n_tiles, slab = tile - m_tile * p.n_tiles;
        const int2 info = table[m_tile - mt0];
        const int cls = n_class(info.y), n = 16 << cls;
        for (int kb = kb0; kb < kb0 + len; ++kb, ++it) {
          if ((it % kProducers) != pme) continue;
          const uint32_t s = it % S, ph = (it / S) & 1u, full = bar_full + 8 * s;
          const long long q0 = PROF ? clock64() : 0;
          long long q1 = q0;
          if (it >= early) {
            if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, p.status, 41)) { alive = false; break; }
            if (PROF) q1 = clock64();
            mbar_arrive_expect_tx(full, direct ? (uint32_t)(box_kb * kWBytes + min(G, KB - kb * G) * info.y * kBlockK)
                                               : stage_bytes(n, kb));
            load_weights(s, kb, slab, info.x);
          }
          const uint32_t tok_dst = smem_base + s * Cfg::kStageBytes + G * kWBytes;
          const int kb_end = min(kb * G + G, KB);
          if (direct) {   // one one-row box per row and K block; past the tile's rows the stage keeps what it held, as padding rows do
            for (int x = kb * G; x < kb_end; ++x)
              for (int j = 0; j < info.y; ++j)
                tma_load_2d(tok_dst + (x - kb * G) * Cfg::kTokBytes + j * kBlockK, &p.tmap_a, x * kBlockK,
                            toks[(m_tile - mt0) * 16 + j], full);
          } else {
            // n rows of each of the group's K blocks, the K blocks n x 128 bytes apart
            tma_load_3d(tok_dst, &sp.tmap_tok[cls], 0, m_tile * kTileM, kb * G, full);
            if (MODE == 1)
              for (int x = kb * G; x < kb_end; ++x)
                bulk_load(smem_u32(ring) + ((it % kScaleSlots) * G + (x - kb * G)) * (NT * 4),
                          p.a_scale + (size_t)x * p.m_cap + (size_t)m_tile * kTileM, n * 4, full);
          }
          if (PROF) {
            t_wait += q1 - q0;
            t_issue += clock64() - q1;
          }
        }
        u += len;
      }
      if (PROF && p.prof && blockIdx.x == 0 && pme == 0) {
        p.prof[0] = (unsigned long long)t_wait;                    // producer 0 waiting for a free stage
        p.prof[1] = (unsigned long long)t_issue;                   // producer 0 issuing copies
        p.prof[2] = (unsigned long long)(clock64() - t_begin);     // producer 0: whole loop
        p.prof[3] = (unsigned long long)it;                        // K groups of the CTA
      }
      // copies still in flight must land before the CTA's shared memory is released
      const uint32_t first = it > (uint32_t)S ? it - S : 0u;
      for (uint32_t j = first; j < it; ++j)
        if ((j % kProducers) == pme) (void)mbar_wait(bar_full + 8 * (j % S), (j / S) & 1u, abort_flag + 1, p.status, 46);
    }
  } else if (issuer) {
    if (lane == 0) {
      // ------------------------------ MMA issuers (two take alternate groups) ------------------------------
      const uint32_t me = (uint32_t)(warp - 1);
      uint32_t it = 0;
      bool alive = true;
      long long t_acc = 0, t_tma = 0, t_issue = 0;
      for (int u = u0; u < u1 && alive;) {
        const int tile = u / K, kb0 = u - tile * K;
        const int len = min(K - kb0, u1 - u);
        const int n = 16 << n_class(table[tile / p.n_tiles - mt0].y);
        const uint32_t idesc = make_idesc_e4m3(kSlabRows, n);
        const uint32_t tok_step = direct ? Cfg::kTokBytes : n * kBlockK;   // from one K block's token rows to the next's
        for (int kb = 0; kb < len; ++kb, ++it) {
          if ((it % kIssuers) != me) continue;
          const uint32_t s = it % S, ph = (it / S) & 1u;
          const uint32_t b = it % kAccs, bph = (it / kAccs) & 1u;
          const long long q0 = PROF ? clock64() : 0;
          if (!mbar_wait(bar_tempty + 8 * b, bph ^ 1u, abort_flag, p.status, 42)) { alive = false; break; }
          const long long q1 = PROF ? clock64() : 0;
          if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, p.status, 43)) { alive = false; break; }
          const long long q2 = PROF ? clock64() : 0;
          tc_fence_after();
          const uint32_t w_addr = smem_base + s * Cfg::kStageBytes;
          for (int g = 0; g < G && (kb0 + kb) * G + g < KB; ++g)
            tc_mma_f8_kblock(tmem_base + (b * G + g) * NT, kmajor_sw128_desc_lo(w_addr + g * kWBytes),
                             kmajor_sw128_desc_lo(w_addr + G * kWBytes + g * tok_step), kKmajorSw128DescHi, idesc);
          tc_commit(bar_empty + 8 * s);
          tc_commit(bar_tfull + 8 * b);
          if (PROF) {
            t_acc += q1 - q0;
            t_tma += q2 - q1;
            t_issue += clock64() - q2;
          }
        }
        u += len;
      }
      tc_commit(bar_drain + 8 * me);
      (void)mbar_wait(bar_drain + 8 * me, 0u, abort_flag + 1, p.status, 45);
      if (PROF && p.prof && blockIdx.x == 0 && me == 0) {
        p.prof[4] = (unsigned long long)t_acc;     // issuer 0 waiting for a free accumulator
        p.prof[5] = (unsigned long long)t_tma;     // issuer 0 waiting for operands
        p.prof[6] = (unsigned long long)t_issue;   // issuer 0 issuing MMAs and commits
      }
    }
  } else {
    // ------------------------------ promotion + epilogue ------------------------------
    const int q = warp & 3;              // TMEM lane quarter: weight rows 32q .. 32q+31 of the slab
    const int h = (warp - 4) >> 2;       // takes the token chunks h, h + H, ...
    float* panel = panels + (warp - 4) * (Cfg::kPanelBytes / 4);   // (rows in place)
    uint32_t it = 0, xi = 0, si = 0, ri = 0;
    bool alive = true;
    long long t_wait = 0;
    const long long t_begin = PROF ? clock64() : 0;
    const int nblk_per_expert = p.n_per_expert / kBlockK;
    // weight scales of a tile, two per lane (K block lane and lane + 32)
    auto load_sb = [&](int tile, float& lo, float& hi) {
      const int m_tile = tile / p.n_tiles, slab = tile - m_tile * p.n_tiles;
      const int wblock = MODE == 1 ? (q < 2 ? (slab * 64) / kBlockK : (p.inter + slab * 64) / kBlockK) : slab;
      const float* sb = p.b_scale + ((size_t)table[m_tile - mt0].x * nblk_per_expert + wblock) * KB;
      lo = lane < KB ? __ldg(sb + lane) : 0.f;
      hi = lane + 32 < KB ? __ldg(sb + lane + 32) : 0.f;
    };
    float sb_lo = 0.f, sb_hi = 0.f;
    if (u0 < u1) load_sb(u0 / K, sb_lo, sb_hi);
    for (int u = u0; u < u1 && alive;) {
      const int tile = u / K, kb0 = u - tile * K;
      const int len = min(K - kb0, u1 - u);
      const int m_tile = tile / p.n_tiles, slab = tile - m_tile * p.n_tiles;
      const int cnt = table[m_tile - mt0].y;
      const int n = 16 << n_class(cnt);
      const int row0 = m_tile * kTileM;
      u += len;
      float nx_lo = 0.f, nx_hi = 0.f;   // the next tile's weight scales arrive under this one's K loop
      if (u < u1) load_sb(tile + 1, nx_lo, nx_hi);
      float2 acc[CH * 8];
#pragma unroll
      for (int j = 0; j < CH * 8; ++j) acc[j] = make_float2(0.f, 0.f);
      if (direct) {   // the token scales where the caller keeps them; lane l reads row l % 16's
        const int t = toks[(m_tile - mt0) * 16 + (lane & 15)];
        __syncwarp();
        for (int x = kb0 * G + lane / 16; x < min((kb0 + len) * G, KB); x += 2)
          panel[x * 16 + (lane & 15)] = t >= 0 ? p.hscale[(size_t)t * p.hs_stride_t + (size_t)x * p.hs_stride_kb] : 0.f;
        __syncwarp();
      }

      for (int kg = kb0; kg < kb0 + len; ++kg, ++it) {
        const uint32_t b = it % kAccs, bph = (it / kAccs) & 1u;
        const int kb = kg * G;                      // even, so both K blocks' scales lie in the same half of the lanes
        const bool two = kb + 1 < KB;               // the last group of an odd K has one K block
        const float sb_half = kb < 32 ? sb_lo : sb_hi;
        const float sb0 = __shfl_sync(0xffffffffu, sb_half, kb & 31), sb1 = __shfl_sync(0xffffffffu, sb_half, (kb + 1) & 31);
        const long long q0 = PROF ? clock64() : 0;
        bool ok = mbar_wait(bar_tfull + 8 * b, bph, abort_flag, p.status, 44);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { alive = false; break; }
        tc_fence_after();
        if (PROF) t_wait += clock64() - q0;
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + b * (G * NT) + h * 16;
        const float4* sa = reinterpret_cast<const float4*>(ring + (it % kScaleSlots) * (G * NT) + h * 16);   // GEMM1
        if constexpr (NT == 16) {
          if (direct) sa = reinterpret_cast<const float4*>(panel + kb * 16);
          uint32_t r0[16], r1[16];
          tmem_ld_16(t_row, r0);
          if (two) tmem_ld_16(t_row + NT, r1);
          tmem_wait_on(r0, r1);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_tempty + 8 * b);
          promote16<MODE>(acc, r0, sa, sb0);
          if (two) promote16<MODE>(acc, r1, sa + NT / 4, sb1);
        } else {
          // my chunks: the tile's token columns [16 h, + 16) and [32 + 16 h, + 16) of both K blocks
          const bool has0 = 16 * h < n, has1 = 32 + 16 * h < n;
          uint32_t r00[16], r01[16], r10[16], r11[16];
          if (has0) tmem_ld_16(t_row, r00);
          if (has1) tmem_ld_16(t_row + 32, r01);
          if (has0 && two) tmem_ld_16(t_row + NT, r10);
          if (has1 && two) tmem_ld_16(t_row + NT + 32, r11);
          tmem_wait_on(r00, r01, r10, r11);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_tempty + 8 * b);   // everything this warp needs is in registers
          if (has0) promote16<MODE>(acc, r00, sa, sb0);
          if (has1) promote16<MODE>(acc + 8, r01, sa + 8, sb0);
          if (has0 && two) promote16<MODE>(acc, r10, sa + NT / 4, sb1);
          if (has1 && two) promote16<MODE>(acc + 8, r11, sa + NT / 4 + 8, sb1);
        }
      }
      if (!alive) break;
      sb_lo = nx_lo;
      sb_hi = nx_hi;

      if (len < K) {
        // the tile's range is cut: partial sums to scratch, the CTA that arrives last adds them in range order
        const int c_first = (tile * K) / per_cta, c_last = (tile * K + K - 1) / per_cta;
        // a CTA has at most two cut tiles: slot 0 for one that an earlier CTA began, slot 1 for one that it begins
        float* scr = p.splitk_scratch + (size_t)(2 * blockIdx.x + (kb0 == 0 ? 1 : 0)) * NT * kSlabRows + q * 32 + lane;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
          const int t0 = 16 * (H * c + h);
          if (t0 < n) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              scr[(t0 + 2 * j) * kSlabRows] = acc[8 * c + j].x;
              scr[(t0 + 2 * j + 1) * kSlabRows] = acc[8 * c + j].y;
            }
          }
        }
        __threadfence();
        __syncwarp();
        const uint32_t sph = si & 1u;
        ++si;
        if (lane == 0) mbar_arrive(bar_split);
        bool oks = mbar_wait(bar_split, sph, abort_flag, p.status, 49);
        oks = __all_sync(0xffffffffu, oks);
        if (!oks) { alive = false; break; }
        if (warp == 4 && lane == 0) {
          __threadfence();   // the other warps' pieces (ordered before this point by the barrier) before the count
          const int prev = atomicAdd(p.splitk_count + c_first, 1);
          if (prev == c_last - c_first) p.splitk_count[c_first] = 0;   // every piece has arrived: leave the counter clean
          *split_flag = prev;
          mbar_arrive(bar_split + 8);
        }
        oks = mbar_wait(bar_split + 8, sph, abort_flag, p.status, 50);
        oks = __all_sync(0xffffffffu, oks);
        if (!oks) { alive = false; break; }
        const int prev = *split_flag;
        if (prev != c_last - c_first) continue;   // another CTA finishes this tile
        __threadfence();
#pragma unroll
        for (int j = 0; j < CH * 8; ++j) acc[j] = make_float2(0.f, 0.f);
        for (int k = c_first; k <= c_last; ++k) {
          const float* src = p.splitk_scratch + (size_t)(2 * k + (k == c_first ? 1 : 0)) * NT * kSlabRows + q * 32 + lane;
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            const int t0 = 16 * (H * c + h);
            if (t0 < n) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                acc[8 * c + j].x += __ldcg(src + (t0 + 2 * j) * kSlabRows);
                acc[8 * c + j].y += __ldcg(src + (t0 + 2 * j + 1) * kSlabRows);
              }
            }
          }
        }
      }

      if (MODE == 1) {
        // lanes 0-63 hold g and lanes 64-127 hold u of the same 64 columns: the up warps hand u over through shared
        // memory ([token][row]: lanes hit consecutive banks), the gate warps store g * silu(u) and the row maxima
        const int pr = (q & 1) + 2 * h;
        float* x0 = xch + (q & 1) * 32 + lane;
        const uint32_t xph = xi & 1u;
        ++xi;
        if (q >= 2) {
          bool okx = mbar_wait(bar_xfree + 8 * pr, xph ^ 1u, abort_flag, p.status, 47);
          okx = __all_sync(0xffffffffu, okx);
          if (!okx) { alive = false; break; }
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            const int t0 = 16 * (H * c + h);
            if (t0 < cnt) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                x0[(t0 + 2 * j) * 64] = acc[8 * c + j].x;
                x0[(t0 + 2 * j + 1) * 64] = acc[8 * c + j].y;
              }
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_xready + 8 * pr);
        } else {
          bool okx = mbar_wait(bar_xready + 8 * pr, xph, abort_flag, p.status, 48);
          okx = __all_sync(0xffffffffu, okx);
          if (!okx) { alive = false; break; }
          __half* dst = p.act + (size_t)row0 * p.inter + slab * 64 + q * 32 + lane;
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            const int t0 = 16 * (H * c + h);
            if (t0 < cnt) {
              uint32_t mx = 0;   // lane t keeps the maximum of the chunk's row t
#pragma unroll
              for (int t = 0; t < 16; ++t) {
                if (t0 + t < cnt) {
                  const float g = (t & 1) ? acc[8 * c + t / 2].y : acc[8 * c + t / 2].x;
                  const __half hv = __float2half_rn(silu_mul(g, x0[(t0 + t) * 64]));
                  dst[(size_t)(t0 + t) * p.inter] = hv;
                  const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(__half2float(hv))));
                  if (lane == t) mx = m;
                }
              }
              if (lane < 16 && t0 + lane < cnt) atomicMax(p.row_amax + row0 + t0 + lane, mx);
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_xfree + 8 * pr);
        }
        if (p.tile_done) {
          // Requantisation inside this kernel (decode calls): an expert's weight slabs count their arrivals, and the CTA
          // that stores the last one finds all of the expert's (at most NT) activation rows and their final maxima in L2
          // and turns them into e4m3 codes with one scale per row (max|act| / 448, solution/python/moe_fused.cu:175-195
          // of the reference).
          const uint32_t rph = ri & 1u;
          ++ri;
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_rq);            // this warp's stores and row maxima are issued
          if (warp == 4) {
            bool okr = mbar_wait(bar_rq, rph, abort_flag, p.status, 51);
            okr = __all_sync(0xffffffffu, okr);
            if (!okr) { alive = false; break; }
            if (lane == 0) {
              __threadfence();   // the warps' stores (ordered before this point by the barrier) before the count
              const int prev = atomicAdd(p.tile_done + m_tile, 1);
              *rq_flag = prev == p.n_tiles - 1 ? 1 : 0;
              mbar_arrive(bar_rq + 8);
            }
          }
          bool okq = mbar_wait(bar_rq + 8, rph, abort_flag, p.status, 52);
          okq = __all_sync(0xffffffffu, okq);
          if (!okq) { alive = false; break; }
          if (*rq_flag) {
            __threadfence();
            const int tid = threadIdx.x - 128;
            const int vecs = p.inter / 8;              // 8 halves = 16 bytes in, 8 bytes out
            for (int j = 0; j < cnt; ++j) {
              const int m = row0 + j;
              const float amax = fmaxf(__uint_as_float(__ldcg(p.row_amax + m)), 1e-8f);
              const float sc = fmaxf(amax / 448.0f, 1e-8f), inv = 1.0f / sc;
              if (tid == 0) p.row_scale_out[m] = sc;
              const uint4* src = reinterpret_cast<const uint4*>(p.act + (size_t)m * p.inter);
              uint2* dstq = reinterpret_cast<uint2*>(p.act_q_out + (size_t)m * p.inter);
              for (int v = tid; v < vecs; v += 32 * kPromoWarps) {
                const uint4 raw = __ldcg(src + v);
                dstq[v] = requant8(raw, sc, inv);
              }
            }
          }
        }
      } else {
        // A lane's eight token values of one output column become eight columns of one token: 16 bytes per
        // red.global.add instead of 2.
        __nv_bfloat16* dst = p.out + slab * kSlabRows + q * 32 + (lane & 24);
#pragma unroll
        for (int g8 = 0; g8 < CH * 2; ++g8) {
          const int t0 = 16 * (H * (g8 / 2) + h) + 8 * (g8 & 1);
          if (t0 < cnt) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[2 * j] = acc[4 * g8 + j].x;
              v[2 * j + 1] = acc[4 * g8 + j].y;
            }
            transpose8(v, lane);
            const int t = t0 + (lane & 7);
            if (t < cnt) {
              // the three loads together: behind the check of the token the other two would wait for it
              const int tok = p.row_token[row0 + t];
              const float rs = p.row_scale[row0 + t] * p.row_weight[row0 + t];
              uint32_t wv[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                __nv_bfloat162 b2 = __floats2bfloat162_rn(v[2 * j] * rs, v[2 * j + 1] * rs);
                wv[j] = *reinterpret_cast<uint32_t*>(&b2);
              }
              if (tok >= 0) red_add_bf16x8(dst + (size_t)tok * p.out_stride, wv[0], wv[1], wv[2], wv[3]);
            }
          }
        }
      }
    }
    if (PROF && p.prof && blockIdx.x == 0 && warp == 4 && lane == 0) {
      p.prof[7] = (unsigned long long)t_wait;                  // promotion warp 0 waiting for an accumulator
      p.prof[8] = (unsigned long long)(clock64() - t_begin);   // promotion warp 0: whole role
      p.prof[9] = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::kTmemCols);
  if (threadIdx.x == 0 && abort_flag[0] && p.status_mirror) {
    // a wait of this CTA ran out: let the host see the status word without a copy of its own
    p.status_mirror[1] = p.status[kStatusDetail];
    p.status_mirror[0] = p.status[kStatusCode];
    __threadfence_system();
  }
}

template <int MODE, int NT>
cudaError_t launch_one(const StreamParams& p, int grid, cudaStream_t stream) {
  using Cfg = SCfg<MODE, NT>;
  return launch_chained(p.g.prof ? stream_gemm_kernel<MODE, NT, true> : stream_gemm_kernel<MODE, NT, false>, dim3(grid),
                        dim3(Cfg::kThreads), Cfg::kSmemBytes, stream, p);
}

template <int MODE, int NT>
cudaError_t configure_one() {
  const cudaError_t e = cudaFuncSetAttribute(stream_gemm_kernel<MODE, NT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             SCfg<MODE, NT>::kSmemBytes);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(stream_gemm_kernel<MODE, NT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              SCfg<MODE, NT>::kSmemBytes);
}

}  // namespace

cudaError_t configure_stream_gemm() {
  cudaError_t e;
  if ((e = configure_one<1, 16>()) != cudaSuccess) return e;
  if ((e = configure_one<2, 16>()) != cudaSuccess) return e;
  if ((e = configure_one<1, 64>()) != cudaSuccess) return e;
  return configure_one<2, 64>();
}

bool stream_gemm_fits(int kblocks, int max_tiles, int num_sms) {
  const int grid = num_sms < kStreamMaxCtas ? num_sms : kStreamMaxCtas;
  // a lane keeps two weight scales; a CTA's range covers a contiguous part of at most max_tiles M tiles
  return kblocks <= kMaxKBlocks && max_tiles / grid + 2 <= kTileTable;
}

cudaError_t launch_stream_gemm(int mode, int nt, const StreamParams& p, int max_tiles, int num_sms, cudaStream_t stream) {
  const int grid = num_sms < kStreamMaxCtas ? num_sms : kStreamMaxCtas;
  if (!stream_gemm_fits(p.g.kblocks, max_tiles, num_sms)) return cudaErrorInvalidValue;
  switch (nt) {
    case 16: return mode == 1 ? launch_one<1, 16>(p, grid, stream) : launch_one<2, 16>(p, grid, stream);
    case 64: return mode == 1 ? launch_one<1, 64>(p, grid, stream) : launch_one<2, 64>(p, grid, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace b200moe
