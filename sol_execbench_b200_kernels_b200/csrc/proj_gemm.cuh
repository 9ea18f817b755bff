// Input projection of the Mamba mixer (problem 029):
//   projected[M, N] = bf16( hidden[M, K] . weight[N, K]^T + bias[N] ),  all operands bf16, fp32 accumulation,
// one rounding at the end (the reference's CUTLASS builder GEMM with a row-broadcast bias in the epilogue:
// kernels/029_mamba_conv1d_with_gating/kernel.cu:36-160, launched from kernel.cu:274-312).
//
// A persistent tcgen05 kernel, kind::f16 with bf16 operands.  The accumulator of a tile stays in TMEM over the whole
// K loop (nothing has to pass through registers per K block here, unlike the block-scaled FP8 kernels), TMEM holds
// two 256-column accumulators, and the epilogue of a tile runs on its own warps while the next tile's MMAs fill the
// other accumulator.
//
//   kPair = true   two CTAs on neighbouring SMs own a 256-row x 256-column tile: each stages its own 128 rows of
//                  `hidden` and HALF of the 256 weight rows of a K block (32 KiB per CTA and 64-wide K block), the
//                  even CTA issues cta_group::2 MMAs (M = 256, N = 256, K = 16) for both; each CTA finds its
//                  128 x 256 fp32 accumulator in its own TMEM.  Used for M > 128.
//   kPair = false  one CTA owns a 128-row x tile_n-column tile (tile_n <= 256) and stages all its weight rows.  Used
//                  for M <= 128, where the second CTA of a pair would have no rows.  That launch is bound by how fast
//                  the SMs pull the weights from HBM, so the host picks the narrowest tile (a multiple of 32 columns)
//                  with which one round of tiles still covers N, and the ring takes the whole shared memory: the
//                  staging tiles then lie in the ring, idle once a CTA's only tile has been accumulated.  At M = 128,
//                  K = 8192, N = 32768: 147 CTAs with 224 columns and 5 stages instead of 128 with 256 and 4.
//
// Warp roles (192 threads): warp 0 TMA producer, warp 1 TMEM allocation and (in the even CTA) MMA issue, warps 2-5
// epilogue: a warp reads TMEM lanes 32 (w % 4) .. +31 in chunks of 64 columns, adds the bias in fp32, rounds to bf16
// into one of two 16 KiB staging tiles (128-byte rows, 16-byte chunks swizzled by the row) and one thread issues the
// TMA store of the chunk, so the store of a chunk overlaps the conversion of the next.
//
// Every wait is on a barrier of the waiting CTA and is bounded; the other CTA of a pair reaches it with
// shared::cluster addresses (remote mbarrier.arrive, TMA completion bytes, tcgen05.commit).  No multicast form.
#pragma once

#include "mamba_conv.cuh"

namespace so {

using namespace gu;

constexpr int kPjThreads = 192;
constexpr int kPjTileM = 128;                 // rows per CTA
constexpr int kPjTileN = 256;                 // columns per tile
constexpr int kPjBlockK = 64;                 // bf16 per K block: one 128-byte swizzle span
constexpr uint32_t kPjATileBytes = kPjTileM * 128;
constexpr uint32_t kPjOutChunkBytes = kPjTileM * 128;   // 128 rows x 64 bf16
constexpr uint32_t kPjOutBytes = 2 * kPjOutChunkBytes;
constexpr uint32_t kPjTmemCols = 512;         // two 256-column fp32 accumulators

constexpr int kPjMaxStages = 8;
constexpr uint32_t kPjFixedBytes = 256 /*barriers*/ + 1024 /*alignment*/;

template <bool kPair>
struct PjCfg {
  static constexpr int pair_b_rows = 128;  // weight rows each CTA of a pair stages per K block
  static constexpr int pair_stages = 6;
  static constexpr int rows_per_tile = kPair ? 2 * kPjTileM : kPjTileM;
  __host__ __device__ static constexpr uint32_t stage_bytes(int b_rows) {
    return kPjATileBytes + static_cast<uint32_t>(b_rows) * 128;
  }
  static constexpr uint32_t pair_smem_bytes = pair_stages * (kPjATileBytes + pair_b_rows * 128) + kPjOutBytes + kPjFixedBytes;
};

enum : unsigned { kWaitPjSlot = 40, kWaitPjFull = 41, kWaitPjAccFree = 42, kWaitPjAccFull = 43 };
// sites of the range-checked debug build (-DGU_BOUNDS=1, see GU_IN_RANGE)
enum : unsigned { kSitePjLoad = 49, kSitePjStage = 50, kSitePjStore = 51, kSitePjBias = 52, kSitePjTile = 53,
                  kSitePjConv = 54 };

struct ProjParams {
  const __nv_bfloat16* bias;  // [N]
  __nv_bfloat16* out;         // [M, N] (lone CTAs: a last chunk of 32 columns is stored without TMA)
  int m, n, kb;               // kb = ceil(K / 64)
  int m_tiles, n_tiles, num_tiles;
  int group_m;                // raster: tiles walk `group_m` row tiles at a time, row tile fastest
  int tile_n, stages;         // lone CTAs: columns per tile (a multiple of 32, at most 256) and ring depth
  int staging_in_ring;        // lone CTAs: no CTA has a second tile, so the staging tiles may lie in the idle ring
};

// The convolution tail in the epilogue (CTA pairs only): the first `channels` columns are not stored as they are but masked,
// convolved along the sequence, gated and written transposed.
//
// What it saves is the round trip of half of the projection through HBM and most of a launch (the tail by itself takes
// 37.8 us at 2 x 1000 tokens).  The arithmetic is the tail's, some 5000 issue slots per warp and 256-column tile, and hides
// behind the next tile's 65 000 cycles of MMAs; column tiles run in ascending order, so the tiles at the end of a group of
// row tiles, which nothing hides, are gate tiles.  (Not so with one round of tiles: 1 x 128 tokens on lone CTAs took 104 us
// this way and takes 99 with the tail behind.)  A lane holds one token row of 64 channels, so the taps at l-1, l-2, l-3 are
// its neighbours' values (shuffles; the three lanes at a warp's edge read what the warp above left in shared memory), and
// a channel's 32 positions are one 64-byte store per warp, whatever the alignment of the rows.  The first three rows of a
// CTA's 128 need rows of another CTA: those outputs are left to mamba_conv1d_edges_kernel, and the three rows on either
// side of each edge are stored into `projected` for it.  (Overlapping the row blocks by three instead would add a block
// in 42, a whole round of tiles at some sizes.)
struct ConvParams {
  const uint16_t* mask;          // [M] bf16 bits
  const __nv_bfloat16* weight;   // [channels, 4]
  const __nv_bfloat16* bias;     // [channels]
  uint16_t* out;                 // [batch, channels, sequence] bf16 bits
  int sequence, channels;
};

// Instruction descriptor, kind::f16: D fp32 (bits 4-5 = 1), A and B bf16 (format 1 at bits 7-9 and 10-12), both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t umma_idesc_bf16_f32(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
template <bool kPair>
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  if constexpr (kPair) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
__device__ __forceinline__ void tma_store_wait_read1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }

// One lane of a converged warp polls; every lane gets the outcome.
__device__ __forceinline__ bool pj_wait_elected(WaitCtx& ctx, bool elected, uint32_t bar, uint32_t parity, unsigned code) {
  bool ok = true;
  if (elected) ok = mbar_wait(ctx, bar, parity, code);
  ok = __all_sync(0xffffffffu, ok);
  __syncwarp();
  return ok;
}

__device__ __forceinline__ void pj_tile_coords(const ProjParams& p, int tile, int& tm, int& tn) {
  const int per_group = p.group_m * p.n_tiles;
  const int group = tile / per_group;
  const int first = group * p.group_m;
  const int rows = min(p.group_m, p.m_tiles - first);
  const int within = tile - group * per_group;
  tm = first + within % rows;
  tn = within / rows;
}

// What a chunk of 64 channels leaves in shared memory (in its staging tile, which it does not use otherwise):
constexpr uint32_t kConvHaloBytes = 4 * 3 * 128;  // [warp][row 29, 30, 31][64 channels]: masked rows for the warp below
constexpr uint32_t kConvTapBytes = 32 * 16;       // [channel pair] taps, then [channel pair] bias (4 bytes)

// One token row of 32 channels (16 packed words `x`, masked) -> 32 outputs.  `halo`: these channels of the three rows above
// this warp's first, 128 bytes per row; `taps` / `biases`: of these channels; `hist`: rows of history that the lane's
// position has, at most 3.
__device__ __forceinline__ void conv_row_32(long long sequence, const uint32_t (&x)[16], const uint8_t* halo, const uint4* taps,
                                            const uint4* biases, int lane, int hist, bool keep, bool store, uint16_t* dst) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {  // 4 words = 8 channels
    const uint4 bq = biases[g];
    const uint32_t bias[4] = {bq.x, bq.y, bq.z, bq.w};
    uint32_t prev[3][4];  // [k - 1]: the values k positions back
#pragma unroll
    for (int k = 1; k <= 3; ++k) {
      uint4 edge = make_uint4(0u, 0u, 0u, 0u);
      if (lane < k) edge = *reinterpret_cast<const uint4*>(halo + (3 + lane - k) * 128 + 16 * g);
      const uint32_t e[4] = {edge.x, edge.y, edge.z, edge.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, x[4 * g + i], k);
        prev[k - 1][i] = hist >= k ? (lane < k ? e[i] : up) : 0u;
      }
    }
    uint32_t conv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 w[4];
      unpack_taps(taps[4 * g + i], w);
      conv[i] = conv_pair(bf16x2_to_float2(prev[2][i]), bf16x2_to_float2(prev[1][i]), bf16x2_to_float2(prev[0][i]),
                          bf16x2_to_float2(x[4 * g + i]), w, bf16x2_to_float2(bias[i]));
    }
    __nv_bfloat162 lowest = *reinterpret_cast<const __nv_bfloat162*>(&conv[0]);
#pragma unroll
    for (int i = 1; i < 4; ++i) lowest = __hmin2_nan(lowest, *reinterpret_cast<const __nv_bfloat162*>(&conv[i]));
    const bool small = __hbge2(lowest, __floats2bfloat162_rn(-20.f, -20.f));
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      uint32_t r[2];
      silu_2x2(conv[i], conv[i + 1], small, r[0], r[1]);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!keep) r[h] = 0u;
        if (store) {
          __stcs(reinterpret_cast<unsigned short*>(dst), static_cast<unsigned short>(r[h]));
          __stcs(reinterpret_cast<unsigned short*>(dst + sequence), static_cast<unsigned short>(r[h] >> 16));
        }
        dst += 2 * sequence;
      }
    }
  }
}

template <bool kPair, bool kConv>
__device__ __forceinline__ void proj_gemm_body(const CUtensorMap& tm_a, const CUtensorMap& tm_w, const CUtensorMap& tm_out,
                                               const ProjParams& p, const ConvParams* cv) {
  using Cfg = PjCfg<kPair>;
  extern __shared__ uint8_t smem_raw[];
  // operand tiles need 1024-byte alignment for the 128-byte swizzle pattern; both CTAs of a pair get the same offsets
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

  const uint32_t stages = kPair ? Cfg::pair_stages : p.stages;
  const int tile_n = kPair ? kPjTileN : p.tile_n;
  const int b_rows = kPair ? Cfg::pair_b_rows : p.tile_n;  // weight rows this CTA stages per K block
  const uint32_t stage_bytes = Cfg::stage_bytes(b_rows);
  const uint32_t ring = smem_base;
  const bool in_ring = !kPair && p.staging_in_ring;
  const uint32_t stag = in_ring ? ring : ring + stages * stage_bytes;
  const uint32_t bars = ring + stages * stage_bytes + (in_ring ? 0u : kPjOutBytes);
  const uint32_t bar_full = bars;                             // [stages] pair: the even CTA's, 2 arrivals + both CTAs' bytes
  const uint32_t bar_empty = bar_full + 8 * kPjMaxStages;      // [stages] one commit: the slot's MMAs have read it
  const uint32_t bar_acc_full = bar_empty + 8 * kPjMaxStages;  // [2] one commit: the tile's accumulator is complete
  const uint32_t bar_acc_free = bar_acc_full + 16;            // [2] pair: the even CTA's; 4 epilogue warps per CTA
  const uint32_t tmem_slot = bar_acc_free + 16;
  const uint32_t abort_slot = tmem_slot + 4;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - smem_base));
  volatile int* abort_gen = reinterpret_cast<volatile int*>(smem_gen + (abort_slot - smem_base));

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = kPair ? cluster_ctarank() : 0u;
  const int unit = kPair ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int units = kPair ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);

  if (threadIdx.x == 0) {
    pdl_trigger();
    for (uint32_t s = 0; s < stages; ++s) {
      mbar_init(bar_full + 8 * s, kPair ? 2 : 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int q = 0; q < 2; ++q) {
      mbar_init(bar_acc_full + 8 * q, 1);
      mbar_init(bar_acc_free + 8 * q, kPair ? 8 : 4);
    }
    *abort_gen = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_out);
  }
  if (warp == 1) {
    if constexpr (kPair) {
      tmem_alloc_pair(tmem_slot, kPjTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, kPjTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  if constexpr (kPair) cluster_sync_all();  // barriers and the abort flag of both CTAs exist before anything reaches across
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_gen;
  if (warp == 0 && lane == 0 && unit < p.num_tiles) {
    // the first tile's first weights on their way into L2 while the kernel in front drains
    int tm, tn;
    pj_tile_coords(p, unit, tm, tn);
    const int wrow = tn * tile_n + static_cast<int>(rank) * b_rows;
    for (int j = 0; j < min(static_cast<int>(stages), p.kb); ++j)
      if (wrow < p.n && GU_IN_RANGE(wrow >= 0 && ((j * kPjBlockK * 2) & 15) == 0, kSitePjLoad))
        tma_prefetch_2d(&tm_w, j * kPjBlockK, wrow);
  }
  pdl_wait();

  WaitCtx ctx{abort_slot, false, kPair};

  if (warp == 0) {
    // ---------------- TMA producer: the whole warp walks the loop, one elected lane waits and issues ----------------
    const bool elected = elect_one() != 0u;
    const uint32_t full_base = kPair ? mapa_shared(bar_full, 0) : bar_full;
    const uint64_t read_once = l2_policy_evict_first();
    (void)read_once;
    uint32_t slots = 0;  // ring slots filled so far: stage = low part, barrier phase = the next bit
    for (int tile = unit; tile < p.num_tiles; tile += units) {
      int tm, tn;
      pj_tile_coords(p, tile, tm, tn);
      const int row0 = tm * Cfg::rows_per_tile + static_cast<int>(rank) * kPjTileM;
      const int wrow0 = tn * tile_n + static_cast<int>(rank) * b_rows;  // (rank is 0 without pairs)
      for (int j = 0; j < p.kb; ++j, ++slots) {
        const uint32_t stage = slots % stages, phase = (slots / stages) & 1u;
        const bool ok = pj_wait_elected(ctx, elected, bar_empty + 8 * stage, phase ^ 1u, kWaitPjSlot);
        const uint32_t full = full_base + 8 * stage;
        const uint32_t dst = ring + stage * stage_bytes;
        // (loads may start past the last row of a ragged tile, where they read zeros, but never before row 0, past the
        // padded row range, or at a K offset that is not 16-byte aligned)
        if (ok && elected && GU_IN_RANGE(stage < stages && stages <= kPjMaxStages, kSitePjStage) &&
            GU_IN_RANGE(tm >= 0 && tm < p.m_tiles && tn >= 0 && tn < p.n_tiles, kSitePjTile) &&
            GU_IN_RANGE(j >= 0 && j < p.kb && ((j * kPjBlockK * 2) & 15) == 0 && row0 >= 0 &&
                            row0 < p.m_tiles * Cfg::rows_per_tile && wrow0 >= 0 && wrow0 < p.n_tiles * tile_n,
                        kSitePjLoad)) {
          // rows past M / N and columns past K read as zero
          if constexpr (kPair) {
            mbar_arrive_expect_tx_cluster(full, stage_bytes);
            tma_load_2d_pair(dst, &tm_a, full, j * kPjBlockK, row0);
            tma_load_2d_pair(dst + kPjATileBytes, &tm_w, full, j * kPjBlockK, wrow0);
          } else {
            mbar_arrive_expect_tx(full, stage_bytes);
            tma_load_2d(dst, &tm_a, full, j * kPjBlockK, row0);
            // one row tile: the weights pass through L2 once (evict-first: 93.5 us against 96.4 at M = 128)
            tma_load_2d_hint(dst + kPjATileBytes, &tm_w, full, j * kPjBlockK, wrow0, read_once);
          }
        }
        __syncwarp();
      }
    }
    // the last commits into this CTA's ring barriers must have landed before the CTA may go away
    for (uint32_t s = 0; s < stages; ++s, ++slots)
      pj_wait_elected(ctx, elected, bar_empty + 8 * (slots % stages), ((slots / stages) & 1u) ^ 1u, kWaitPjSlot);
  } else if (warp == 1) {
    if (rank == 0) {
      // ---------------- MMA issuer: the whole warp walks the loop, one elected lane waits and issues ----------------
      const bool elected = elect_one() != 0u;
      const uint32_t idesc = umma_idesc_bf16_f32(Cfg::rows_per_tile, tile_n);
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint32_t empty_odd = kPair ? mapa_shared(bar_empty, 1) : 0u;
      const uint32_t acc_full_odd = kPair ? mapa_shared(bar_acc_full, 1) : 0u;
      const uint64_t adesc0 = umma_desc_k_sw128(ring);
      const uint64_t bdesc0 = umma_desc_k_sw128(ring + kPjATileBytes);
      uint32_t blocks = 0, tiles_done = 0;
      for (int tile = unit; tile < p.num_tiles; tile += units, ++tiles_done) {
        const uint32_t acc = tiles_done & 1u, acc_phase = (tiles_done >> 1) & 1u;
        const uint32_t d = tmem_u + acc * kPjTileN;
        bool ok = pj_wait_elected(ctx, elected, bar_acc_free + 8 * acc, acc_phase ^ 1u, kWaitPjAccFree);
        for (int j = 0; j < p.kb; ++j, ++blocks) {
          const uint32_t stage = blocks % stages, phase = (blocks / stages) & 1u;
          const uint64_t adesc = adesc0 + stage * (stage_bytes >> 4);
          const uint64_t bdesc = bdesc0 + stage * (stage_bytes >> 4);
          ok = pj_wait_elected(ctx, elected, bar_full + 8 * stage, phase, kWaitPjFull) && ok;
          if (ok && elected) {
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < kPjBlockK / 16; ++kk)  // 16 bf16 along K inside the swizzle span: +2 in the address field
              umma_bf16<kPair>(d, adesc + 2 * kk, bdesc + 2 * kk, idesc, (j > 0 || kk > 0) ? 1u : 0u);
            if constexpr (kPair) {
              umma_commit_pair(bar_empty + 8 * stage);
              umma_commit_pair(empty_odd + 8 * stage);
              if (j + 1 == p.kb) {
                umma_commit_pair(bar_acc_full + 8 * acc);
                umma_commit_pair(acc_full_odd + 8 * acc);
              }
            } else {
              umma_commit(bar_empty + 8 * stage);
              if (j + 1 == p.kb) umma_commit(bar_acc_full + 8 * acc);
            }
          }
          __syncwarp();
        }
      }
      // the last hand-backs (the odd CTA's among them) must have landed here before this CTA may go away
      for (uint32_t b = tiles_done; b < tiles_done + 2; ++b)
        pj_wait_elected(ctx, elected, bar_acc_free + 8 * (b & 1u), ((b >> 1) & 1u) ^ 1u, kWaitPjAccFree);
    }
  } else {
    // -------------------------------- epilogue (warps 2-5) ---------------------------------
    const int et = static_cast<int>(threadIdx.x) - 64;  // 0 .. 127
    const int quarter = warp & 3;                        // TMEM lane quarter this warp may read
    const int row = quarter * 32 + lane;                 // row inside this CTA's 128
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t acc_free = kPair ? mapa_shared(bar_acc_free, 0) : bar_acc_free;
    uint8_t* stag_gen = smem_gen + (stag - smem_base);
    uint32_t tiles_done = 0;
    for (int tile = unit; tile < p.num_tiles; tile += units, ++tiles_done) {
      int tm, tn;
      pj_tile_coords(p, tile, tm, tn);
      const int row0 = tm * Cfg::rows_per_tile + static_cast<int>(rank) * kPjTileM;
      const int col0 = tn * tile_n;
      const int chunks = (tile_n + 63) / 64;
      const uint32_t acc = tiles_done & 1u, acc_phase = (tiles_done >> 1) & 1u;
      // (convolution) this lane's row: its mask, position and destination
      uint32_t mask2 = 0u;
      int hist = 0;
      bool keep = false, conv_store = false, edge_row = false;
      uint16_t* conv_out = nullptr;
      if constexpr (kConv) {
        if (row0 + row < p.m && col0 < cv->channels) {
          const int r = row0 + row, b = r / cv->sequence, l = r - b * cv->sequence;
          const uint32_t mb = ld_dep(cv->mask + r);
          mask2 = mb | (mb << 16);
          keep = conv_keeps(mb);
          hist = min(l, kConvTaps - 1);
          conv_store = hist <= row;  // all its taps lie among this CTA's rows
          edge_row = row < kConvTaps - 1 || row >= kPjTileM - (kConvTaps - 1);  // stored for mamba_conv1d_edges_kernel
          conv_out = cv->out + static_cast<long long>(b) * cv->channels * cv->sequence + l;
        }
      }
      // taps and bias of a chunk, a channel pair per thread, fetched one chunk ahead (read where they are used they cost
      // an L2 latency per eight channels: 1 x 512 tokens took 266 us that way)
      uint4 taps_next = make_uint4(0u, 0u, 0u, 0u);
      uint32_t cbias_next = 0u;
      auto fetch_taps = [&](int first) {
        const int ch = first + 2 * (et & 31);
        if (kConv && ch < cv->channels) {
          if (et < 32) taps_next = ld_dep(reinterpret_cast<const uint4*>(cv->weight + static_cast<long long>(ch) * kConvTaps));
          else if (et < 64) cbias_next = ld_dep(reinterpret_cast<const uint32_t*>(cv->bias + ch));
        }
      };
      fetch_taps(col0);
      const bool ok = pj_wait_elected(ctx, lane == 0, bar_acc_full + 8 * acc, acc_phase, kWaitPjAccFull);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < chunks; ++c) {
        const int colc = col0 + 64 * c;
        const bool narrow = !kPair && 64 * c + 64 > tile_n;  // the last 32 columns of a tile
        float v[64];
        tmem_ld32(lane_addr + acc * kPjTileN + 64 * c, v);
        tmem_ld32(lane_addr + acc * kPjTileN + 64 * c + 32, v + 32);  // (narrow: columns of no tile, not used)
        uint4 bq[8];  // this chunk's 64 bias values (the same for every row: broadcast loads)
#pragma unroll
        for (int q = 0; q < 8; ++q)
          bq[q] = (colc + 8 * q < p.n && GU_IN_RANGE(colc + 8 * q >= 0 && colc + 8 * q + 8 <= p.n, kSitePjBias))
                      ? ld_dep(reinterpret_cast<const uint4*>(p.bias + colc + 8 * q))
                      : make_uint4(0, 0, 0, 0);
        tmem_ld_wait_pin<64>(v);
        if (c + 1 == chunks) {
          // the whole accumulator is in registers or stored: hand it back to the issuer
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (kPair) mbar_arrive_cluster(acc_free + 8 * acc);
            else mbar_arrive(acc_free + 8 * acc);
          }
        }
        // the staging tile of this chunk was last read by the store issued two chunks ago
        if (et == 0) tma_store_wait_read1();
        named_bar_sync(1, 128);
        if constexpr (kConv) {
          if (colc < cv->channels) {  // all 64 columns are channels: both are multiples of 64
            uint32_t x[2][16];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const uint32_t bw[4] = {bq[q].x, bq[q].y, bq[q].z, bq[q].w};
              uint32_t o[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float b_lo = __uint_as_float(bw[i] << 16), b_hi = __uint_as_float(bw[i] & 0xffff0000u);
                o[i] = pack_bf16x2(v[8 * q + 2 * i] + b_lo, v[8 * q + 2 * i + 1] + b_hi);
                x[q >> 2][4 * (q & 3) + i] = mask_mul_bf16x2(o[i], mask2);
              }
              if (edge_row && ok && !ctx.aborted && GU_IN_RANGE(row0 + row >= 0 && row0 + row < p.m && colc + 8 * q + 8 <= p.n, kSitePjStore))
                *reinterpret_cast<uint4*>(p.out + static_cast<size_t>(row0 + row) * p.n + colc + 8 * q) =
                    make_uint4(o[0], o[1], o[2], o[3]);
            }
            uint8_t* halo = stag_gen + (c & 1) * kPjOutChunkBytes;
            uint4* taps = reinterpret_cast<uint4*>(halo + kConvHaloBytes);
            uint32_t* biases = reinterpret_cast<uint32_t*>(halo + kConvHaloBytes + kConvTapBytes);
            if (et < 32) taps[et] = taps_next;
            else if (et < 64) biases[et - 32] = cbias_next;
            if (c + 1 < chunks) fetch_taps(colc + 64);
            if (lane >= 29)
#pragma unroll
              for (int q = 0; q < 8; ++q)
                *reinterpret_cast<uint4*>(halo + (quarter * 3 + lane - 29) * 128 + 16 * q) =
                    make_uint4(x[q >> 2][4 * (q & 3)], x[q >> 2][4 * (q & 3) + 1], x[q >> 2][4 * (q & 3) + 2], x[q >> 2][4 * (q & 3) + 3]);
            named_bar_sync(2, 128);
            const bool store = conv_store && ok && !ctx.aborted &&
                               GU_IN_RANGE(row0 + row >= 0 && row0 + row < p.m && colc >= 0 && colc + 64 <= cv->channels, kSitePjConv);
            const uint8_t* above = halo + (quarter == 0 ? 0 : quarter - 1) * 3 * 128;  // (the first warp's edge is not stored)
#pragma unroll
            for (int h = 0; h < 2; ++h)
              conv_row_32(cv->sequence, x[h], above + 64 * h, taps + 16 * h, reinterpret_cast<const uint4*>(biases) + 4 * h, lane, hist,
                          keep, store, conv_out + static_cast<long long>(colc + 32 * h) * cv->sequence);
            if (et == 0) tma_store_commit();  // an empty group: one per chunk, see below
            continue;
          }
        }
        uint8_t* dst_row = stag_gen + (c & 1) * kPjOutChunkBytes + row * 128;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t bw[4] = {bq[q].x, bq[q].y, bq[q].z, bq[q].w};
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float b_lo = __uint_as_float(bw[i] << 16), b_hi = __uint_as_float(bw[i] & 0xffff0000u);
            o[i] = pack_bf16x2(v[8 * q + 2 * i] + b_lo, v[8 * q + 2 * i + 1] + b_hi);
          }
          if (!narrow) {
            *reinterpret_cast<uint4*>(dst_row + ((q ^ (row & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
          } else if (q < 4 && row0 + row < p.m && colc + 8 * q < p.n && ok && !ctx.aborted &&
                     GU_IN_RANGE(row0 + row >= 0 && colc + 8 * q + 8 <= p.n, kSitePjStore)) {
            // a 64-column TMA store would write into the next tile; N is a multiple of 8
            *reinterpret_cast<uint4*>(p.out + static_cast<size_t>(row0 + row) * p.n + colc + 8 * q) =
                make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        fence_proxy_async_smem();
        named_bar_sync(2, 128);
        // (a store may reach past the last row or column, where it is clipped, but starts inside the tensor)
        if (et == 0) {
          if (!narrow && ok && !ctx.aborted && row0 < p.m && colc < p.n &&
              GU_IN_RANGE(row0 >= 0 && colc >= 0 && ((colc * 2) & 15) == 0, kSitePjStore))
            tma_store_2d(&tm_out, stag + (c & 1) * kPjOutChunkBytes, colc, row0);  // rows past M, columns past N are clipped
          // one group per chunk, also when the chunk lies outside the tensor and nothing is stored (an empty group):
          // "all groups but the newest have been read" above then always means "the store two chunks back has"
          tma_store_commit();
        }
      }
    }
    if (et == 0) tma_store_wait_all0();
  }

  // ------------------------------- teardown --------------------------------
  if (*abort_gen) {
    // give copies that were already in flight time to land before shared memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) spin_backoff_ns(1000u);
  }
  tc_fence_before();
  __syncwarp();
  if constexpr (kPair) cluster_sync_all();  // neither CTA leaves while the other may still reach into it
  else __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    __syncwarp();
    if constexpr (kPair) tmem_dealloc_pair(tmem_base, kPjTmemCols);
    else tmem_dealloc(tmem_base, kPjTmemCols);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPjThreads, 1)
proj_gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                      const __grid_constant__ CUtensorMap tm_out, const ProjParams p) {
  proj_gemm_body<true, false>(tm_a, tm_w, tm_out, p, nullptr);
}

__global__ void __launch_bounds__(kPjThreads, 1)
proj_gemm_lone_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                      const __grid_constant__ CUtensorMap tm_out, const ProjParams p) {
  proj_gemm_body<false, false>(tm_a, tm_w, tm_out, p, nullptr);
}

// With the convolution tail in the epilogue (see ConvParams).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPjThreads, 1)
proj_conv_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_w,
                      const __grid_constant__ CUtensorMap tm_out, const ProjParams p, const ConvParams cv) {
  proj_gemm_body<true, true>(tm_a, tm_w, tm_out, p, &cv);
}

}  // namespace so
