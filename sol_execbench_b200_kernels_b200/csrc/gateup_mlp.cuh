// Weight-streaming kernels of the MLP block for up to 16 tokens and large weights: the gate/up projection with its result
// re-quantised to e4m3, and the down projection.
//
// As in gateup_stream.cuh the weights are the MMA's "M" operand and the tokens (padded to 16) its "N" operand, a work unit
// is two 128 x 128 weight tiles, and the (column block, step) units are cut into gridDim.x equal contiguous ranges, so
// every SM pulls the same number of weight bytes whatever the matrix's height; whole tiles leave SMs idle in their last
// round (8 tokens of 8192 x 28672: 224 tiles on 148 SMs, the block 131 us; 114 this way, 107 at HBM's rate).
// Every hop through global memory takes 1.5 us while HBM is busy, so partial sums travel without flags or fences: a thread
// stores pairs {sum, launch stamp}, 8 bytes at once, and the owner's threads read them until every stamp is this
// launch's: one trip instead of store, fence, flag, poll, load.  (A down projection to 4096 columns has 32 column blocks
// for 148 ranges: an owner collects four or five.)  The stamp is a launch count kept in the scratch, so a recorded launch
// can be replayed.
//
// Warps: 0 TMA producer, 1 TMEM allocation + MMA issue, 2-5 consumers (a thread per output column).
#pragma once

#include "gateup_stream.cuh"

namespace gu {

enum : int {
  kMlpGateUp = 0,  // a unit is the gate and the up tile of a K block; SwiGLU, e4m3 + one scale per token and 128 columns
  kMlpDown = 1,    // a unit is two K blocks of the one matrix; bf16
};
enum : unsigned { kWaitMlpPartial = 22 };
enum : unsigned { kSiteMlpLoad = 81, kSiteMlpStage = 82, kSiteMlpScale = 83, kSiteMlpPartial = 84, kSiteMlpStore = 85 };

constexpr int kMlpTokens = 16;  // MMA N
constexpr uint32_t kMlpXTileBytes = kMlpTokens * 128;
constexpr int kMlpMaxStages = 5;
constexpr uint32_t kMlpBarBytes = 256;
constexpr uint32_t kMlpMaxBytes = 4 * kMlpTokens * 4;  // the four consumer warps' row maxima
constexpr size_t kMlpSlotPairs = size_t(2) * kMlpTokens * 128;  // {sum, stamp} pairs that a range may hand over

constexpr int mlp_blocks_per_unit(int op) { return op == kMlpDown ? 2 : 1; }  // K blocks
constexpr uint32_t mlp_stage_bytes(int op) { return 2 * kOperandTileBytes + mlp_blocks_per_unit(op) * kMlpXTileBytes; }
// beside the ring; `kept`: steps of a column block that a CTA's range touches
constexpr uint32_t mlp_fixed_bytes(int op, int64_t kept) {
  return kMlpBarBytes + kMlpMaxBytes + 1024 + static_cast<uint32_t>(kept) * mlp_blocks_per_unit(op) * kMlpTokens * 4;
}

struct MlpStepParams {
  const float* scale_x;     // [M, kb]
  const float* scale_gate;  // [nb, kb]; the one matrix's scales in the down projection
  const float* scale_up;
  void* out;                // e4m3 [M, ld_out] with scale_out [M, nb], or bf16 [M, ld_out]
  float* scale_out;
  long long ld_out;
  int m, kb, nb;
  int stages;               // ring depth
  unsigned int* sync;       // [0] the last launch's stamp on this scratch, [1] tickets of the running one
  uint2* partials;          // [gridDim.x][kMlpSlotPairs]
};

template <int kOp>
__global__ void __launch_bounds__(kStreamThreads, 1)
mlp_step_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w0,
                const __grid_constant__ CUtensorMap tm_w1, const MlpStepParams p) {
  constexpr bool kDown = kOp == kMlpDown;
  constexpr int kBlocks = kDown ? 2 : 1, kSums = kDown ? 1 : 2;
  constexpr uint32_t kStageBytes = 2 * kOperandTileBytes + kBlocks * kMlpXTileBytes;
  constexpr int T = kMlpTokens;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

  // equal unit ranges; reverse block order: a range only ever waits for ranges with a HIGHER index, i.e. blocks with a
  // LOWER blockIdx, which the hardware dispatches first
  const int ranges = gridDim.x;
  const int my_range = ranges - 1 - static_cast<int>(blockIdx.x);
  const int steps = (p.kb + kBlocks - 1) / kBlocks;  // units of one column block
  const long long units = static_cast<long long>(p.nb) * steps;
  auto range_start = [&](int r) { return units * r / ranges; };
  const long long u_begin = range_start(my_range), u_end = range_start(my_range + 1);
  const int count = static_cast<int>(u_end - u_begin);
  const int kept = min(count, steps);
  const int nbk0 = static_cast<int>(u_begin / steps);
  const int j0 = static_cast<int>(u_begin - static_cast<long long>(nbk0) * steps);
  // whether step j has a second weight tile (the last step of an odd number of K blocks has none)
  auto second = [&](int j) { return !kDown || 2 * j + 1 < p.kb; };

  const uint32_t ring = smem_base;
  const uint32_t bars = ring + p.stages * kStageBytes;
  const uint32_t bar_full = bars;                            // [kMlpMaxStages]
  const uint32_t bar_empty = bars + 8 * kMlpMaxStages;       // [kMlpMaxStages]
  const uint32_t bar_acc_full = bars + 16 * kMlpMaxStages;   // [kStreamAccStages]
  const uint32_t bar_acc_empty = bar_acc_full + 8 * kStreamAccStages;
  const uint32_t tmem_slot = bar_acc_empty + 8 * kStreamAccStages;
  const uint32_t abort_slot = tmem_slot + 4;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - smem_base));
  volatile int* abort_gen = reinterpret_cast<volatile int*>(smem_gen + (abort_slot - smem_base));
  volatile unsigned int* epoch_gen = reinterpret_cast<volatile unsigned int*>(smem_gen + (abort_slot + 4 - smem_base));
  float* max_smem = reinterpret_cast<float*>(smem_gen + (bars - smem_base) + kMlpBarBytes);  // [4][T]
  float* sx_smem = max_smem + kMlpMaxBytes / 4;                                             // [kept][kBlocks][T]

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    pdl_trigger();
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < kStreamAccStages; ++s) {
      mbar_init(bar_acc_full + 8 * s, 1);
      mbar_init(bar_acc_empty + 8 * s, 4);  // one arrival per consumer warp
    }
    *abort_gen = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_w0);
    tma_prefetch_desc(&tm_w1);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kStreamAccStages * 2 * T);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_gen;

  const uint64_t stream_once = l2_policy_evict_first();  // weights are read exactly once
  auto in_range = [&](int stage, int nbk, int j) {
    (void)stage; (void)nbk; (void)j;  // (only the range-checked build looks at them)
    return GU_IN_RANGE(stage >= 0 && stage < p.stages && p.stages <= kMlpMaxStages, kSiteMlpStage) &&
           GU_IN_RANGE(load_coords_ok(p.kb, j * kBlocks, nbk * 128, p.nb * 128), kSiteMlpLoad);
  };
  auto load_weights = [&](int stage, int nbk, int j) {
    const uint32_t full = bar_full + 8 * stage, dst = ring + stage * kStageBytes;
    if constexpr (kDown) {
      const bool two = second(j);
      mbar_arrive_expect_tx(full, two ? kStageBytes : kStageBytes / 2);
      tma_load_2d_hint(dst, &tm_w0, full, 2 * j * kBlockK, nbk * 128, stream_once);
      if (two) tma_load_2d_hint(dst + kOperandTileBytes, &tm_w0, full, (2 * j + 1) * kBlockK, nbk * 128, stream_once);
    } else {
      mbar_arrive_expect_tx(full, kStageBytes);
      tma_load_2d_hint(dst, &tm_w0, full, j * kBlockK, nbk * 128, stream_once);
      tma_load_2d_hint(dst + kOperandTileBytes, &tm_w1, full, j * kBlockK, nbk * 128, stream_once);
    }
  };
  // (producer) the first ring's weights, before the wait: the block's quantiser lets nothing start before all in front of it
  // has completed, so they are ready (see TileParams::weights_ready)
  int early = 0;
  if (warp == 0 && lane == 0) {
    int nbk = nbk0, j = j0;
    early = min(count, p.stages);
#pragma unroll 1
    for (int i = 0; i < early; ++i) {
      if (in_range(i, nbk, j)) load_weights(i, nbk, j);
      if (++j == steps) { j = 0; ++nbk; }
    }
  }
  pdl_wait();

  WaitCtx ctx{abort_slot, false, false};

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------ TMA producer ------------------------------
      const uint64_t keep = l2_policy_evict_last();  // the X tiles are read by every CTA
      int stage = 0, nbk = nbk0, j = j0;
      uint32_t phase = 0;
      for (int u = 0; u < count; ++u) {
        const bool loaded = u < early;
        if ((loaded || mbar_wait(ctx, bar_empty + 8 * stage, phase ^ 1u, kWaitStreamEmpty)) && in_range(stage, nbk, j)) {
          if (!loaded) load_weights(stage, nbk, j);
          const uint32_t full = bar_full + 8 * stage, dst = ring + stage * kStageBytes + 2 * kOperandTileBytes;
          tma_load_2d_hint(dst, &tm_x, full, kBlocks * j * kBlockK, 0, keep);
          if (kDown && second(j)) tma_load_2d_hint(dst + kMlpXTileBytes, &tm_x, full, (2 * j + 1) * kBlockK, 0, keep);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        if (++j == steps) { j = 0; ++nbk; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------- MMA issuer -------------------------------
      constexpr uint32_t idesc = umma_idesc_e4m3_f32(128, T);
      int stage = 0, acc = 0, j = j0;
      uint32_t phase = 0, acc_phase = 0;
      for (int u = 0; u < count; ++u) {
        bool ok = mbar_wait(ctx, bar_acc_empty + 8 * acc, acc_phase ^ 1u, kWaitStreamAccEmpty);
        ok = mbar_wait(ctx, bar_full + 8 * stage, phase, kWaitStreamFull) && ok;
        if (ok) {
          tc_fence_after();
          const uint32_t base = ring + stage * kStageBytes;
          const uint32_t x = base + 2 * kOperandTileBytes;
          const uint64_t w0desc = umma_desc_k_sw128(base);
          const uint64_t w1desc = umma_desc_k_sw128(base + kOperandTileBytes);
          const uint64_t x0desc = umma_desc_k_sw128(x);
          const uint64_t x1desc = umma_desc_k_sw128(x + (kDown ? kMlpXTileBytes : 0u));
          const uint32_t d = tmem_base + acc * (2 * T);
          const bool two = second(j);
#pragma unroll
          for (int kk = 0; kk < kBlockK / 32; ++kk) {
            umma_f8(d, w0desc + 2 * kk, x0desc + 2 * kk, idesc, kk > 0 ? 1u : 0u);
            if (two) umma_f8(d + T, w1desc + 2 * kk, x1desc + 2 * kk, idesc, kk > 0 ? 1u : 0u);
          }
          umma_commit(bar_empty + 8 * stage);
          umma_commit(bar_acc_full + 8 * acc);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        if (++acc == kStreamAccStages) { acc = 0; acc_phase ^= 1u; }
        if (++j == steps) j = 0;
      }
    }
  } else {
    // ------------------------------- consumers --------------------------------
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;  // weight row inside the tile = output column inside the block
    const int ctid = threadIdx.x - 64;    // 0..127
    unsigned int ticket = 0;
    if (ctid == 0) {
      unsigned int s = ld_acquire_gpu(p.sync) + 1u;  // this launch's stamp, never 0
      if (s == 0u) s = 1u;
      *epoch_gen = s;
      ticket = atomicAdd(p.sync + 1, 1u);
    }
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);

    // the token scales, transposed to [step][block][T] so one K block's are contiguous; step e of the range is step
    // (j0 + e) % steps of a column block
    const int total = kept * kBlocks * T;
#pragma unroll 4
    for (int i = ctid; i < total; i += 128) {
      const int t = i % T, eb = i / T;
      int j = j0 + eb / kBlocks;
      if (j >= steps) j -= steps;
      const int blk = j * kBlocks + eb % kBlocks;
      sx_smem[i] = (t < p.m && blk < p.kb) ? ld_dep(p.scale_x + static_cast<size_t>(t) * p.kb + blk) : 0.f;
    }
    named_bar_sync(1, 128);
    const unsigned int epoch = *epoch_gen;

    float g[T], up[kDown ? 1 : T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      g[t] = 0.f;
      if constexpr (!kDown) up[t] = 0.f;
    }
    int acc = 0, nbk = nbk0, j = j0, e = 0;
    uint32_t acc_phase = 0;
    bool owner = j0 == 0;  // this segment starts with the column block's first K block
    float s0_next = 0.f, s1_next = 0.f;  // weight scales of the next unit's two tiles
    auto fetch_scales = [&](int nbk_, int j_) {
      const size_t first = static_cast<size_t>(nbk_) * p.kb + j_ * kBlocks;
      if (!GU_IN_RANGE(nbk_ < p.nb && j_ * kBlocks < p.kb, kSiteMlpScale)) return;
      s0_next = ld_dep(p.scale_gate + first);
      if constexpr (kDown) s1_next = second(j_) ? ld_dep(p.scale_gate + first + 1) : 0.f;
      else s1_next = ld_dep(p.scale_up + first);
    };
    fetch_scales(nbk, j);

    for (int u = 0; u < count; ++u) {
      const float s0 = s0_next, s1 = s1_next;
      const int j_next = j + 1 == steps ? 0 : j + 1, nbk_next = j + 1 == steps ? nbk + 1 : nbk;
      if (u + 1 < count) fetch_scales(nbk_next, j_next);
      const bool ok = mbar_wait(ctx, bar_acc_full + 8 * acc, acc_phase, kWaitStreamAccFull);
      tc_fence_after();
      {
        float v0[T], v1[T];
        if (__all_sync(0xffffffffu, ok)) {
          const uint32_t t0 = lane_addr + acc * (2 * T);
          tmem_ld16(t0, v0);
          tmem_ld16(t0 + T, v1);
          tmem_ld_wait_pin<T>(v0);
          tmem_ld_wait_pin<T>(v1);
        } else {
#pragma unroll
          for (int t = 0; t < T; ++t) { v0[t] = 0.f; v1[t] = 0.f; }
        }
        const float4* sx0 = reinterpret_cast<const float4*>(sx_smem + e * (kBlocks * T));
        const float4* sx1 = sx0 + (kDown ? T / 4 : 0);
        // (down: a step without a second tile leaves v1 as an earlier step's partial, which is not added)
        const bool two = second(j);
#pragma unroll
        for (int t4 = 0; t4 < T / 4; ++t4) {
          const float4 a = sx0[t4];
          const int t = 4 * t4;
          g[t + 0] = fmaf(v0[t + 0], a.x * s0, g[t + 0]);
          g[t + 1] = fmaf(v0[t + 1], a.y * s0, g[t + 1]);
          g[t + 2] = fmaf(v0[t + 2], a.z * s0, g[t + 2]);
          g[t + 3] = fmaf(v0[t + 3], a.w * s0, g[t + 3]);
          if constexpr (kDown) {
            if (two) {
              const float4 b = sx1[t4];
              g[t + 0] = fmaf(v1[t + 0], b.x * s1, g[t + 0]);
              g[t + 1] = fmaf(v1[t + 1], b.y * s1, g[t + 1]);
              g[t + 2] = fmaf(v1[t + 2], b.z * s1, g[t + 2]);
              g[t + 3] = fmaf(v1[t + 3], b.w * s1, g[t + 3]);
            }
          } else {
            up[t + 0] = fmaf(v1[t + 0], a.x * s1, up[t + 0]);
            up[t + 1] = fmaf(v1[t + 1], a.y * s1, up[t + 1]);
            up[t + 2] = fmaf(v1[t + 2], a.z * s1, up[t + 2]);
            up[t + 3] = fmaf(v1[t + 3], a.w * s1, up[t + 3]);
          }
        }
      }
      // every read of this TMEM stage has completed: hand it back to the MMA issuer
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_acc_empty + 8 * acc);
      if (++acc == kStreamAccStages) { acc = 0; acc_phase ^= 1u; }

      const bool block_done = j == steps - 1;
      if (block_done || u + 1 == count) {
        // ------------------------- end of a segment -------------------------
        if (!owner) {
          // started mid-block: hand the partial sums to the block's owner
          if (!ctx.aborted && GU_IN_RANGE(my_range >= 0 && my_range < ranges && row >= 0 && row < 128, kSiteMlpPartial)) {
            uint2* slot = p.partials + static_cast<size_t>(my_range) * kMlpSlotPairs + row;
#pragma unroll
            for (int t = 0; t < T; ++t) {
              if (t < p.m) {
                st_pair(slot + t * 128, g[t], epoch);
                if constexpr (!kDown) st_pair(slot + (T + t) * 128, up[t], epoch);
              }
            }
          }
        } else {
          if (!block_done) {
            // owner of the block's first K block: collect the later ranges' partials, in range order
            const long long block_end = static_cast<long long>(nbk + 1) * steps;
            for (int rr = my_range + 1; rr < ranges && range_start(rr) < block_end; ++rr) {
              const uint2* slot = p.partials + static_cast<size_t>(rr) * kMlpSlotPairs + row;
              uint2 v[kSums * T];
              unsigned long long t0 = 0;
              for (uint32_t it = 1; !ctx.aborted; ++it) {
                bool here = true;
#pragma unroll
                for (int t = 0; t < kSums * T; ++t) {
                  v[t] = make_uint2(0u, epoch);
                  if (t % T < p.m) v[t] = ld_pair(slot + t * 128);
                }
#pragma unroll
                for (int t = 0; t < kSums * T; ++t) here = here && v[t].y == epoch;
                if (here) break;
                if ((it & 63u) == 0u) {
                  const unsigned long long now = globaltimer_ns();
                  if (t0 == 0) {
                    t0 = now;
                  } else if (now - t0 > g_wait_limit_ns || ctx.raised()) {
                    ctx.fail(kWaitMlpPartial, (kWaitMlpPartial << 24) | (blockIdx.x & 0xffffffu));
                  }
                }
              }
#pragma unroll
              for (int t = 0; t < T; ++t) {
                g[t] += __uint_as_float(v[t].x);
                if constexpr (!kDown) up[t] += __uint_as_float(v[T + t].x);
              }
            }
            __syncwarp();
          }
          // epilogue: consecutive lanes hold consecutive output columns
          const size_t col = static_cast<size_t>(nbk) * 128 + row;
          const bool store = GU_IN_RANGE(nbk >= 0 && nbk < p.nb && static_cast<long long>(nbk) * 128 + row < p.ld_out, kSiteMlpStore);
          if constexpr (kDown) {
            __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.out) + col;
#pragma unroll
            for (int t = 0; t < T; ++t)
              if (t < p.m && store) dst[static_cast<size_t>(t) * p.ld_out] = __float2bfloat16_rn(g[t]);
          } else {
            float o[T];
#pragma unroll
            for (int t = 0; t < T; ++t) {
              o[t] = bf16_round(swiglu_bf16(g[t], up[t]));
              // the largest magnitude as an unsigned maximum of the bits (a NaN counts as 0, as in fmaxf)
              const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(o[t]), 0.f)));
              if (lane == 0) max_smem[quarter * T + t] = __uint_as_float(top);
            }
            named_bar_sync(1, 128);
            uint8_t* dst = static_cast<uint8_t*>(p.out) + col;
#pragma unroll
            for (int t = 0; t < T; ++t) {
              if (t < p.m && store) {
                const float amax = fmaxf(fmaxf(max_smem[t], max_smem[T + t]), fmaxf(max_smem[2 * T + t], max_smem[3 * T + t]));
                const float sc = fmaxf(amax, 1e-12f) / 448.0f;
                const uint32_t bits = __float_as_uint(o[t]) >> 16;
                dst[static_cast<size_t>(t) * p.ld_out] = static_cast<uint8_t>(e4m3x4_from_bf16x4(bits, 0u, sc, __frcp_rn(sc)));
                if (ctid == t) p.scale_out[static_cast<size_t>(t) * p.nb + nbk] = sc;
              }
            }
            named_bar_sync(1, 128);  // the maxima have been read: the next block's may be written
          }
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
          g[t] = 0.f;
          if constexpr (!kDown) up[t] = 0.f;
        }
        owner = true;
      }
      j = j_next;
      nbk = nbk_next;
      if (++e == steps) e = 0;
    }
    // whoever drew the last ticket (every CTA has read the count by then) counts the launch: the count becomes its stamp,
    // so that 1 follows 0xffffffff once and the launch after it stamps with 2
    if (ctid == 0 && ticket == gridDim.x - 1u) {
      p.sync[0] = epoch;
      p.sync[1] = 0u;
    }
  }

  // ------------------------------- teardown --------------------------------
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*abort_gen) {
    // give copies that were already in flight time to land before shared memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) spin_backoff_ns(1000u);
  }
  if (warp == 1) tmem_dealloc(tmem_base, kStreamAccStages * 2 * T);
}

}  // namespace gu
