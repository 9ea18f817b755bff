// K-split kernel for launches with few output tiles: a cluster of S CTAs (2 .. 8, neighbouring SMs) owns ONE
// 128-token x 256-accumulator-column tile of the lone-CTA kernel, each CTA walks 1/S of the tile's K blocks, and the
// S partial tiles are added through distributed shared memory.
//
// What bounds such a launch is how many SMs pull weights from HBM, not the tensor cores: a down projection to 4096
// columns has 16 column tiles, so the lone-CTA kernel streams 58.7 MB of weights through 16 SMs (61.5 us at 8 tokens,
// 0.95 TB/s) while 132 idle.  With 8 CTAs per tile 128 SMs stream.  Cutting along K inside a cluster (and not into
// ranges that meet in global memory) needs no scratch, no flags and no waiting on CTAs that may not be resident: the
// hardware schedules the S CTAs together, and the hand-over is one cluster barrier.
//
// Per CTA: TMA producer (warp 0), MMA issuer (warp 1), eight consumer warps as in gateup_tile.cuh; those whose 32
// token rows do not exist take no part.  At the end a CTA writes its fp32 sums into its own (by then idle) operand
// ring, [token][column] at a pitch of 260 words: eight lanes' 16-byte stores (lanes = tokens) hit 32 different banks,
// and a warp reads a token's 128 columns of a projection from another CTA as 512 contiguous bytes.  (The reads decide:
// with 4-byte reads 129 words apart, every lane its own 32-byte packet, joining two 128-token halves took 30 us.)
// After the cluster barrier CTA r finishes the r-th share of the tile's token rows: a warp takes a row, adds the S
// partial sums in ascending K order and applies the epilogue of its mode (SwiGLU to bf16, SwiGLU to e4m3 + scale, plain
// bf16).  A whole row in one warp makes the row maximum of the e4m3 mode a shuffle.
#pragma once

#include "gateup_pair.cuh"

namespace gu {

enum : int { kSplitGateUp = 0, kSplitFp8 = 1, kSplitGemm = 2 };
enum : unsigned { kWaitSplitEmpty = 18, kWaitSplitFull = 19, kWaitSplitAccEmpty = 20, kWaitSplitAccFull = 21 };
enum : unsigned { kSiteSplitLoad = 65, kSiteSplitScale = 66, kSiteSplitStage = 67, kSiteSplitStore = 68, kSiteSplitPart = 69 };

constexpr int kSplitMaxCtas = 8;                // portable cluster size
constexpr uint32_t kSplitPitch = 2 * kTileN + 4;  // words per token row of the partial tile
constexpr uint32_t kSplitSmemBytes = kTileStages * kTileStageBytes + 256 /*barriers*/ + 1024 /*alignment slack*/;
static_assert(kTileM * kSplitPitch * 4 <= kTileStages * kTileStageBytes, "the partial tile fits the operand ring");

struct SplitParams {
  const float* scale_x;     // [M, kb]
  const float* scale_gate;  // [nb, kb]; the one B matrix's scales in the plain GEMM
  const float* scale_up;
  void* out;                // bf16 [M, ld_out], or e4m3 [M, N] with scale_out [M, N/128]
  float* scale_out;
  long long ld_out;
  int m, kb;
  int num_m_blocks, n_blocks128;
  uint32_t x_bytes;         // bytes of an X box (see x_box_rows)
  int weights_ready;        // the weights were complete before any kernel began that this one may overlap: a step of
                            // gu_mlp_block behind its quantiser, and nothing else (see pdl_wait)
};

__device__ __forceinline__ float4 ld_shared_cluster_f32x4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_addr)
               : "memory");
  return v;
}

template <int kOp>
__global__ void __launch_bounds__(kTileThreads, 1)
gateup_split_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_gate,
                    const __grid_constant__ CUtensorMap tm_up, const SplitParams p) {
  constexpr bool kSingle = kOp == kSplitGemm;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;  // the same offset in every CTA of the cluster
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

  const uint32_t ring = smem_base;
  const uint32_t bars = smem_base + kTileStages * kTileStageBytes;
  const uint32_t bar_full = bars;                         // [kTileStages]
  const uint32_t bar_empty = bars + 8 * kTileStages;      // [kTileStages]
  const uint32_t bar_acc_full = bars + 16 * kTileStages;  // [2]
  const uint32_t bar_acc_empty = bar_acc_full + 16;       // [2]
  const uint32_t tmem_slot = bar_acc_empty + 16;
  const uint32_t abort_slot = tmem_slot + 4;
  volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + (tmem_slot - smem_base));
  volatile int* abort_gen = reinterpret_cast<volatile int*>(smem_gen + (abort_slot - smem_base));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int splits = static_cast<int>(cluster_nctarank());
  const int rank = static_cast<int>(cluster_ctarank());
  const int tile = static_cast<int>(blockIdx.x) / splits;
  const int nb = tile / p.num_m_blocks, mb = tile - nb * p.num_m_blocks;  // tiles that share weights run side by side
  const int jb = p.kb * rank / splits, je = p.kb * (rank + 1) / splits;  // (the host keeps splits <= kb)
  const int rows = min(kTileM, p.m - mb * kTileM);                        // tokens of this tile

  if (threadIdx.x == 0) {
    pdl_trigger();
    for (int s = 0; s < kTileStages; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_acc_full + 8 * s, 1);
      mbar_init(bar_acc_empty + 8 * s, 2 * ((rows + 31) / 32));  // one arrival per consumer warp that has tokens
    }
    *abort_gen = 0;
    fence_mbar_init();
    fence_proxy_async_smem();
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_gate);
    tma_prefetch_desc(&tm_up);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTileTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_gen;

  WaitCtx ctx{abort_slot, false, false};

  if (warp < 4) {
    reg_dealloc<64>();
    if (warp == 0 && lane == 0) {
      // ------------------------------ TMA producer ------------------------------
      const int w0 = kSingle ? 2 * nb * kTileN : nb * kTileN;
      const int w1 = kSingle ? w0 + kTileN : w0;
      const uint64_t read_once = l2_policy_evict_first();
      auto in_range = [&](int stage, int j) {
        (void)stage; (void)j;
        return GU_IN_RANGE(stage >= 0 && stage < kTileStages, kSiteSplitStage) &&
               GU_IN_RANGE(load_coords_ok(p.kb, j, mb * kTileM, p.num_m_blocks * kTileM) &&
                               load_coords_ok(p.kb, j, w0, p.n_blocks128 * kTileN) &&
                               load_coords_ok(p.kb, j, w1, (p.n_blocks128 + 1) * kTileN), kSiteSplitLoad);
      };
      auto load_weights = [&](int stage, int j) {
        const uint32_t full = bar_full + 8 * stage, dst = ring + stage * kTileStageBytes;
        mbar_arrive_expect_tx(full, 2 * kOperandTileBytes + p.x_bytes);
        if (p.num_m_blocks == 1) {  // the weights pass through L2 once
          tma_load_2d_hint(dst + kOperandTileBytes, &tm_gate, full, j * kBlockK, w0, read_once);
          tma_load_2d_hint(dst + 2 * kOperandTileBytes, kSingle ? &tm_gate : &tm_up, full, j * kBlockK, w1, read_once);
        } else {
          tma_load_2d(dst + kOperandTileBytes, &tm_gate, full, j * kBlockK, w0);
          tma_load_2d(dst + 2 * kOperandTileBytes, kSingle ? &tm_gate : &tm_up, full, j * kBlockK, w1);  // rows past N read as zero
        }
      };
      auto load_x = [&](int stage, int j) {
        tma_load_2d(ring + stage * kTileStageBytes, &tm_x, bar_full + 8 * stage, j * kBlockK, mb * kTileM);
      };
      // the first ring's worth of weights does not have to wait for the kernel that produces the activations
      const int early = p.weights_ready ? min(kTileStages, je - jb) : 0;
      for (int i = 0; i < early; ++i)
        if (in_range(i, jb + i)) load_weights(i, jb + i);
      // and where that is not known, into L2 (doing both took bandwidth from the kernel in front: 53.6 against 50.9 us
      // for the MLP block at 8 x 4096 x 14336)
      for (int j = jb; early == 0 && j < min(jb + kTileStages, je); ++j) {
        if (!in_range(0, j)) continue;
        tma_prefetch_2d(&tm_gate, j * kBlockK, w0);
        if (!kSingle || 2 * nb + 1 < p.n_blocks128) tma_prefetch_2d(kSingle ? &tm_gate : &tm_up, j * kBlockK, w1);
      }
      pdl_wait();
      for (int i = 0; i < early; ++i)
        if (in_range(i, jb + i)) load_x(i, jb + i);
      int stage = early % kTileStages;
      uint32_t phase = early == kTileStages ? 1u : 0u;
      for (int j = jb + early; j < je; ++j) {
        if (mbar_wait(ctx, bar_empty + 8 * stage, phase ^ 1u, kWaitSplitEmpty) && in_range(stage, j)) {
          load_weights(stage, j);
          load_x(stage, j);
        }
        if (++stage == kTileStages) { stage = 0; phase ^= 1u; }
      }
    } else if (warp == 1 && lane == 0) {
      // ------------------------------- MMA issuer -------------------------------
      constexpr uint32_t idesc = umma_idesc_e4m3_f32(kTileM, 2 * kTileN);
      // no MMA can start before X is loaded, which is after this; a bounded wait begun earlier would count the time of
      // the kernel in front
      pdl_wait();
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int j = jb; j < je; ++j) {
        bool ok = mbar_wait(ctx, bar_acc_empty + 8 * acc, acc_phase ^ 1u, kWaitSplitAccEmpty);
        ok = mbar_wait(ctx, bar_full + 8 * stage, phase, kWaitSplitFull) && ok;
        if (ok) {
          tc_fence_after();
          const uint32_t a_addr = ring + stage * kTileStageBytes;
          const uint64_t adesc = umma_desc_k_sw128(a_addr);
          const uint64_t bdesc = umma_desc_k_sw128(a_addr + kOperandTileBytes);
          const uint32_t d = tmem_base + acc * (2 * kTileN);
#pragma unroll
          for (int kk = 0; kk < kBlockK / 32; ++kk) umma_f8(d, adesc + 2 * kk, bdesc + 2 * kk, idesc, kk > 0 ? 1u : 0u);
          umma_commit(bar_empty + 8 * stage);
          umma_commit(bar_acc_full + 8 * acc);
        }
        if (++stage == kTileStages) { stage = 0; phase ^= 1u; }
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    reg_alloc<216>();
    // ------------------------------- consumers --------------------------------
    pdl_wait();  // the scales of x come from the kernel in front; the epilogue may overwrite what it reads
    const int quarter = warp & 3;         // TMEM lane quarter this warp may read
    const int half = (warp - 4) >> 2;     // which 64 of the 128 columns of either projection
    const int row = quarter * 32 + lane;  // token row inside the tile
    if (quarter * 32 < rows) {
      const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * 64;
      const int m_global = min(mb * kTileM + row, p.m - 1);
      const int b0 = kSingle ? 2 * nb : nb, b1 = kSingle ? min(2 * nb + 1, p.n_blocks128 - 1) : nb;
      const float* sx_row = p.scale_x + static_cast<size_t>(m_global) * p.kb;
      const float* sg_row = p.scale_gate + static_cast<size_t>(b0) * p.kb;
      const float* su_row = (kSingle ? p.scale_gate : p.scale_up) + static_cast<size_t>(b1) * p.kb;
      float2 g[32], u[32];  // 64 + 64 running sums
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        g[i] = make_float2(0.f, 0.f);
        u[i] = make_float2(0.f, 0.f);
      }
      float sx0 = 0.f, sg0 = 0.f, su0 = 0.f, sx1 = 0.f, sg1 = 0.f, su1 = 0.f;
      const bool in = GU_IN_RANGE(m_global >= 0 && m_global < p.m && b0 < p.n_blocks128 && b1 < p.n_blocks128 &&
                                  jb >= 0 && je <= p.kb, kSiteSplitScale);
      if (in) {
        if (jb < je) { sx0 = ld_dep(sx_row + jb); sg0 = ld_dep(sg_row + jb); su0 = ld_dep(su_row + jb); }
        if (jb + 1 < je) { sx1 = ld_dep(sx_row + jb + 1); sg1 = ld_dep(sg_row + jb + 1); su1 = ld_dep(su_row + jb + 1); }
      }
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int j = jb; j < je; ++j) {
        // scales are fetched two K blocks ahead of their use
        float sx2 = 0.f, sg2 = 0.f, su2 = 0.f;
        if (in && j + 2 < je) { sx2 = ld_dep(sx_row + j + 2); sg2 = ld_dep(sg_row + j + 2); su2 = ld_dep(su_row + j + 2); }
        const float2 sg2v = make_float2(sx0 * sg0, sx0 * sg0);
        const float2 su2v = make_float2(sx0 * su0, sx0 * su0);
        const bool ok = mbar_wait(ctx, bar_acc_full + 8 * acc, acc_phase, kWaitSplitAccFull);
        tc_fence_after();
        float v[64];
        if (__all_sync(0xffffffffu, ok)) {
          const uint32_t t = lane_addr + acc * (2 * kTileN);
          tmem_ld32(t, v);
          tmem_ld32(t + 32, v + 32);
          tmem_ld_wait_pin<64>(v);
#pragma unroll
          for (int i = 0; i < 32; ++i) g[i] = __ffma2_rn(make_float2(v[2 * i], v[2 * i + 1]), sg2v, g[i]);
          tmem_ld32(t + kTileN, v);
          tmem_ld32(t + kTileN + 32, v + 32);
          tmem_ld_wait_pin<64>(v);
        } else {
#pragma unroll
          for (int i = 0; i < 64; ++i) v[i] = 0.f;
        }
        // the partial is in registers: hand the TMEM stage back before the last FMAs
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_acc_empty + 8 * acc);
#pragma unroll
        for (int i = 0; i < 32; ++i) u[i] = __ffma2_rn(make_float2(v[2 * i], v[2 * i + 1]), su2v, u[i]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
        sx0 = sx1; sg0 = sg1; su0 = su1;
        sx1 = sx2; sg1 = sg2; su1 = su2;
      }
      // The last partial has been read, so every load into the ring has landed and every MMA has read it: the ring is
      // free for the partial tile.
      if (row < rows && GU_IN_RANGE(row >= 0 && row < kTileM && half >= 0 && half < 2, kSiteSplitPart)) {
        float4* part = reinterpret_cast<float4*>(smem_gen + 4 * (static_cast<uint32_t>(row) * kSplitPitch + half * 64));
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          part[i] = make_float4(g[2 * i].x, g[2 * i].y, g[2 * i + 1].x, g[2 * i + 1].y);
          part[kTileN / 4 + i] = make_float4(u[2 * i].x, u[2 * i].y, u[2 * i + 1].x, u[2 * i + 1].y);
        }
      }
    }
  }
  __syncwarp();
  cluster_sync_all();  // every CTA's partial tile is in its shared memory

  if (warp >= 4) {
    // ---- finish this CTA's share of the token rows; a warp takes whole rows, a lane columns 4 lane .. 4 lane + 3 ----
    const int r_end = rows * (rank + 1) / splits;
    for (int r = rows * rank / splits + (warp - 4); r < r_end; r += 8) {
      float4 g = make_float4(0.f, 0.f, 0.f, 0.f), u = g;  // of the first and the second 128 accumulator columns
      if (GU_IN_RANGE(r >= 0 && r < rows && rows <= kTileM, kSiteSplitPart)) {
        const uint32_t local = ring + 4 * (static_cast<uint32_t>(r) * kSplitPitch + 4 * lane);
#pragma unroll 4
        for (int s = 0; s < splits; ++s) {  // ascending K
          const uint32_t src = mapa_shared(local, static_cast<uint32_t>(s));
          const float4 a = ld_shared_cluster_f32x4(src), b = ld_shared_cluster_f32x4(src + 4 * kTileN);
          g.x += a.x; g.y += a.y; g.z += a.z; g.w += a.w;
          u.x += b.x; u.y += b.y; u.z += b.z; u.w += b.w;
        }
      }
      const size_t m_global = static_cast<size_t>(mb) * kTileM + r;
      if (!GU_IN_RANGE(static_cast<long long>(m_global) < p.m && (kSingle ? 2 * nb : nb) < p.n_blocks128, kSiteSplitStore)) continue;
      if constexpr (kOp == kSplitGemm) {
        uint16_t* dst = static_cast<uint16_t*>(p.out) + m_global * p.ld_out + 2 * nb * kTileN + 4 * lane;
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(g.x, g.y), pack_bf16x2(g.z, g.w));
        if (2 * nb + 1 < p.n_blocks128)
          *reinterpret_cast<uint2*>(dst + kTileN) = make_uint2(pack_bf16x2(u.x, u.y), pack_bf16x2(u.z, u.w));
      } else {
        const uint32_t o01 = swiglu_bf16x2(make_float2(g.x, g.y), make_float2(u.x, u.y));
        const uint32_t o23 = swiglu_bf16x2(make_float2(g.z, g.w), make_float2(u.z, u.w));
        if constexpr (kOp == kSplitGateUp) {
          uint16_t* dst = static_cast<uint16_t*>(p.out) + m_global * p.ld_out + nb * kTileN + 4 * lane;
          *reinterpret_cast<uint2*>(dst) = make_uint2(o01, o23);
        } else {
          float amax = amax_bf16x2(amax_bf16x2(0.f, o01), o23);
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, d));
          const float sc = fmaxf(amax, 1e-12f) / 448.0f;
          const uint32_t q = e4m3x4_from_bf16x4(o01, o23, sc, __frcp_rn(sc));
          uint8_t* dst = static_cast<uint8_t*>(p.out) + m_global * p.ld_out + nb * kTileN + 4 * lane;
          *reinterpret_cast<uint32_t*>(dst) = q;
          if (lane == 0) p.scale_out[m_global * p.n_blocks128 + nb] = sc;
        }
      }
    }
  }

  // ------------------------------- teardown --------------------------------
  tc_fence_before();
  __syncwarp();
  if (*abort_gen) {
    // give copies that were already in flight time to land before shared memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) spin_backoff_ns(1000u);
  }
  __syncwarp();
  cluster_sync_all();  // no CTA leaves while another may still read its partial tile
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, kTileTmemCols);
}

}  // namespace gu
