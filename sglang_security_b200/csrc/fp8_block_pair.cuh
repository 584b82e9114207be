// CTA-pair form of the block-scaled FP8 GEMM (fp8_block_gemm.cu) for large problems.
//
// Two SMs work on 256 tokens x 256 channels with tcgen05.mma.cta_group::2: each CTA brings its 128 tokens (A) and half of
// the channels (B), 32 KiB per K block of 128 where a 128 x 256 tile of its own takes 48 KiB (0.50 us a block, which is
// what L2 gives an SM), and drains its own 128 x 256 partial sums as the single-CTA kernel does: a thread owns one token
// and 128 channels of one weight scale block, so the combined scale is one number a block.
// The two 128-channel halves are MMAs of their own (N = 128) with their own accumulator barriers: an epilogue warpgroup
// starts, and gives its accumulator back, a quarter of a block's time earlier (whole 256-channel MMAs: 3 to 6 % slower).
// The epilogue's arrival at the leader is mbarrier.arrive with its default order: with .release.cluster, a fence that waits
// for all the warp's copies, every block took 1.15 us instead of 0.45.
// What bounds it: the chain from one block's MMAs through the epilogue to the leave to overwrite (0.45 us a block; 0.37 in
// gemm_pair_kernel, which has none), then the power cap.  Single-CTA tiles / this, us: 2048 x 28672 x 4096 235 / 214,
// 4096 x 14336 119 / 106; 3001 tokens 348 / 314 and 178 / 160 (before the scale ring 381 and 237).
#pragma once
#include "gemm_pair.cuh"

namespace b200 {

constexpr int kBlkPairStages = 6;
constexpr int kBlkPairStageBytes = 2 * 128 * 128;       // A 128 x 128, B 128 x 128
constexpr int kBlkPairRow = 48;                         // bytes of a staged output row: 16 channels + padding
constexpr int kBlkPairSmem = 1024 + kBlkPairStages * kBlkPairStageBytes + 8 * 32 * kBlkPairRow +
                             kBlkScaleSlots * kBlkScaleBytes + (2 * kBlkPairStages + 8) * 8 + 16;
static_assert(kBlkPairSmem <= kPairSmemMax, "one CTA per SM");

namespace tc {
__device__ __forceinline__ void mbar_arrive_peer(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
}  // namespace tc
template <typename OutT>
__global__ void __launch_bounds__(kBlkThreads, 1)
fp8_block_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const BlockGemmParams p) {
  constexpr int STAGES = kBlkPairStages, STAGE_BYTES = kBlkPairStageBytes, A_BYTES = 128 * 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // the same offset in both CTAs
  const uint32_t stg = base + STAGES * STAGE_BYTES;
  const uint32_t scl = stg + 8 * 32 * kBlkPairRow;
  const uint32_t bars = scl + kBlkScaleSlots * kBlkScaleBytes;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 4 + a); };
  const uint32_t tmem_slot = bars + 8u * (2 * STAGES + 8), gave_up = tmem_slot + 4;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t half = cluster_ctarank();              // which CTA of the pair; 0 leads
  const int cluster_id = static_cast<int>(blockIdx.x) >> 1, clusters = static_cast<int>(gridDim.x) >> 1;
  const int m_blocks = ceil_div(p.M, 256);
  const int num_tiles = m_blocks * ceil_div(p.N, 256);
  const int num_kb = ceil_div(p.K, 128);
  bool dead = false;                                    // a wait of this thread ran out: the rest only poll

  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmap_a);
    tc::prefetch_tmap(&tmap_b);
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(full_bar(s), 1);
      tc::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 4; ++a) {
      tc::mbar_init(tfull_bar(a), 2);              // the MMAs' commit and the scale warp
      tc::mbar_init(tempty_bar(a), 8);             // four epilogue warps of each CTA
    }
    asm volatile("st.shared.u32 [%0], 0;\n" ::"r"(gave_up) : "memory");
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc_pair(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                   // the pair's barriers exist before anything targets them
  tc::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  griddep_wait();
  griddep_launch_dependents();

  // whole-warp loops, one elected thread per instruction (see gemm_pair.cuh)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" :: "n"(kBlkOtherRegs));
    if (warp == 0) {
      int stage = 0;
      uint32_t phase = 0;
      const uint32_t bar0 = map_to_rank(bars, 0);         // the leader's full barriers
      for (int tile = cluster_id; tile < num_tiles; tile += clusters) {
        const int m_row = (tile % m_blocks) * 256 + static_cast<int>(half) * 128;
        const int n_row = (tile / m_blocks) * 256 + static_cast<int>(half) * 64;
        for (int kb = 0; kb < num_kb; ++kb) {
          tc::mbar_wait_bounded(empty_bar(stage), phase ^ 1u, dead, gave_up);
          const uint32_t at = base + stage * STAGE_BYTES;
          if (tc::elect_one()) {
            if (half == 0) tc::mbar_arrive_expect_tx(full_bar(stage), 2u * STAGE_BYTES);
            tc::tma_load_2d_pair(at, &tmap_a, bar0 + 8u * stage, kb * 128, m_row);
            tc::tma_load_2d_pair(at + A_BYTES, &tmap_b, bar0 + 8u * stage, kb * 128, n_row);
            tc::tma_load_2d_pair(at + A_BYTES + A_BYTES / 2, &tmap_b, bar0 + 8u * stage, kb * 128, n_row + 128);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      for (int i = 0; i < STAGES; ++i) {                  // every commit that targets this CTA has arrived
        tc::mbar_wait_bounded(empty_bar(stage), phase ^ 1u, dead, gave_up);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    } else if (warp == 1 && half == 0) {
      constexpr uint32_t idesc = tc::make_idesc(0, 0, 256, 128, 0, 0);
      int stage = 0;
      uint32_t phase = 0, it = 0;
      for (int tile = cluster_id; tile < num_tiles; tile += clusters) {
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int buf = it & 1;
          const uint32_t buf_phase = (it >> 1) & 1u;
          tc::mbar_wait_bounded(full_bar(stage), phase, dead, gave_up);
          const uint64_t adesc = tc::make_smem_desc_sw128(base + stage * STAGE_BYTES, 1024, 16);
          const uint64_t bdesc = tc::make_smem_desc_sw128(base + stage * STAGE_BYTES + A_BYTES, 1024, 16);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int acc = buf * 2 + h;
            tc::mbar_wait_bounded(tempty_bar(acc), buf_phase ^ 1u, dead, gave_up);
            tc::tc_fence_after();
            if (tc::elect_one()) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                tc::mma_pair<false>(tmem_base + buf * 256 + h * 128, adesc + 2 * k, bdesc + h * (A_BYTES / 2 / 16) + 2 * k, idesc,
                                    k != 0 ? 1u : 0u);
              if (h == 1) tc::commit_pair(empty_bar(stage), 3);
              tc::commit_pair(tfull_bar(acc), 3);
            }
            __syncwarp();
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    } else if (warp == 2) {
      feed_block_scales(
          p, scl, cluster_id, num_tiles, clusters, 0, num_kb, lane,
          [&](int tile, int& row0, int& blk) {
            row0 = (tile % m_blocks) * 256 + static_cast<int>(half) * 128;
            blk = (tile / m_blocks) * 2 + (lane & 1);
          },
          [&](uint32_t it) {
            const int acc = (it & 1) * 2;
            const uint32_t before = ((it >> 1) & 1u) ^ 1u;
            tc::mbar_wait_bounded(tfull_bar(acc), before, dead, gave_up);
            tc::mbar_wait_bounded(tfull_bar(acc + 1), before, dead, gave_up);
            if (lane < 2) tc::mbar_arrive(tfull_bar(acc + lane));
          });
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" :: "n"(kBlkEpilogueRegs));
    const int quarter = warp & 3;                       // TMEM lanes this warp may read
    const int g = (warp - 4) >> 2;                      // which 128 channels of the tile
    OutT* out = static_cast<OutT*>(p.out);
    const OutT* bias = static_cast<const OutT*>(p.bias);
    const uint32_t lane_addr = (static_cast<uint32_t>(quarter * 32) << 16) + g * 128;
    const uint32_t my_stage = stg + (warp - 4) * 32 * kBlkPairRow;
    const uint32_t tempty0 = map_to_rank(tempty_bar(g), 0);   // the leader's
    uint32_t it = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += clusters) {
      const int row0 = (tile % m_blocks) * 256 + static_cast<int>(half) * 128 + quarter * 32;
      const int col0 = (tile / m_blocks) * 256 + g * 128;
      float2 acc[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = make_float2(0.f, 0.f);
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int buf = it & 1;
        tc::mbar_wait_bounded(tfull_bar(buf * 2 + g), (it >> 1) & 1u, dead, gave_up);
        tc::tc_fence_after();
        const float s = block_scale(scl, it, quarter * 32 + lane, g);
        const float2 s2 = make_float2(s, s);
        const uint32_t taddr = tmem_base + lane_addr + buf * 256;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t r[16];
          tc::tmem_ld16(taddr + c * 16, r);
          tc::tmem_ld_wait();
          if (c == 7) {                                 // the whole partial is in registers: hand the buffer back before the math
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive_peer(tempty0 + buf * 16);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[c * 8 + j] = ffma2(make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), s2, acc[c * 8 + j]);
        }
      }
      if (bias) {
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          if (col0 + 2 * j < p.N) acc[j].x += to_float<OutT>(bias[col0 + 2 * j]);
          if (col0 + 2 * j + 1 < p.N) acc[j].y += to_float<OutT>(bias[col0 + 2 * j + 1]);
        }
      }
      // 16 channels at a time through shared memory: a store then covers 32 bytes of a row, not 16
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int cc = col0 + c * 16;
        if (p.vec_ok && cc + 16 <= p.N) {
          __syncwarp();
#pragma unroll
          for (int v = 0; v < 2; ++v)
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(my_stage + lane * kBlkPairRow + v * 16),
                         "r"(pack_out2<OutT>(acc[c * 8 + v * 4].x, acc[c * 8 + v * 4].y)),
                         "r"(pack_out2<OutT>(acc[c * 8 + v * 4 + 1].x, acc[c * 8 + v * 4 + 1].y)),
                         "r"(pack_out2<OutT>(acc[c * 8 + v * 4 + 2].x, acc[c * 8 + v * 4 + 2].y)),
                         "r"(pack_out2<OutT>(acc[c * 8 + v * 4 + 3].x, acc[c * 8 + v * 4 + 3].y))
                         : "memory");
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int r = i * 16 + (lane >> 1), v = lane & 1;
            const uint4 w = lds128(my_stage + r * kBlkPairRow + v * 16);
            if (row0 + r < p.M) *reinterpret_cast<uint4*>(out + static_cast<int64_t>(row0 + r) * p.ldc + cc + v * 8) = w;
          }
        } else if (row0 + lane < p.M) {
          OutT* orow = out + static_cast<int64_t>(row0 + lane) * p.ldc;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (cc + 2 * j < p.N) orow[cc + 2 * j] = from_float<OutT>(acc[c * 8 + j].x);
            if (cc + 2 * j + 1 < p.N) orow[cc + 2 * j + 1] = from_float<OutT>(acc[c * 8 + j].y);
          }
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncwarp();
  cluster_sync_all();                                   // the peer may still signal this CTA's barriers
  if (warp == 1) {
    tc::report_gave_up(gave_up, p.wait_error);
    tc::tmem_dealloc_pair(tmem_base, 512);
  }
}

}  // namespace b200
