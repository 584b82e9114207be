// CTA-pair tcgen05 GEMM for sm_100a:  out[M, N] = epilogue( x[M, K] . w[N, K]^T ), both operands K-major.
//
// Two SMs work on one output tile with tcgen05.mma.cta_group::2: 256 output channels (the weight is the
// 256-row A operand, 128 rows per CTA) x `bn` tokens (the activation is the B operand, bn / 2 rows per CTA).
// Why a pair: an SM then takes in 16 KiB of weight + 64 bn bytes of activation per 128-byte K block, where a
// 128x256 tile of its own took 48 KiB.  Why the tokens are the N side: bn is a run-time multiple of 32, so a ragged
// token count is cut into equal tiles (777 tokens: 4 x 224 instead of 7 x 128) and the width is chosen for full
// waves (pair_pick).  What bounds it: wide tiles the tensor cores (0.37 us per K block of 256 x 256, the library's
// rate too), narrow ones the ring's round trip of ~1.3 us, small problems the ~4 us of launch, fill and epilogue.
// Measured against one CTA per 128x256 / 128x128 tile with a one-lane producer and issuer (N x K of Llama-3.1-8B's
// qkv / o / gate_up / down, weights from HBM, us before -> now): e4m3 M 300: 14.9 / 13.3 / 46.8 / 37.8 -> 11.3 / 9.7 /
// 35.9 / 21.5; e4m3 M 2048: 44.8 / 30.7 / 194 / 93.3 -> 39.3 / 27.8 / 174 / 85.0; bf16 M 777: 54.5 / 42.4 / 163 / 129 ->
// 34.2 / 25.3 / 142 / 73.2.
//
//   warp 0    TMA producer, in both CTAs; the bytes of both are credited to the leader's full barrier
//   warp 1    MMA issuer (leader only); commits multicast to both CTAs' empty / accumulator barriers
//   warps 2-9 epilogue: TMEM lane = output channel, column = token; 32 tokens at a time are scaled, rounded
//             and turned through shared memory so that the stores are 16-byte and coalesced
//
// splits > 1 (few tiles): a cluster holds `splits` pairs, each a slice of K of the same tile; the fp32 partials
// are parked in the idle operand ring and summed over distributed shared memory in rank order (deterministic).
// Every wait is bounded (tc::mbar_wait_bounded).
#pragma once
#include "gemm_tc.cuh"

namespace b200 {

struct PairParams {
  void* out;            // [M, N] OutT, row stride ldc
  int64_t ldc;
  const float* sa;      // per-token scale (stride sa_stride, 0 = one for all) or null
  const float* sb;      // per-channel scale (stride sb_stride) or null
  int sa_stride, sb_stride;
  const void* bias;     // [N] OutT or null
  int M, N, K;
  int bn;               // tokens of a tile: a multiple of 32, at most 256
  int stages;           // operand ring
  int splits, kb_per_split;
  int vec_ok;           // rows of `out` take 16-byte stores
  int early_w;          // the first weight tiles may be read before the dependency wait
  float act_pos, act_neg;
  int* wait_error;      // tc::report_gave_up
};

constexpr int kPairMaxStages = 10, kPairMaxSplits = 4;
constexpr int kPairThreads = 320;
constexpr int kPairStageRow = 144;                       // bytes of a staged token pair: 32 channels + padding
constexpr int kPairStageWarp = 16 * kPairStageRow;       // 32 tokens
constexpr int kPairFixedBytes = 1024 + 8 * kPairStageWarp + 2 * 256 * 4 + (2 * kPairMaxStages + 4) * 8 + 16;
constexpr int kPairSmemMax = 227 * 1024;

namespace tc {
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* m, uint32_t leader_bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(c0), "r"(c1)
      : "memory");
}
template <bool F16>
__device__ __forceinline__ void mma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  if (F16)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(bar),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n"
               "tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::"r"(slot), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t remote_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(remote_bar) : "memory");
}
}  // namespace tc

template <int KIND, typename OutT, bool ACT = false>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                 const PairParams p) {
  constexpr int ELT = GemmKindTraits<KIND>::ELT;
  constexpr int BLOCK_K = 128 / ELT;
  constexpr int W_BYTES = 128 * 128;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // the same offset in every CTA
  const int x_bytes = p.bn * 64;
  const int stage_bytes = W_BYTES + x_bytes;                     // whole 1 KiB swizzle atoms: bn is a multiple of 32
  const uint32_t stg = base + p.stages * stage_bytes;            // staged output, one part per epilogue warp
  const uint32_t sa_at = stg + 8 * kPairStageWarp;               // [2][256] token scales
  const uint32_t bars = sa_at + 2 * 256 * 4;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (kPairMaxStages + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * kPairMaxStages + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * kPairMaxStages + 2 + a); };
  const uint32_t tmem_slot = bars + 8u * (2 * kPairMaxStages + 4), gave_up = tmem_slot + 4;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const uint32_t half = crank & 1u;                // which CTA of the pair; 0 leads
  const uint16_t pair_mask = static_cast<uint16_t>(3u << (crank & ~1u));
  const int S = p.splits;
  const int ks = static_cast<int>(crank >> 1);     // K slice of this pair
  const int cluster_id = static_cast<int>(blockIdx.x) / (2 * S);
  const int clusters = static_cast<int>(gridDim.x) / (2 * S);

  const int tok_blocks = ceil_div(p.M, p.bn);
  const int num_tiles = tok_blocks * ceil_div(p.N, 256);
  const int num_kb = ceil_div(p.K, BLOCK_K);
  const int kb0 = S > 1 ? ks * p.kb_per_split : 0;
  const int kb1 = S > 1 ? min(num_kb, kb0 + p.kb_per_split) : num_kb;

  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmap_w);
    tc::prefetch_tmap(&tmap_x);
    for (int s = 0; s < p.stages; ++s) {
      tc::mbar_init(full_bar(s), 1);
      tc::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < 2; ++a) {
      tc::mbar_init(tfull_bar(a), 1);
      tc::mbar_init(tempty_bar(a), 16);            // the epilogue warps of both CTAs
    }
    asm volatile("st.shared.u32 [%0], 0;\n" ::"r"(gave_up) : "memory");
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc_pair(tmem_slot, 512);
  tc::tc_fence_before();
  __syncthreads();
  cluster_sync_all();                              // the pair's barriers exist before anything targets them
  tc::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  // where the weight does not depend on the previous kernel, its first stages are requested before the dependency wait
  int w_ahead = 0;
  const uint32_t stage_tx = 2u * (W_BYTES + x_bytes);
  if (warp == 0 && cluster_id < num_tiles && p.early_w) {
    const int n_row = (cluster_id / tok_blocks) * 256 + static_cast<int>(half) * 128;
    w_ahead = min(p.stages, kb1 - kb0);
    if (tc::elect_one()) {
      for (int i = 0; i < w_ahead; ++i) {
        if (half == 0) tc::mbar_arrive_expect_tx(full_bar(i), stage_tx);
        tc::tma_load_2d_pair(base + i * stage_bytes, &tmap_w, map_to_rank(full_bar(i), crank & ~1u),
                             (kb0 + i) * BLOCK_K, n_row);
      }
    }
    __syncwarp();
  }
  griddep_wait();
  griddep_launch_dependents();
  bool dead = false;                               // a wait of this thread ran out: the rest only poll

  // Producer and issuer loops run on whole warps and elect a thread only for the instructions themselves: inside
  // a one-lane branch the operands of TMA and tcgen05 instructions are not known to be warp-uniform, and moving
  // them cost ~600 clocks per K block (0.305 us at any tile width, 4 stages or 10).
  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t bar0 = map_to_rank(bars, crank & ~1u);      // the leader's full barriers
    for (int tile = cluster_id; tile < num_tiles; tile += clusters) {
      const int n_row = (tile / tok_blocks) * 256 + static_cast<int>(half) * 128;
      const int t_row = (tile % tok_blocks) * p.bn + static_cast<int>(half) * (p.bn / 2);
      for (int kb = kb0; kb < kb1; ++kb) {
        const uint32_t at = base + stage * stage_bytes;
        const bool ahead = w_ahead > 0;
        if (ahead)
          --w_ahead;
        else
          tc::mbar_wait_bounded(empty_bar(stage), phase ^ 1u, dead, gave_up);
        if (tc::elect_one()) {
          if (!ahead) {
            if (half == 0) tc::mbar_arrive_expect_tx(full_bar(stage), stage_tx);
            tc::tma_load_2d_pair(at, &tmap_w, bar0 + 8u * stage, kb * BLOCK_K, n_row);
          }
          tc::tma_load_2d_pair(at + W_BYTES, &tmap_x, bar0 + 8u * stage, kb * BLOCK_K, t_row);
        }
        __syncwarp();
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    for (int i = 0; i < p.stages; ++i) {           // every commit that targets this CTA has arrived
      tc::mbar_wait_bounded(empty_bar(stage), phase ^ 1u, dead, gave_up);
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    if (half == 0) {
      const uint32_t idesc = tc::make_idesc(GemmKindTraits<KIND>::FMT, GemmKindTraits<KIND>::FMT, 256, p.bn, 0, 0);
      int stage = 0, local = 0;
      uint32_t phase = 0;
      for (int tile = cluster_id; tile < num_tiles; tile += clusters, ++local) {
        const int acc = local & 1;
        tc::mbar_wait_bounded(tempty_bar(acc), ((local >> 1) & 1u) ^ 1u, dead, gave_up);
        tc::tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * 256;
        for (int kb = kb0; kb < kb1; ++kb) {
          tc::mbar_wait_bounded(full_bar(stage), phase, dead, gave_up);
          tc::tc_fence_after();
          const uint64_t adesc = tc::make_smem_desc_sw128(base + stage * stage_bytes, 1024, 16);
          const uint64_t bdesc = tc::make_smem_desc_sw128(base + stage * stage_bytes + W_BYTES, 1024, 16);
          if (tc::elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k)            // 32 bytes of K further on: 2 in the address field
              tc::mma_pair<KIND != kKindFp8>(tmem_d, adesc + 2 * k, bdesc + 2 * k, idesc, kb != kb0 || k != 0 ? 1u : 0u);
            tc::commit_pair(empty_bar(stage), pair_mask);
          }
          __syncwarp();
          if (++stage == p.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (tc::elect_one()) tc::commit_pair(tfull_bar(acc), pair_mask);
        __syncwarp();
      }
    }
  } else {
    const int quarter = warp & 3;                  // TMEM lanes this warp may read
    const int col_half = (warp - 2) >> 2;          // the two warps of a quarter share the tokens
    OutT* out = static_cast<OutT*>(p.out);
    const uint32_t my_stage = stg + (warp - 2) * kPairStageWarp;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    // NT tokens (first column c0 of the tile) x the 32 channels of this warp -> out.  Two tokens of a channel are
    // one staged word; a lane reads back 8 channels of a token pair and stores 16 bytes of each token.
    auto emit = [&](auto nt, const float* v, uint32_t sa_addr, int c0, int tok0, int chan, float sb, float bias) {
      constexpr int NT = decltype(nt)::value;
      uint32_t packed[NT / 2];
#pragma unroll
      for (int j = 0; j < NT; j += 4) {
        const uint4 s4 = lds128(sa_addr + (c0 + j) * 4);
        float y[4] = {fmaf(v[j], __uint_as_float(s4.x) * sb, bias), fmaf(v[j + 1], __uint_as_float(s4.y) * sb, bias),
                      fmaf(v[j + 2], __uint_as_float(s4.z) * sb, bias), fmaf(v[j + 3], __uint_as_float(s4.w) * sb, bias)};
        if (ACT) {
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] = xielu_fast(y[e], p.act_pos, p.act_neg);
        }
        packed[j / 2] = pack_out2<OutT>(y[0], y[1]);
        packed[j / 2 + 1] = pack_out2<OutT>(y[2], y[3]);
      }
      const int chan0 = chan - lane;               // first channel of the warp
      if (p.vec_ok && chan0 + 32 <= p.N) {
        __syncwarp();                              // the previous chunk has been read back
#pragma unroll
        for (int j = 0; j < NT / 2; ++j)
          asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(my_stage + j * kPairStageRow + lane * 4), "r"(packed[j]) : "memory");
        __syncwarp();
#pragma unroll
        for (int i = 0; i < NT / 16; ++i) {
          const int row = i * 8 + (lane >> 2), c = lane & 3;
          const uint4 lo = lds128(my_stage + row * kPairStageRow + c * 32);
          const uint4 hi = lds128(my_stage + row * kPairStageRow + c * 32 + 16);
          const int t = tok0 + c0 + 2 * row;
          OutT* dst = out + static_cast<int64_t>(t) * p.ldc + chan0 + c * 8;
          if (t < p.M)
            *reinterpret_cast<uint4*>(dst) = make_uint4(__byte_perm(lo.x, lo.y, 0x5410), __byte_perm(lo.z, lo.w, 0x5410),
                                                        __byte_perm(hi.x, hi.y, 0x5410), __byte_perm(hi.z, hi.w, 0x5410));
          if (t + 1 < p.M)
            *reinterpret_cast<uint4*>(dst + p.ldc) = make_uint4(__byte_perm(lo.x, lo.y, 0x7632), __byte_perm(lo.z, lo.w, 0x7632),
                                                                __byte_perm(hi.x, hi.y, 0x7632), __byte_perm(hi.z, hi.w, 0x7632));
        }
      } else if (chan < p.N) {                     // ragged channels or unaligned rows: 2-byte stores
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int t = tok0 + c0 + j;
          const uint16_t w = static_cast<uint16_t>(packed[j / 2] >> (16 * (j & 1)));
          if (t < p.M) *reinterpret_cast<uint16_t*>(out + static_cast<int64_t>(t) * p.ldc + chan) = w;
        }
      }
    };
    int local = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += clusters, ++local) {
      const int acc = local & 1;
      const int chan = (tile / tok_blocks) * 256 + static_cast<int>(half) * 128 + quarter * 32 + lane;
      const int tok0 = (tile % tok_blocks) * p.bn;
      const uint32_t sa_addr = sa_at + acc * 1024;
      for (int c = static_cast<int>(threadIdx.x) - 64; c < p.bn; c += 256) {
        const float v = p.sa && tok0 + c < p.M ? __ldg(p.sa + static_cast<int64_t>(tok0 + c) * p.sa_stride) : 1.0f;
        asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(sa_addr + c * 4), "f"(v) : "memory");
      }
      const float sb = p.sb && chan < p.N ? __ldg(p.sb + static_cast<int64_t>(chan) * p.sb_stride) : 1.0f;
      const float bias = p.bias && chan < p.N ? to_float<OutT>(static_cast<const OutT*>(p.bias)[chan]) : 0.0f;
      named_bar_sync_gemm(1, 256);                 // scales of this tile are in place
      tc::mbar_wait_bounded(tfull_bar(acc), (local >> 1) & 1u, dead, gave_up);
      tc::tc_fence_after();
      __syncwarp();
      if (S > 1) {
        // park the slice's fp32 partial in the idle ring as [token][channel], sum the slices in rank order
        const uint32_t part = base + (quarter * 32 + lane) * 4;
#pragma unroll 1
        for (int c = col_half * 16; c < p.bn; c += 32) {
          uint32_t r[16];
          tc::tmem_ld16(tmem_base + lane_addr + c, r);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j)
            asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(part + (c + j) * 512), "r"(r[j]) : "memory");
        }
        tc::tc_fence_before();
        __syncwarp();
        cluster_sync_all();
        for (int g = ks * 2 + col_half; g < p.bn / 16; g += 2 * S) {
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0.f;
          for (int q = 0; q < S; ++q) {
            const uint32_t src = map_to_rank(part + g * 16 * 512, 2 * q + half);
            float t[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) t[j] = ld_cluster_f32(src + j * 512);
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] += t[j];
          }
          emit(std::integral_constant<int, 16>{}, v, sa_addr, g * 16, tok0, chan, sb, bias);
        }
        __syncwarp();
        cluster_sync_all();                        // the peers have read this partial
        continue;
      }
      // 32 tokens at a time, the next ones on their way from tensor memory meanwhile
      const uint32_t acc_addr = tmem_base + lane_addr + acc * 256;
      uint32_t r[2][32];
      if (col_half * 32 < p.bn) tc::tmem_ld32(acc_addr + col_half * 32, r[0]);
#pragma unroll 1
      for (int c = col_half * 32; c < p.bn; c += 128) {
        tc::tmem_ld_wait();
        if (c + 64 < p.bn) tc::tmem_ld32(acc_addr + c + 64, r[1]);
        emit(std::integral_constant<int, 32>{}, reinterpret_cast<const float*>(r[0]), sa_addr, c, tok0, chan, sb, bias);
        if (c + 64 < p.bn) {
          tc::tmem_ld_wait();
          if (c + 128 < p.bn) tc::tmem_ld32(acc_addr + c + 128, r[0]);
          emit(std::integral_constant<int, 32>{}, reinterpret_cast<const float*>(r[1]), sa_addr, c + 64, tok0, chan, sb, bias);
        }
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive_cluster(map_to_rank(tempty_bar(acc), crank & ~1u));
    }
  }
  if (S > 1 && warp < 2) {                         // the two barriers of the reduction (one tile per cluster)
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc::tc_fence_before();
  __syncwarp();
  cluster_sync_all();                              // the peer may still signal this CTA's barriers
  if (warp == 1) {
    tc::report_gave_up(gave_up, p.wait_error);
    tc::tmem_dealloc_pair(tmem_base, 512);
  }
}

struct PairPlan {
  int bn = 0, splits = 1, kb_per_split = 0, stages = 0, smem = 0;
};

// Ring depth for a tile width, and the shared memory it takes.
inline int pair_stages(int bn, int* smem) {
  const int stage = 128 * 128 + bn * 64;
  int s = (kPairSmemMax - kPairFixedBytes) / stage;
  if (s > kPairMaxStages) s = kPairMaxStages;
  *smem = kPairFixedBytes + s * stage;
  return s;
}

// Tile width and K split for M tokens; clusters_of[s]: clusters of s pairs that are resident at once.
// Estimated microseconds, from B200 measurements (e4m3, N 4096, K 4096 and 20480, 64 pairs): a 128-byte K block
// takes 0.131 / 0.147 / 0.203 / 0.245 / 0.287 / 0.373 at 32 / 64 / 128 / 160 / 192 / 256 tokens (narrow tiles wait
// for the ring, wide ones for the tensor cores), a launch 4 + bn / 250, a split 2 + bn / 125 for the exchange of
// the partials (e4m3, 512 x 4096 x 14336: 27.9 in two slices of 256 tokens, 26.3 in unsplit tiles of 128).  So one
// wave of narrow tiles beats two of wide ones, and a split pays where most pairs would idle; a narrower tile or a
// split has to promise 5 %, since it reads more and the estimate is not better than that.  Over 352 problems of 512 to
// 6000 tokens timed at six widths the pick is 0.3 % slower than the best of them, 7 % at most (wide tiles only from
// 2048 tokens on: 6.0 %, up to 55 %; us, 256 tokens / the pick: bf16 2048 x 896 x 896 10.8 / 8.2, 4096 x 3584 x 5120 108
// / 100, 2300 x 896 x 4864 29.1 / 18.7).
inline PairPlan pair_pick(int M, int N, int num_kb, const int* clusters_of) {
  const int n_blocks = ceil_div(N, 256);
  PairPlan best;
  double best_us = 0;
  for (int nb = ceil_div(M, 256); nb <= ceil_div(M, 32) && nb <= ceil_div(M, 256) + 12; ++nb) {
    const int bn = (ceil_div(M, nb) + 31) / 32 * 32;
    const int64_t tiles = static_cast<int64_t>(ceil_div(M, bn)) * n_blocks;
    const double wide = 0.040 + 0.0013 * bn, narrow = 0.115 + 0.0005 * bn;
    const double per_kb = wide > narrow ? wide : narrow;
    for (int S = 1; S <= kPairMaxSplits; ++S) {
      if (clusters_of[S] <= 0) continue;
      const int per = ceil_div(num_kb, S);
      if (S > 1 && (tiles > clusters_of[S] || per < 4 || (S - 1) * per >= num_kb)) continue;
      const int64_t waves = S > 1 ? 1 : (tiles + clusters_of[1] - 1) / clusters_of[1];
      const double us = waves * (per * per_kb + 0.3) + 4.0 + bn / 250.0 + (S > 1 ? 2.0 + 0.008 * bn : 0.0);
      if (best.bn == 0 || us < 0.95 * best_us) {
        best.bn = bn;
        best.splits = S;
        best.kb_per_split = per;
        best_us = us;
      }
    }
  }
  best.stages = pair_stages(best.bn, &best.smem);
  return best;
}

// Clusters of S pairs that are resident at once on the current device (0: none).
template <int KIND, typename OutT, bool ACT>
int pair_clusters(int S) {
  static std::atomic<int> cached[64][kPairMaxSplits + 1];
  auto kern = gemm_pair_kernel<KIND, OutT, ACT>;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = cached[dev][S].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * S * 8);
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmemMax;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemMax) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = -1;
    }
    cached[dev][S].store(n, std::memory_order_relaxed);
  }
  return n > 0 ? n : 0;
}

// old_weight: the launch just before this one does not write w, whose first tiles are read before the dependency wait up
// to pdl_max_tokens() tokens; above, w is read after it.
template <int KIND, typename OutT, bool ACT = false>
int launch_gemm_pair(const void* x, int64_t ldx, const void* w, int64_t ldw, const GemmEpilogueParams& ep,
                     cudaStream_t st, const char* timer_name, bool old_weight = true) {
  constexpr int ELT = GemmKindTraits<KIND>::ELT;
  int clusters_of[kPairMaxSplits + 1] = {0};
  for (int s = 1; s <= kPairMaxSplits; ++s) clusters_of[s] = pair_clusters<KIND, OutT, ACT>(s);
  B200_REQUIRE(clusters_of[1] > 0, "gemm_pair_kernel: no pair of CTAs is resident on this device");
  const PairPlan plan = pair_pick(ep.M, ep.N, ceil_div(ep.K, 128 / ELT), clusters_of);
  CUtensorMap tw, tx;
  int rc = make_tmap_2d(&tw, w, ep.N, ep.K, ldw * ELT, 128, 128 / ELT, ELT, true);
  if (rc) return rc;
  rc = make_tmap_2d(&tx, x, ep.M, ep.K, ldx * ELT, plan.bn / 2, 128 / ELT, ELT, false);
  if (rc) return rc;
  PairParams p;
  p.out = ep.out;
  p.ldc = ep.ldc;
  p.sa = ep.sa;
  p.sb = ep.sb;
  p.sa_stride = ep.sa_stride;
  p.sb_stride = ep.sb_stride;
  p.bias = ep.bias;
  p.M = ep.M;
  p.N = ep.N;
  p.K = ep.K;
  p.bn = plan.bn;
  p.stages = plan.stages;
  p.splits = plan.splits;
  p.kb_per_split = plan.kb_per_split;
  p.vec_ok = ep.ldc % 8 == 0 && aligned16(ep.out);
  const int family = old_weight ? pdl_gemm_family(ep.M, kPdlGemmBig) : 0;
  p.early_w = family == 0 || ep.M <= pdl_max_tokens();
  p.act_pos = ep.act_pos;
  p.act_neg = ep.act_neg;
  rc = wait_error_arm(timer_name, &p.wait_error);
  if (rc) return rc;
  const int tiles = ceil_div(ep.M, plan.bn) * ceil_div(ep.N, 256);
  const int clusters = plan.splits > 1 || tiles < clusters_of[1] ? tiles : clusters_of[1];
  note_variant("gemm_tn kind=%d bn=%d stages=%d splits=%d out=%s grid=%d", KIND, plan.bn, plan.stages, plan.splits,
               std::is_same<OutT, __half>::value ? "f16" : "bf16", clusters * 2 * plan.splits);
  {
    ScopedKernelTimer timer(timer_name, st);
    B200_CUDA_OK(launch_kernel(gemm_pair_kernel<KIND, OutT, ACT>, dim3(clusters * 2 * plan.splits), dim3(kPairThreads),
                               plan.smem, st, 2 * plan.splits, family, tw, tx, p));
  }
  B200_CHECK_LAUNCH("gemm_pair_kernel");
  return 0;
}

}  // namespace b200
