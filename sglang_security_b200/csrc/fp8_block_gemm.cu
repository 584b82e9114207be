// Block-scaled FP8 GEMM (DeepSeek-style 128x128 weight blocks, 1x128 activation groups) on tcgen05.
// Replaces sgl-kernel fp8_blockwise_scaled_mm (sgl-kernel/csrc/gemm/fp8_blockwise_gemm_kernel.cu:
// 345-423) and the Triton _w8a8_block_fp8_matmul (python/sglang/srt/layers/quantization/
// fp8_kernel.py:435-517):
//   C[m,n] = sum_kb ( A[m, kb] . B[n, kb]^T ) * As[m, kb] * Bs[n/128, kb]      (fp32), then cast
//
// The fp32 scales differ per 128-wide K block, so they cannot ride inside one tensor-core
// accumulation.  Each K block is therefore multiplied into a FRESH TMEM accumulator (2 rotating
// 256-column buffers); the eight epilogue warps pull the finished partial tile out of TMEM and
// "promote" it into fp32 registers with one packed FMA per element pair:
//   acc[m, :] += (As[m,kb] * Bs[nb,kb]) * partial[m, :]
// (a warpgroup owns 128 columns = one weight scale block, so the combined scale is a per-thread scalar) while
// the MMA warp already works on the next K blocks.  TMA / mbarrier ring and issue loops as in gemm_pair.cuh.
#include "fp8_gemm_smallm.cuh"

namespace b200 {

struct BlockGemmParams {
  void* out;
  int64_t ldc;
  const float* as;      // [M, K/128] element (m, kb) at as[m * as_row + kb * as_col]
  int64_t as_row, as_col;
  const float* bs;      // [ceil(N/128), ceil(K/128)] row-major, row stride bs_row
  int64_t bs_row;
  const void* bias;
  int M, N, K;
  // few tiles: a cluster of `splits` CTAs takes one tile, each a slice of K; see the epilogue
  int splits, kb_per_split;
  int* wait_error;  // tc::report_gave_up
  int vec_ok;       // rows of `out` take 16-byte stores
};

// The scales of a K block (128 token scales, one of each of the tile's two weight blocks) travel through a ring in shared
// memory that a warp of its own fills AHEAD blocks early.  Its arrival is part of the accumulator's barrier: that phase is
// over when the MMAs have ended and the block's scales are in place, so the epilogue has one wait a block and reads them
// beside tensor memory.  Read from global memory by the epilogue, as before, they were an exposed round trip a block
// (e4m3, us: 3001 x 28672 x 4096 362, 310 with the ring and the pair; 4096 x 14336 228 and 152), and a barrier of their
// own cost 7 % of what was left.
// Reuse: block it + AHEAD is written once block it - NBUF's phase is over.  Those MMAs were issued after the epilogue had
// given back the accumulator of block it - 2 NBUF, whose scales it had read by then: 2 NBUF + AHEAD <= SLOTS.
constexpr int kBlkScaleSlots = 16, kBlkScaleAhead = 8;
constexpr int kBlkScaleBytes = (128 + 4) * 4;
constexpr int kBlkThreads = 384;   // TMA, MMA, scales, one idle; 2 x 4 epilogue warps
// a K block's sums are 128 registers a thread at most: 128 x 88 + 256 x 208 <= 384 x 168 at launch
constexpr int kBlkOtherRegs = 88, kBlkEpilogueRegs = 208;

__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}

// The scale warp: K blocks [kb0, kb1) of tiles tile0, tile0 + step, ...  where(tile, row0, blk): the tile's first token and
// this lane's weight block (lanes 0 and 1); hand_over(it): wait for the phase before block it's, then arrive.
template <typename Where, typename HandOver>
__device__ __forceinline__ void feed_block_scales(const BlockGemmParams& p, uint32_t ring, int tile0, int num_tiles, int step,
                                                  int kb0, int kb1, int lane, Where where, HandOver hand_over) {
  const float* as[4];
  const float* bs = nullptr;
  int l_tile = tile0, l_kb = kb0;
  uint32_t l_it = 0, it = 0;
  auto load_next = [&]() {
    if (l_tile < num_tiles) {
      if (l_kb == kb0) {
        int row0, blk;
        where(l_tile, row0, blk);
#pragma unroll
        for (int i = 0; i < 4; ++i) as[i] = p.as + static_cast<int64_t>(min(row0 + lane + 32 * i, p.M - 1)) * p.as_row;
        bs = p.bs + static_cast<int64_t>(min(blk, ceil_div(p.N, 128) - 1)) * p.bs_row;
      }
      const uint32_t dst = ring + (l_it % kBlkScaleSlots) * kBlkScaleBytes;
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async4(dst + (lane + 32 * i) * 4, as[i] + l_kb * p.as_col);
      if (lane < 2) cp_async4(dst + 512 + lane * 4, bs + l_kb);
      ++l_it;
      if (++l_kb == kb1) {
        l_kb = kb0;
        l_tile += step;
      }
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int i = 0; i < kBlkScaleAhead; ++i) load_next();
  for (int tile = tile0; tile < num_tiles; tile += step) {
#pragma unroll 1
    for (int kb = kb0; kb < kb1; ++kb, ++it) {
      cp_async_wait<kBlkScaleAhead - 1>();
      __syncwarp();
      hand_over(it);
      load_next();
    }
  }
  cp_async_wait<0>();
}
// the scale of block `it` for token `row` of the CTA and weight block `blk` of the tile
__device__ __forceinline__ float block_scale(uint32_t ring, uint32_t it, int row, int blk) {
  const uint32_t at = ring + (it % kBlkScaleSlots) * kBlkScaleBytes;
  return lds_f32(at + row * 4) * lds_f32(at + 512 + blk * 4);
}

}  // namespace b200
#include "fp8_block_pair.cuh"
namespace b200 {

static WaitCounter wait_counter_registered(tc::wait_counter());

// Tile 128 x 256: a 128 x 128 tile moves 64 KiB through shared memory (TMA in + UMMA out) per 256
// tensor-core clocks, twice what an SM's shared memory delivers, and plateaued at 1.59 PFLOP/s
// whatever the epilogue did (measured).  With N = 256 the tile spans TWO weight scale blocks: two
// epilogue warpgroups take one 128-column block each, so the combined scale stays a per-thread
// scalar.  One K block (512 tensor-core clocks) per TMEM hand-off, two 256-column accumulators.
// BN = 128 (twice the tiles, each warpgroup takes 64 columns of the one scale block) is kept for
// problems whose 128 x 256 tiles would leave SMs idle.
template <int BN>
struct BlkCfg {
  static constexpr int STAGES = BN == 256 ? 4 : 6;   // 48 / 32 KiB each: A 128 x 128, B BN x 128
  static constexpr int NBUF = 512 / BN;              // TMEM accumulator buffers of BN columns
  static constexpr int SMEM = STAGES * (128 + BN) * 128 + kBlkScaleSlots * kBlkScaleBytes + (2 * STAGES + 2 * NBUF) * 8 + 16 + 1024;
  static_assert(2 * NBUF + kBlkScaleAhead <= kBlkScaleSlots, "a slot is written after its last reader");
};

template <typename OutT, int BN>
__global__ void __launch_bounds__(kBlkThreads, 1)
fp8_block_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a,
                      const __grid_constant__ CUtensorMap tmap_b, const BlockGemmParams p) {
  constexpr int BLOCK = 128, STAGES = BlkCfg<BN>::STAGES, NBUF = BlkCfg<BN>::NBUF;
  constexpr int COLS = BN / 2;  // columns per epilogue warpgroup
  constexpr int A_BYTES = BLOCK * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t scl = smem_base + STAGES * STAGE_BYTES;
  const uint32_t bars = scl + kBlkScaleSlots * kBlkScaleBytes;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bars + 8u * (2 * STAGES + NBUF + a); };
  const uint32_t tmem_slot = bars + 8u * (2 * STAGES + 2 * NBUF), gave_up = tmem_slot + 4;
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int m_blocks = ceil_div(p.M, BLOCK), n_blocks = ceil_div(p.N, BN);
  const int num_tiles = m_blocks * n_blocks;
  const int num_kb = ceil_div(p.K, BLOCK);
  const int S = BN == 128 ? p.splits : 1;   // wide tiles are never split
  const int rank = S > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int kb0 = S > 1 ? rank * p.kb_per_split : 0;
  const int kb1 = S > 1 ? min(num_kb, kb0 + p.kb_per_split) : num_kb;
  const int tile0 = static_cast<int>(blockIdx.x) / S, tile_step = static_cast<int>(gridDim.x) / S;
  bool dead = false;                     // a wait of this thread ran out: the rest only poll

  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmap_a);
    tc::prefetch_tmap(&tmap_b);
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(full_bar(s), 1);
      tc::mbar_init(empty_bar(s), 1);
    }
    for (int a = 0; a < NBUF; ++a) {
      tc::mbar_init(tfull_bar(a), 2);      // the MMAs' commit and the scale warp
      tc::mbar_init(tempty_bar(a), 8);
    }
    asm volatile("st.shared.u32 [%0], 0;\n" ::"r"(gave_up) : "memory");
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, NBUF * BN);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  griddep_wait();  // activations / scales come from the previous kernel
  griddep_launch_dependents();

  // whole-warp loops, one elected thread per instruction (see gemm_pair.cuh)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kBlkOtherRegs));
    if (warp == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = tile0; tile < num_tiles; tile += tile_step) {
        const int m_blk = tile % m_blocks, n_blk = tile / m_blocks;
        for (int kb = kb0; kb < kb1; ++kb) {
          tc::mbar_wait_bounded(empty_bar(stage), phase ^ 1u, dead, gave_up);
          const uint32_t sa = smem_base + stage * STAGE_BYTES;
          if (tc::elect_one()) {
            tc::mbar_arrive_expect_tx(full_bar(stage), STAGE_BYTES);
            tc::tma_load_2d(sa, &tmap_a, full_bar(stage), kb * BLOCK, m_blk * BLOCK);
            tc::tma_load_2d(sa + A_BYTES, &tmap_b, full_bar(stage), kb * BLOCK, n_blk * BN);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    } else if (warp == 1) {
      constexpr uint32_t idesc = tc::make_idesc(0, 0, BLOCK, BN, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t it = 0;  // running K-block counter across tiles -> TMEM buffer ring
      for (int tile = tile0; tile < num_tiles; tile += tile_step) {
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int buf = it % NBUF;
          const uint32_t buf_phase = (it / NBUF) & 1u;
          tc::mbar_wait_bounded(tempty_bar(buf), buf_phase ^ 1u, dead, gave_up);
          tc::mbar_wait_bounded(full_bar(stage), phase, dead, gave_up);
          tc::tc_fence_after();
          const uint64_t adesc = tc::make_smem_desc_sw128(smem_base + stage * STAGE_BYTES, 1024, 16);
          const uint64_t bdesc = tc::make_smem_desc_sw128(smem_base + stage * STAGE_BYTES + A_BYTES, 1024, 16);
          const uint32_t tmem_d = tmem_base + buf * BN;
          if (tc::elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k) tc::mma_f8f6f4(tmem_d, adesc + 2 * k, bdesc + 2 * k, idesc, k != 0 ? 1u : 0u);
            tc::mma_commit(empty_bar(stage));
            tc::mma_commit(tfull_bar(buf));
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    } else if (warp == 2) {
      feed_block_scales(
          p, scl, tile0, num_tiles, tile_step, kb0, kb1, lane,
          [&](int tile, int& row0, int& blk) {
            row0 = (tile % m_blocks) * BLOCK;
            blk = ((tile / m_blocks) * BN + (lane & 1) * COLS) / BLOCK;
          },
          [&](uint32_t it) {
            tc::mbar_wait_bounded(tfull_bar(it % NBUF), ((it / NBUF) & 1u) ^ 1u, dead, gave_up);
            if (lane == 0) tc::mbar_arrive(tfull_bar(it % NBUF));
          });
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kBlkEpilogueRegs));
    const int quarter = warp & 3;          // TMEM lane quarter this warp may read
    const int half = (warp - 4) >> 2;      // which half of the tile's columns
    OutT* out = static_cast<OutT*>(p.out);
    const OutT* bias = static_cast<const OutT*>(p.bias);
    const int nsb = ceil_div(p.N, BLOCK);  // weight scale blocks along N
    uint32_t it = 0;
    for (int tile = tile0; tile < num_tiles; tile += tile_step) {
      const int m_blk = tile % m_blocks, n_blk = tile / m_blocks;
      const int row = m_blk * BLOCK + quarter * 32 + lane;
      const bool row_ok = row < p.M;
      const int col_base = n_blk * BN + half * COLS;
      const int sblk = col_base / BLOCK;
      const bool blk_ok = sblk < nsb;      // the tile's second half may lie past N
      float2 acc[COLS / 2];
#pragma unroll
      for (int j = 0; j < COLS / 2; ++j) acc[j] = make_float2(0.f, 0.f);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int buf = it % NBUF;
        const uint32_t buf_phase = (it / NBUF) & 1u;
        tc::mbar_wait_bounded(tfull_bar(buf), buf_phase, dead, gave_up);
        tc::tc_fence_after();
        const float s = block_scale(scl, it, quarter * 32 + lane, half);
        const float2 s2 = make_float2(s, s);
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * BN +
                               half * COLS;
#pragma unroll
        for (int c = 0; c < COLS / 16; ++c) {
          uint32_t r[16];
          tc::tmem_ld16(taddr + c * 16, r);
          tc::tmem_ld_wait();
          if (c == COLS / 16 - 1) {  // the whole partial is in registers: hand the buffer back before the math
            tc::tc_fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(tempty_bar(buf));
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            acc[c * 8 + j] = ffma2(
                make_float2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), s2,
                acc[c * 8 + j]);
        }
      }
      if (S > 1) {
        // the slices' promoted fp32 sums meet over distributed shared memory: parked in the idle operand ring as
        // [column][row], then rank r adds its share of the column groups in rank order (deterministic)
        const uint32_t part = smem_base + (quarter * 32 + lane) * 4;
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) {
          asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(part + (half * COLS + 2 * j) * 512), "f"(acc[j].x) : "memory");
          asm volatile("st.shared.f32 [%0], %1;\n" ::"r"(part + (half * COLS + 2 * j + 1) * 512), "f"(acc[j].y) : "memory");
        }
        __syncwarp();
        cluster_sync_all();
        for (int g = rank * 2 + half; g < BN / 8; g += 2 * S) {
          float sum[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) sum[j] = 0.f;
          for (int q = 0; q < S; ++q) {
            const uint32_t src = map_to_rank(part + g * 8 * 512, q);
            float t[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) t[j] = ld_cluster_f32(src + j * 512);
#pragma unroll
            for (int j = 0; j < 8; ++j) sum[j] += t[j];
          }
          const int col0 = n_blk * BN + g * 8;
          if (!row_ok || col0 >= p.N) continue;
          OutT* o8 = out + static_cast<int64_t>(row) * p.ldc + col0;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (bias && col0 + j < p.N) sum[j] += to_float<OutT>(bias[col0 + j]);
          if (col0 + 8 <= p.N && p.vec_ok) {
            *reinterpret_cast<uint4*>(o8) = make_uint4(pack_out2<OutT>(sum[0], sum[1]), pack_out2<OutT>(sum[2], sum[3]),
                                                       pack_out2<OutT>(sum[4], sum[5]), pack_out2<OutT>(sum[6], sum[7]));
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (col0 + j < p.N) o8[j] = from_float<OutT>(sum[j]);
          }
        }
        __syncwarp();
        cluster_sync_all();                // the peers have read this slice
      } else if (row_ok && blk_ok) {
        OutT* orow = out + static_cast<int64_t>(row) * p.ldc;
        const int col0 = col_base;
        if (col0 + COLS <= p.N && p.vec_ok) {
#pragma unroll
          for (int v = 0; v < COLS / 8; ++v) {
            uint32_t packed[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float2 x = acc[v * 4 + e];
              if (bias) {
                x.x += to_float<OutT>(bias[col0 + v * 8 + e * 2]);
                x.y += to_float<OutT>(bias[col0 + v * 8 + e * 2 + 1]);
              }
              packed[e] = pack_out2<OutT>(x.x, x.y);
            }
            *reinterpret_cast<uint4*>(orow + col0 + v * 8) =
                make_uint4(packed[0], packed[1], packed[2], packed[3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < COLS / 2; ++j) {
            const int c = col0 + 2 * j;
            if (c < p.N) orow[c] = from_float<OutT>(acc[j].x + (bias ? to_float<OutT>(bias[c]) : 0.f));
            if (c + 1 < p.N)
              orow[c + 1] = from_float<OutT>(acc[j].y + (bias ? to_float<OutT>(bias[c + 1]) : 0.f));
          }
        }
      }
    }
  }

  if (S > 1 && warp < 4) {               // the reduction's two barriers (one tile per cluster)
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::report_gave_up(gave_up, p.wait_error);
    tc::tmem_dealloc(tmem_base, NBUF * BN);
  }
}

// Clusters of S CTAs of the 128-wide instance that are resident at once on the current device (0: none).
template <typename OutT, int BN>
static int block_clusters(int S) {
  static std::atomic<int> cached[64][9];
  auto kern = fp8_block_gemm_kernel<OutT, BN>;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = cached[dev][S].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S * 8);
    cfg.blockDim = dim3(kBlkThreads);
    cfg.dynamicSmemBytes = BlkCfg<BN>::SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BlkCfg<BN>::SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = -1;
    }
    cached[dev][S].store(n, std::memory_order_relaxed);
  }
  return n > 0 ? n : 0;
}

template <typename OutT, int BN>
static int launch_block_gemm_bn(const void* a, int64_t lda, const void* b, int64_t ldb,
                                const BlockGemmParams& p_in, cudaStream_t st) {
  constexpr int SMEM = BlkCfg<BN>::SMEM;
  BlockGemmParams p = p_in;
  CUtensorMap ta, tb;
  int rc = wait_error_arm("fp8_block_gemm", &p.wait_error);
  if (rc) return rc;
  rc = make_tmap_2d(&ta, a, p.M, p.K, lda, 128, 128, 1, false);
  if (rc) return rc;
  rc = make_tmap_2d(&tb, b, p.N, p.K, ldb, BN, 128, 1, true);
  if (rc) return rc;
  auto kern = fp8_block_gemm_kernel<OutT, BN>;
  const int resident = block_clusters<OutT, BN>(1);   // also raises the shared memory limit
  B200_REQUIRE(resident > 0, "fp8_block_gemm_kernel does not fit this device");
  const int tiles = ceil_div(p.M, 128) * ceil_div(p.N, BN);
  const int sms = device_sm_count();
  const int num_kb = ceil_div(p.K, 128);
  p.vec_ok = p.ldc % 8 == 0 && aligned16(p.out);
  p.splits = 1;
  p.kb_per_split = num_kb;
  if (BN == 128) {
    // Largest split whose clusters are all resident, with 4 K blocks or more per slice, where it takes 12 blocks or
    // more off the chain: the exchange of the partials costs as much as that (split - whole, us, median of 25 to 34
    // problems of 33 to 777 tokens: 3 blocks saved +1.7, 8 +1.0, 10 0, 12 -0.4, 16 -1.2, 24 -2.9; 4096 x 14336, 128
    // tokens 31.8 -> 16.3 in 4).  With more tiles than half the SMs there is nothing to split for.
    for (int S = sms / tiles < 8 ? sms / tiles : 8; S > 1; --S) {
      const int per = ceil_div(num_kb, S);
      if (per < 4 || num_kb - per < 12 || (S - 1) * per >= num_kb || block_clusters<OutT, BN>(S) < tiles) continue;
      p.splits = S;
      p.kb_per_split = per;
      break;
    }
  }
  const int grid = p.splits > 1 ? tiles * p.splits : (tiles < sms ? tiles : sms);
  note_variant("fp8_block_gemm bn=%d tiles=%d splits=%d", BN, tiles, p.splits);
  {
    ScopedKernelTimer timer("fp8_block_gemm", st);
    B200_CUDA_OK(launch_kernel(kern, dim3(grid), dim3(kBlkThreads), SMEM, st, p.splits, pdl_gemm_family(p.M, kPdlGemmBig), ta, tb, p));
  }
  B200_CHECK_LAUNCH("fp8_block_gemm_kernel");
  return 0;
}

// Pairs of CTAs that are resident at once on the current device (0: none).
template <typename OutT>
static int block_pairs() {
  static std::atomic<int> cached[64];
  auto kern = fp8_block_pair_kernel<OutT>;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kBlkThreads);
    cfg.dynamicSmemBytes = kBlkPairSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kBlkPairSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = -1;
    }
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n > 0 ? n : 0;
}

template <typename OutT>
static int launch_block_pair(const void* a, int64_t lda, const void* b, int64_t ldb, const BlockGemmParams& p_in, int pairs,
                             cudaStream_t st) {
  BlockGemmParams p = p_in;
  CUtensorMap ta, tb;
  int rc = wait_error_arm("fp8_block_gemm", &p.wait_error);
  if (rc) return rc;
  rc = make_tmap_2d(&ta, a, p.M, p.K, lda, 128, 128, 1, false);
  if (rc) return rc;
  rc = make_tmap_2d(&tb, b, p.N, p.K, ldb, 64, 128, 1, true);
  if (rc) return rc;
  const int tiles = ceil_div(p.M, 256) * ceil_div(p.N, 256);
  p.vec_ok = p.ldc % 8 == 0 && aligned16(p.out);
  p.splits = 1;
  p.kb_per_split = ceil_div(p.K, 128);
  note_variant("fp8_block_gemm pair tiles=%d", tiles);
  {
    ScopedKernelTimer timer("fp8_block_gemm", st);
    B200_CUDA_OK(launch_kernel(fp8_block_pair_kernel<OutT>, dim3(2 * (tiles < pairs ? tiles : pairs)), dim3(kBlkThreads),
                               kBlkPairSmem, st, 2, pdl_gemm_family(p.M, kPdlGemmBig), ta, tb, p));
  }
  B200_CHECK_LAUNCH("fp8_block_pair_kernel");
  return 0;
}

template <typename OutT>
static int launch_block_gemm(const void* a, int64_t lda, const void* b, int64_t ldb,
                             const BlockGemmParams& p, cudaStream_t st) {
  // Estimated us of the three forms, waves x (K blocks x rate + tile) + launch.  Over 137 problems of 300 to 3001 tokens
  // timed on all of them (K 512 to 14336, N 1000 to 28672, profiles/fp8_block_forms.json) the pick is 0.9 % slower than the
  // best on average, and in five more than a tenth (600 x 1000 x 2064 19.9, 14.6 in pairs).  Narrow tiles that are split
  // over K (fewer than half the SMs) are one wave, which is always theirs.
  const int num_kb = ceil_div(p.K, 128), sms = device_sm_count(), pairs = block_pairs<OutT>();
  const int mb = ceil_div(p.M, 128), nb = ceil_div(p.N, 256);
  const double narrow = ceil_div(mb * ceil_div(p.N, 128), sms) * (0.28 * num_kb + 2.7) + 3.7;
  const double wide = ceil_div(mb * nb, sms) * (0.41 * num_kb + 6.0) + 2.9;
  const double pair = pairs > 0 ? ceil_div(ceil_div(p.M, 256) * nb, pairs) * (0.37 * num_kb + 5.5) + 2.8 : wide;
  if (pair < wide && pair < narrow) return launch_block_pair<OutT>(a, lda, b, ldb, p, pairs, st);
  if (wide < narrow) return launch_block_gemm_bn<OutT, 256>(a, lda, b, ldb, p, st);
  return launch_block_gemm_bn<OutT, 128>(a, lda, b, ldb, p, st);
}

}  // namespace b200

extern "C" {

static int fp8_gemm_block128_impl(const void* a, int64_t lda, const void* b, int64_t ldb,
                                  const float* as, int64_t as_row_stride, int64_t as_col_stride,
                                  const float* bs, int64_t bs_row_stride, const void* bias,
                                  void* out, int64_t ldc, int M, int N, int K, int out_dtype,
                                  void* stream, void* comm) {
  using namespace b200;
  if (M == 0 || N == 0) return 0;
  B200_REQUIRE(a && b && as && bs && out, "b200_fp8_gemm_block128: null pointer");
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "b200_fp8_gemm_block128: bad shape %dx%dx%d", M, N, K);
  B200_REQUIRE(lda % 16 == 0 && ldb % 16 == 0 && aligned16(a) && aligned16(b),
               "b200_fp8_gemm_block128: A/B must be 16-byte aligned with lda/ldb %% 16 == 0");
  B200_REQUIRE(out_dtype == B200_BF16 || out_dtype == B200_F16,
               "b200_fp8_gemm_block128: out dtype %d", out_dtype);
  cudaStream_t st0 = static_cast<cudaStream_t>(stream);
  // (block-scaled: up to 32 tokens; from there the promotion loops over 64 and 128 tokens per channel are slower
  // than the big tile: 64 tokens, us, qkv / o / gate_up / down 21.3 / 15.1 / 56.0 / 33.7 against 11.8 / 9.7 / 28.0 / 17.3)
  const bool fuse_ar = M <= 64 && comm_can_fuse(comm, M, N);
  if (fuse_ar || (M <= smallm_max_m() && (M <= 32 || smallm_forced()))) {  // decode regime: weight streaming, swap-AB + cluster split-K
    SmallMParams sp = {};
    if (fuse_ar) {
      sp.use_comm = 1;
      sp.comm = static_cast<const Comm*>(comm)->dev;
    }
    sp.out = out;
    sp.ldc = ldc;
    sp.as = as;
    sp.as_row = as_row_stride;
    sp.as_col = as_col_stride;
    sp.bs = bs;
    sp.bs_row = bs_row_stride;
    sp.bias = bias;
    sp.M = M;
    sp.N = N;
    sp.K = K;
    const int rc = dispatch_smallm<true>(a, lda, b, ldb, sp, out_dtype, st0, "fp8_block_gemm_smallm");
    if (rc || !comm || fuse_ar) return rc;
    return comm_all_reduce_rows(comm, out, ldc, M, N, out_dtype, stream);
  }
  BlockGemmParams p;
  p.out = out;
  p.ldc = ldc;
  p.as = as;
  p.as_row = as_row_stride;
  p.as_col = as_col_stride;
  p.bs = bs;
  p.bs_row = bs_row_stride;
  p.bias = bias;
  p.M = M;
  p.N = N;
  p.K = K;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = out_dtype == B200_BF16 ? launch_block_gemm<__nv_bfloat16>(a, lda, b, ldb, p, st)
                                        : launch_block_gemm<__half>(a, lda, b, ldb, p, st);
  if (rc || !comm) return rc;
  return comm_all_reduce_rows(comm, out, ldc, M, N, out_dtype, stream);
}

int b200_fp8_gemm_block128(const void* a, int64_t lda, const void* b, int64_t ldb, const float* as,
                           int64_t as_row_stride, int64_t as_col_stride, const float* bs,
                           int64_t bs_row_stride, const void* bias, void* out, int64_t ldc, int M,
                           int N, int K, int out_dtype, void* stream) {
  return fp8_gemm_block128_impl(a, lda, b, ldb, as, as_row_stride, as_col_stride, bs, bs_row_stride,
                                bias, out, ldc, M, N, K, out_dtype, stream, nullptr);
}

int b200_fp8_gemm_block128_ar(void* comm, const void* a, int64_t lda, const void* b, int64_t ldb,
                              const float* as, int64_t as_row_stride, int64_t as_col_stride,
                              const float* bs, int64_t bs_row_stride, const void* bias, void* out,
                              int64_t ldc, int M, int N, int K, int out_dtype, void* stream) {
  B200_REQUIRE(comm, "b200_fp8_gemm_block128_ar: null communicator");
  return fp8_gemm_block128_impl(a, lda, b, ldb, as, as_row_stride, as_col_stride, bs, bs_row_stride,
                                bias, out, ldc, M, N, K, out_dtype, stream, comm);
}

int b200_fp8_linear(const b200_fp8_linear_args* a) {
  using namespace b200;
  B200_REQUIRE(a, "b200_fp8_linear: null pointer");
  B200_REQUIRE(a->M >= 0 && a->M <= 0x7fffffff && a->N >= 0 && a->N <= 0x7fffffff && a->K > 0 && a->K <= 0x7fffffff,
               "b200_fp8_linear: bad shape %lldx%lldx%lld", static_cast<long long>(a->M), static_cast<long long>(a->N),
               static_cast<long long>(a->K));
  if (a->M == 0 || a->N == 0) return 0;
  B200_REQUIRE(a->scratch && (reinterpret_cast<uintptr_t>(a->scratch) & 255u) == 0, "b200_fp8_linear: scratch");
  const int M = static_cast<int>(a->M), N = static_cast<int>(a->N), K = static_cast<int>(a->K), dtype = static_cast<int>(a->dtype);
  char* q = static_cast<char*>(a->scratch);
  float* scales = reinterpret_cast<float*>(q + (a->M * a->K + 255) / 256 * 256);
  if (a->block) {
    const int rc = b200_fp8_quant_group128(a->x, a->ldx, q, K, scales, 1, M, M, K, 1e-10f, dtype, a->stream);
    return rc ? rc : b200_fp8_gemm_block128(q, K, a->w, a->ldw, scales, 1, M, a->w_scale, a->w_scale_stride, a->bias, a->out,
                                            a->ldc, M, N, K, dtype, a->stream);
  }
  const int rc = b200_fp8_quant_per_token(a->x, a->ldx, q, K, scales, nullptr, M, K, 0, 0.f, dtype, a->stream);
  return rc ? rc : b200_fp8_gemm_rowcol(q, K, a->w, a->ldw, scales, M > 1 ? 1 : 0, a->w_scale, static_cast<int>(a->w_scale_stride),
                                        a->bias, a->out, a->ldc, M, N, K, dtype, a->stream);
}

}  // extern "C"
