// Int4 weight-only GEMM whose dequantised weights go from registers to TENSOR MEMORY, for 17 to 512 tokens.
//
// Replaces, above the GEMV's range, the reference's AWQLinearMethod.apply = awq_dequantize + matmul
// (python/sglang/srt/layers/quantization/awq.py:197-215); reads the stream copy of the weight (w4a16_gemv2.cu).
//
// Why: the fused kernel of w4a16.cu writes each 16-bit weight tile to shared memory and the tensor cores read it back,
// and the packed words pass through shared memory as well: ~600 of its ~1100 clocks per 128 channels x 128 k.  Here the
// weight is the 128-row A operand in tensor memory (tcgen05.st, one channel per lane), so shared memory carries the packed
// words and the activations only.
//
//   warp 0      TMA producer of the activations (bn tokens x 64 k, B operand)
//   warp 1      MMA issuer: per 64 k four tcgen05.mma of 128 channels x bn tokens, A from tensor memory
//   warps 2, 3  packed words, zeros and scales by cp.async: 4.5 KiB per 64 k, a deep ring
//   warps 4-11  dequantisers, two groups on alternate stages: thread = channel; 8 words -> 32 pairs (w - z) * s, rounded as
//               awq_dequant_kernel does -> tcgen05.st; then the epilogue.
// A CTA has one tile (a block of tokens x 128 channels, or a cluster rank's part of its K).
//
// A 16-channel x 64-k tile of the stream is 32 pieces of 16 bytes, piece 4 g + t = columns g and g + 8 at k = 8 t ..+7
// of both 32-k halves.  It lands in shared memory as piece t of all g next to each other, so that the 16-byte reads of a
// warp (t fixed, lanes over g) touch each bank once.
//
// Bound by the dequantisers: ~200 instructions a warp and stage, ~400 clocks of an SM per 128 channels x 64 k with two CTAs
// on it (scales read from global memory by the dequantisers had cost 600).  us, w4a16.cu -> here (f16, Qwen2.5-32B at
// TP 2, qkv / o / gate_up / down): 24 tokens 11.1 / 10.0 / 46.4 / 25.5 -> 8.6 / 7.4 / 29.4 / 19.4; 128 tokens 18.4 / 19.1 /
// 50.8 / 35.6 -> 13.4 / 12.1 / 43.1 / 27.6.
#include "gemm_tc.cuh"

namespace b200 {

static WaitCounter wait_counter_registered(tc::wait_counter());

struct TsParams {
  const uint4* qw;      // stream layout
  const void* zeros;    // [K/g, N] MAGIC + z
  const void* scales;   // [K/g, N]
  const void* bias;     // [N] or null
  void* out;
  int64_t ldc;
  int M, N, K, group;
  int bn;               // tokens of a tile, a multiple of 16
  int nx, nr;           // stages of the activation and of the packed ring
  int raw_bytes;        // of a packed stage: 4 KiB of words, then a zero and a scale row of 128 channels per group in it
  int kb_per_split;     // 64-k blocks per cluster rank
  int* wait_error;
};

constexpr int kTsMaxX = 8, kTsMaxR = 24, kTsMinR = 6, kTsMaxA = 4;   // ring limits
constexpr int kTsWordBytes = 4096, kTsRowBytes = 256;
constexpr int kTsThreads = 384;
constexpr int kTsBarBytes = (2 * kTsMaxX + 2 * kTsMaxR + 2 * kTsMaxA + 1) * 8 + 16;

template <int CTAS>
struct TsCfg {
  static constexpr int NA = CTAS == 3 ? 2 : 4;                 // A buffers of 64 k (32 columns), NA / 2 per dequantising group
  static constexpr int MAX_BN = CTAS == 3 ? 64 : CTAS == 2 ? 128 : 192;
  static constexpr int D_COL = NA * 32;
  static constexpr int TMEM_COLS = CTAS == 3 ? 128 : CTAS == 2 ? 256 : 512;
  static constexpr int BUDGET = CTAS == 3 ? 75 * 1024 : CTAS == 2 ? 113 * 1024 : 225 * 1024;
  static_assert(D_COL + MAX_BN <= TMEM_COLS, "tensor memory");
  // The packed ring may have an odd number of slots, which then pass from one dequantising group to the other.  A group that
  // waits for the words of stage i has stored stage i - 2, so the MMAs of stage i - 2 - NA are done, and with them the words
  // of all stages up to that one had landed: a slot's phase before the one waited for is complete, and its parity is not
  // taken for that of the phase before last.
  static_assert(NA + 2 <= kTsMinR, "a group may not be a lap of the packed ring ahead");
};

template <typename T>
struct TsMagic;
template <>
struct TsMagic<__half> {
  using T2 = __half2;
  static constexpr uint32_t kBits = 0x64006400u;
};
template <>
struct TsMagic<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static constexpr uint32_t kBits = 0x43004300u;
};

// 8 nibbles -> 4 pairs of neighbouring k: w - z, exact, then one multiplication in 16 bits.  A nibble under a magic exponent is
// magic + w, zb = magic + z.  f16 has room for a nibble four bits up, 1024 + 16 w: times 1/16 less (64 + z) (zh) is w - z as
// well, exactly, and takes the place of the subtraction, so that a word needs one shift instead of three (integer instructions
// issue at half rate).
template <typename T>
__device__ __forceinline__ uint32_t ts_and_or(uint32_t w, uint32_t mask) {
  uint32_t magic = TsMagic<T>::kBits, b;
  asm("" : "+r"(mask), "+r"(magic));   // registers: one LOP3
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(b) : "r"(w), "r"(mask), "r"(magic));
  return b;
}
template <typename T>
__device__ __forceinline__ void ts_dequant8(uint32_t w, uint32_t zb, uint32_t zh, uint32_t s, uint32_t* r) {
  using T2 = typename TsMagic<T>::T2;
  auto as2 = [](uint32_t v) { return *reinterpret_cast<const T2*>(&v); };
  auto put = [&](int i, T2 d) {
    d = __hmul2(d, as2(s));
    r[i] = *reinterpret_cast<const uint32_t*>(&d);
  };
  if constexpr (std::is_same<T, __half>::value) {
    const T2 inv16 = as2(0x2c002c00u);
    const uint32_t w8 = w >> 8;
    put(0, __hsub2(as2(ts_and_or<T>(w, 0x000f000fu)), as2(zb)));
    put(1, __hfma2(as2(ts_and_or<T>(w, 0x00f000f0u)), inv16, as2(zh)));
    put(2, __hsub2(as2(ts_and_or<T>(w8, 0x000f000fu)), as2(zb)));
    put(3, __hfma2(as2(ts_and_or<T>(w8, 0x00f000f0u)), inv16, as2(zh)));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) put(i, __hsub2(as2(ts_and_or<T>(w >> (4 * i), 0x000f000fu)), as2(zb)));
  }
}
// f16: -(64 + z) in both halves from 1024 + z
__device__ __forceinline__ uint32_t ts_high_zero(uint32_t zb) {
  const __half2 d = __hsub2(__half2(__float2half(960.f), __float2half(960.f)), *reinterpret_cast<const __half2*>(&zb));
  return *reinterpret_cast<const uint32_t*>(&d);
}
__device__ __forceinline__ uint32_t ts_ld_pair(uint32_t addr) {   // one 16-bit value in both halves
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];\n" : "=h"(v) : "r"(addr));
  return v | (static_cast<uint32_t>(v) << 16);
}

template <typename T, int CTAS>
__global__ void __launch_bounds__(kTsThreads, CTAS)
w4a16_ts_kernel(const __grid_constant__ CUtensorMap tmap_x, const TsParams p) {
  using C = TsCfg<CTAS>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int x_bytes = p.bn * 128;
  const uint32_t raw = base + p.nx * x_bytes;
  const uint32_t bars = raw + p.nr * p.raw_bytes;
  auto xfull = [&](int s) { return bars + 8u * s; };
  auto xempty = [&](int s) { return bars + 8u * (kTsMaxX + s); };
  auto rfull = [&](int s) { return bars + 8u * (2 * kTsMaxX + s); };
  auto rempty = [&](int s) { return bars + 8u * (2 * kTsMaxX + kTsMaxR + s); };
  auto afull = [&](int s) { return bars + 8u * (2 * kTsMaxX + 2 * kTsMaxR + s); };
  auto aempty = [&](int s) { return bars + 8u * (2 * kTsMaxX + 2 * kTsMaxR + kTsMaxA + s); };
  const uint32_t dfull = bars + 8u * (2 * kTsMaxX + 2 * kTsMaxR + 2 * kTsMaxA);   // the accumulator is complete
  const uint32_t tmem_slot = dfull + 8, gave_up = tmem_slot + 4;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int S = CTAS > 1 ? static_cast<int>(cluster_nctarank()) : 1;
  const int crank = S > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tok_blocks = ceil_div(p.M, p.bn);
  const int KB = p.K >> 6;
  const int kb0 = S > 1 ? min(KB, crank * p.kb_per_split) : 0;
  const int kb1 = S > 1 ? min(KB, kb0 + p.kb_per_split) : KB;
  const int tile = static_cast<int>(blockIdx.x) / S;
  const int tok0 = (tile % tok_blocks) * p.bn, n0 = (tile / tok_blocks) * 128;
  bool dead = false;

  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tmap_x);
    for (int s = 0; s < p.nx; ++s) {
      tc::mbar_init(xfull(s), 1);
      tc::mbar_init(xempty(s), 1);
    }
    for (int s = 0; s < p.nr; ++s) {
      tc::mbar_init(rfull(s), 64);
      tc::mbar_init(rempty(s), 4);
    }
    for (int s = 0; s < C::NA; ++s) {
      tc::mbar_init(afull(s), 4);
      tc::mbar_init(aempty(s), 1);
    }
    tc::mbar_init(dfull, 1);
    asm volatile("st.shared.u32 [%0], 0;\n" ::"r"(gave_up) : "memory");
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, C::TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));

  T* out = static_cast<T*>(p.out);
  auto store16 = [&](const float* v, int tok, int n, float bias) {   // channel n of 16 tokens; tok: token of v[0]
    if (n >= p.N) return;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (tok + j < p.M) out[static_cast<int64_t>(tok + j) * p.ldc + n] = from_float<T>(v[j] + bias);
  };

  if (warp == 0) {
    griddep_wait();                                // the activations are the previous kernel's
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; phase ^= 1u) {    // a lap of the ring
      const int lap_end = min(kb1, kb + p.nx);
      for (int s = 0; kb < lap_end; ++kb, ++s) {
        tc::mbar_wait_bounded(xempty(s), phase ^ 1u, dead, gave_up);
        if (tc::elect_one()) {
          tc::mbar_arrive_expect_tx(xfull(s), x_bytes);
          tc::tma_load_2d(base + s * x_bytes, &tmap_x, xfull(s), kb * 64, tok0);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    const uint32_t idesc = tc::make_idesc(fmt, fmt, 128, p.bn, 0, 0);
    const uint32_t tmem_d = tmem_base + C::D_COL;
    int s = 0, a = 0;
    uint32_t phase = 0, aphase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      tc::mbar_wait_bounded(xfull(s), phase, dead, gave_up);
      tc::mbar_wait_bounded(afull(a), aphase, dead, gave_up);
      tc::tc_fence_after();
      const uint64_t bdesc = tc::make_smem_desc_sw128(base + s * x_bytes, 1024, 16);
      if (tc::elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k)                // 32 bytes of K further on: 2 in the address field
          tc::mma_f16_ts(tmem_d, tmem_base + a * 32 + k * 8, bdesc + 2 * k, idesc, kb != kb0 || k != 0 ? 1u : 0u);
        tc::mma_commit(xempty(s));
        tc::mma_commit(aempty(a));
      }
      __syncwarp();
      if (++s == p.nx) {
        s = 0;
        phase ^= 1u;
      }
      if (++a == C::NA) {
        a = 0;
        aphase ^= 1u;
      }
    }
    if (tc::elect_one()) tc::mma_commit(dfull);
    __syncwarp();
  } else if (warp < 4) {
    // packed words: piece i of a stage = strip i / 32, piece i % 32 = 4 g + t of that tile -> strip * 512 + t * 128 + g * 16
    const int l = static_cast<int>(threadIdx.x) - 64;          // 0 .. 63
    const uint32_t dst0 = raw + (l >> 5) * 512 + (lane & 3) * 128 + (lane >> 2) * 16;
    const T* zeros = static_cast<const T*>(p.zeros);
    const T* scales = static_cast<const T*>(p.scales);
    const int strip0 = n0 / 16 + (l >> 5), col = n0 + (lane & 15) * 8;
    const uint4* src = p.qw + static_cast<int64_t>(strip0) * KB * 32 + lane;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; phase ^= 1u) {    // a lap of the ring
      const int lap_end = min(kb1, kb + p.nr);
      for (int s = 0; kb < lap_end; ++kb, ++s) {
        tc::mbar_wait_bounded(rempty(s), phase ^ 1u, dead, gave_up);
#pragma unroll
        for (int j = 0; j < 4; ++j)                // strips past N hold channels that are never stored
          if ((strip0 + 2 * j) * 16 < p.N)
            cp_async16(dst0 + s * p.raw_bytes + j * 1024, src + (static_cast<int64_t>(2 * j) * KB + kb) * 32);
        // zero and scale rows: 16 pieces of 8 channels each; the second group of a stage (32 k) by the second warp
        const int64_t row = static_cast<int64_t>((kb * 64 + (l >> 5) * 32) / p.group) * p.N + col;
        if (col < p.N && (l < 32 || p.group < 64))
          cp_async16(raw + s * p.raw_bytes + kTsWordBytes + (l >> 5) * (2 * kTsRowBytes) + lane * 16, (lane < 16 ? zeros : scales) + row);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];\n" ::"r"(rfull(s)) : "memory");
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    griddep_launch_dependents();
  } else {
    const int grp = (warp - 4) >> 2;
    const int r = (warp & 3) * 32 + lane;          // channel of the tile = lane of tensor memory
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const bool hi = (lane & 8) != 0;               // columns 8 .. 15 of a 16-channel tile
    const uint32_t src0 = raw + (r >> 4) * 512 + (lane & 7) * 16;
    const uint32_t sz0 = raw + kTsWordBytes + r * 2, sz1 = p.group < 64 ? sz0 + 2 * kTsRowBytes : sz0;
    // this group's stages are every second one of the CTA's
    int rs = grp, a = grp;
    uint32_t rphase = 0, aphase = 0;
    for (int kb = kb0 + grp; kb < kb1; kb += 2) {
      tc::mbar_wait_bounded(rfull(rs), rphase, dead, gave_up);
      const uint32_t at = rs * p.raw_bytes;
      uint32_t w[8];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint4 v = lds128(src0 + at + t * 128);
        w[t] = hi ? v.y : v.x;
        w[4 + t] = hi ? v.w : v.z;
      }
      const uint32_t z2[2] = {ts_ld_pair(sz0 + at), ts_ld_pair(sz1 + at)};
      const uint32_t s2[2] = {ts_ld_pair(sz0 + at + kTsRowBytes), ts_ld_pair(sz1 + at + kTsRowBytes)};
      const uint32_t zh[2] = {ts_high_zero(z2[0]), ts_high_zero(z2[1])};
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(rempty(rs));
      uint32_t o[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) ts_dequant8<T>(w[i], z2[i >> 2], zh[i >> 2], s2[i >> 2], o + 4 * i);
      tc::mbar_wait_bounded(aempty(a), aphase ^ 1u, dead, gave_up);
      tc::tc_fence_after();
      __syncwarp();
      tc::tmem_st32(tmem_base + lane_addr + a * 32, o);
      tc::tmem_st_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(afull(a));
      rs += 2;
      if (rs >= p.nr) {
        rs -= p.nr;
        rphase ^= 1u;
      }
      if (C::NA == 4) a ^= 2;
      if (a < 2) aphase ^= 1u;
    }
    // ---- epilogue
    griddep_wait();
    const int n = n0 + r;
    const int toks = min(p.bn, p.M - tok0);
    const float bias = p.bias && n < p.N ? to_float<T>(static_cast<const T*>(p.bias)[n]) : 0.f;
    const uint32_t tmem_d = tmem_base + lane_addr + C::D_COL;
    if (kb1 > kb0) tc::mbar_wait_bounded(dfull, 0, dead, gave_up);
    tc::tc_fence_after();
    __syncwarp();
    if (S == 1) {
      for (int c = grp * 16; c < toks; c += 32) {
        uint32_t v[16];
        tc::tmem_ld16(tmem_d + c, v);
        tc::tmem_ld_wait();
        store16(reinterpret_cast<const float*>(v), tok0 + c, n, bias);
      }
    } else {
      // fixed-order cluster reduction: token m of the partial goes to rank m % S, slot [rank][m / S][channel] of its
      // idle rings; then each rank adds the slots of its own tokens in rank order
      const int tpr = ceil_div(toks, S);
      const uint32_t push = base + (crank * tpr * 128 + r) * 4;
      cluster_sync_all();                          // every peer's rings are idle
      for (int c = grp * 16; c < toks; c += 32) {
        uint32_t v[16];
        if (kb1 > kb0) {
          tc::tmem_ld16(tmem_d + c, v);
          tc::tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = 0u;
        }
        int q = c % S, slot = c / S;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (c + j < toks)
            asm volatile("st.shared::cluster.u32 [%0], %1;\n" ::"r"(map_to_rank(push + slot * 512, q)), "r"(v[j]) : "memory");
          if (++q == S) {
            q = 0;
            ++slot;
          }
        }
      }
      __syncwarp();
      cluster_sync_all();                          // all partials have arrived
      for (int j = grp; j < tpr; j += 2) {
        const int m = j * S + crank;
        if (m >= toks) break;
        float sum = 0.f;
        for (int q = 0; q < S; ++q) {
          float x;
          asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(x) : "r"(base + ((q * tpr + j) * 128 + r) * 4) : "memory");
          sum += x;
        }
        if (n < p.N) out[static_cast<int64_t>(tok0 + m) * p.ldc + n] = from_float<T>(sum + bias);
      }
    }
  }

  if (S > 1 && warp < 4) {                         // the two barriers of the reduction
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::report_gave_up(gave_up, p.wait_error);
    tc::tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

struct TsPlan {
  int ctas, bn, S, kb_per_split, nx, nr, smem;
};

template <int CTAS>
static void ts_rings(TsPlan* pl, int raw) {
  using C = TsCfg<CTAS>;
  const int x = pl->bn * 128, room = C::BUDGET - kTsBarBytes - 1024;
  const int nx = (room - kTsMinR * raw) / x;
  pl->nx = nx > kTsMaxX ? kTsMaxX : nx;
  const int nr = (room - pl->nx * x) / raw;
  pl->nr = nr > kTsMaxR ? kTsMaxR : nr;
  pl->smem = pl->nx * x + pl->nr * raw + kTsBarBytes + 1024;
}

// Tile width, K split and form for M tokens; false where the kernels of w4a16.cu / w4a16_stream_gemm.cu are faster.
// Measured (f16, us): a 64-k stage takes 0.22 + 0.0004 bn of a CTA alone on its SM, 0.19 + 0.0007 bn times their number where
// several share one; a split 2 + 0.02 bn for the exchange of the partials.
// At most 1.63 CTAs an SM (241 of 148).  Every split of 19 to 74 tiles timed (K 2560, 5120 and 13824; 24, 64 and 128 tokens):
// up to 1.75 an SM all clusters run in one wave, then soon in two (5120 deep, 64 tokens: 264 CTAs in sixes 13.1 us, 276 20.2;
// 256 in eights 10.9, 272 16.1).  Between 1.63 and 1.75 the picks would be 4 % faster on average (13824 deep, 42 tiles, 64
// tokens: three parts 25.1 / six 22.4), but up to 11 % slower where K is short and the exchange counts (2560 deep, 32 tiles, 24
// tokens: four parts 6.6 / eight 7.3).  Three CTAs an SM, each half of K, only where that fills them and two would leave every second SM
// half idle (27648 x 5120, 16 / 64 tokens: 34.6 / 38.6 with two, 29.9 / 34.9 with three).
// Above 128 tokens a weight is dequantised again for every block of tokens: worth it while the tiles fit one wave, which the
// 128-token tiles of w4a16.cu take as long for without a split of K (us, there / here: 3584 x 5120, 200 tokens 27.4 / 20.2;
// 1536 x 4096, 300 23.0 / 13.0; 5120 x 13824, 512 130 / 76; but 27648 x 5120, 512 121 / 139).
static bool ts_plan(int M, int N, int K, int raw, TsPlan* pl) {
  if (M < 17 || M > 512 || N % 16 != 0 || K % 64 != 0) return false;
  const int KB = K / 64, n_tiles = ceil_div(N, 128), sms = device_sm_count();
  int tiles = 0;
  auto width = [&](int max_bn) {
    pl->bn = ceil_div(ceil_div(M, ceil_div(M, max_bn)), 16) * 16;
    tiles = n_tiles * ceil_div(M, pl->bn);
  };
  pl->S = 1;
  pl->ctas = 2;
  width(TsCfg<2>::MAX_BN);
  if (M > 128 && tiles > sms) {
    pl->ctas = 1;
    width(TsCfg<1>::MAX_BN);
    if (tiles > sms) return false;
  } else if (M <= TsCfg<3>::MAX_BN && tiles > sms && 2 * tiles <= 3 * sms && KB >= 8) {
    pl->ctas = 3;
    pl->S = 2;
  } else {
    double best = 0;
    for (int S = 1; S <= 8; ++S) {
      const int per = ceil_div(KB, S), load = ceil_div(tiles * S, sms);
      if (S > 1 && (per < 4 || (S - 1) * per >= KB || tiles * S > sms * 1.63)) continue;
      const double us = per * (load == 1 ? 0.22 + 0.0004 * pl->bn : load * (0.19 + 0.0007 * pl->bn)) +
                        (S > 1 ? 2.0 + 0.02 * pl->bn : 0.0);
      if (S == 1 || us < best) {
        best = us;
        pl->S = S;
      }
    }
  }
  pl->kb_per_split = ceil_div(KB, pl->S);
  if (pl->ctas == 3)
    ts_rings<3>(pl, raw);
  else if (pl->ctas == 2)
    ts_rings<2>(pl, raw);
  else
    ts_rings<1>(pl, raw);
  return true;
}
static int ts_raw_bytes(int group) { return kTsWordBytes + (group < 64 ? 4 : 2) * kTsRowBytes; }

template <typename T, int CTAS>
static int launch_ts(const TsPlan& pl, const CUtensorMap& tx, const TsParams& p, cudaStream_t st) {
  auto kern = w4a16_ts_kernel<T, CTAS>;
  B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, TsCfg<CTAS>::BUDGET));
  const int tiles = ceil_div(p.M, p.bn) * ceil_div(p.N, 128);
  note_variant("w4a16_ts ctas=%d bn=%d splits=%d nx=%d nr=%d tiles=%d", CTAS, p.bn, pl.S, p.nx, p.nr, tiles);
  {
    ScopedKernelTimer timer("w4a16_gemm", st);
    B200_CUDA_OK(launch_kernel(kern, dim3(tiles * pl.S), dim3(kTsThreads), pl.smem, st, pl.S,
                               pdl_family(p.M, kPdlGemmSmall), tx, p));
  }
  B200_CHECK_LAUNCH("w4a16_ts_kernel");
  return 0;
}

template <typename T>
static int dispatch_ts(const void* x, int64_t ldx, TsParams p, cudaStream_t st) {
  p.raw_bytes = ts_raw_bytes(p.group);
  TsPlan pl;
  B200_REQUIRE(ts_plan(p.M, p.N, p.K, p.raw_bytes, &pl), "b200_w4a16_gemm_ts: %d tokens x %d x %d are not taken", p.M, p.N, p.K);
  p.bn = pl.bn;
  p.nx = pl.nx;
  p.nr = pl.nr;
  p.kb_per_split = pl.kb_per_split;
  CUtensorMap tx;
  int rc = make_tmap_2d(&tx, x, p.M, p.K, ldx * 2, p.bn, 64, 2, false);
  if (rc) return rc;
  rc = wait_error_arm("w4a16_ts", &p.wait_error);
  if (rc) return rc;
  return pl.ctas == 3 ? launch_ts<T, 3>(pl, tx, p, st) : pl.ctas == 2 ? launch_ts<T, 2>(pl, tx, p, st) : launch_ts<T, 1>(pl, tx, p, st);
}

}  // namespace b200

extern "C" {

int b200_w4a16_gemm_ts_takes(int M, int N, int K, int group_size) {
  using namespace b200;
  TsPlan pl;
  return group_size > 0 && K % group_size == 0 && (group_size == 32 || group_size % 64 == 0) &&
         ts_plan(M, N, K, ts_raw_bytes(group_size), &pl);
}

int b200_w4a16_gemm_ts(const void* x, int64_t ldx, const void* qweight_stream, const void* zeros, const void* scales,
                       const void* bias, void* out, int64_t ldc, int M, int N, int K, int group_size, int dtype,
                       void* stream) {
  using namespace b200;
  if (M == 0 || N == 0) return 0;
  B200_REQUIRE(x && qweight_stream && zeros && scales && out, "b200_w4a16_gemm_ts: null pointer");
  B200_REQUIRE(M > 0 && N > 0 && N % 16 == 0 && K > 0 && K % 64 == 0 && group_size > 0 && K % group_size == 0 &&
                   (group_size == 32 || group_size % 64 == 0),
               "b200_w4a16_gemm_ts: bad shape M=%d N=%d K=%d group=%d", M, N, K, group_size);
  B200_REQUIRE(aligned16(x) && ldx % 8 == 0 && aligned16(qweight_stream) && aligned16(zeros) && aligned16(scales),
               "b200_w4a16_gemm_ts: x, weight, zeros and scales must be 16-byte aligned, ldx %% 8 == 0");
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16, "b200_w4a16_gemm_ts: dtype %d", dtype);
  TsParams p = {};
  p.qw = static_cast<const uint4*>(qweight_stream);
  p.zeros = zeros;
  p.scales = scales;
  p.bias = bias;
  p.out = out;
  p.ldc = ldc;
  p.M = M;
  p.N = N;
  p.K = K;
  p.group = group_size;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return dtype == B200_F16 ? dispatch_ts<__half>(x, ldx, p, st) : dispatch_ts<__nv_bfloat16>(x, ldx, p, st);
}

}  // extern "C"
