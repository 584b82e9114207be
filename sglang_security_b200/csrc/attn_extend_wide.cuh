// Extend attention without window, sink, gate or cap: two 128-row query tiles per CTA, P kept in tensor memory.
//
// attn_extend_kernel runs QK -> softmax -> PV as one serial chain per 64-key tile and CTA (1.3-1.6 us of latency
// for 0.27 us of tensor work, two chains per SM).  Here one CTA per SM owns two query tiles that take turns: while
// the softmax warps of one tile work, the tensor cores run PV and the next QK of the other.
//
//   warps 0-3, 4-7  softmax of tile 0 / 1: thread = query row; 128 scores in registers, bf16 / f16 P written back
//                   over the scores in tensor memory (A operand of PV, so P never crosses shared memory); O is
//                   rescaled only when a row's maximum grows by more than 2^8
//   warp 8          MMA issuer: per key tile PV0 QK0' PV1 QK1' (whole warp, one elected thread)
//   warps 9-11      gather of 128-key K and V tiles through req_to_token into a ring of tiles, in the
//                   128-byte-swizzled layout; slots of the next tile are fetched a tile ahead
//
// Few query tiles (a short turn behind a long prefix): a cluster of S CTAs takes the query tiles of one CTA, each a
// range of the keys; the unnormalised O, maximum and sum of every row meet in shared memory and are merged in rank
// order over the cluster (deterministic).
//
// Tensor memory: S0 | S1 (128 columns each, P in the first 64 of its S) | O0 | O1 (D columns each).
// Shared memory per 128 keys: Q and K of two QK (128 KiB), V of two PV (64), the gather (64) = 2048 clocks at
// 128 B/clk, as long as the tensor work and the 32768 exponentials take: the three bound it together (D 128: 3450
// clocks measured, 2980 without the exponentials).  64-key tiles with two score buffers, which take the softmax
// off the chain, read Q twice as often and were slower: 2 x 8192 tokens 1055 us against 907, both in a burst.
// Llama-3.1-8B heads, us before -> now: 2 x 8192 fresh tokens 1516 -> 920 in a burst, 1600 -> 1100 where the power cap holds
// the clock down; 8 turns of up to 512 behind 1536 cached 155 -> 115.
#pragma once

namespace b200 {

// Extend kernels are launched as dependents of the KV write before them (or what else stands there): their CTAs are placed,
// and the persistent kernel's barriers and tensor memory ready, when it ends.
inline int extend_pdl() { return pdl_gemm_family(1 << 20, kPdlAttn); }
constexpr int kWideThreads = 384;
constexpr int kWideTile = 128;                     // keys
constexpr int kWideMinKeys = 1024;                 // shorter requests: attn_extend_kernel
constexpr int kWideLoaders = 96;
constexpr int kWideSoftmaxRegs = 192, kWideOtherRegs = 120;   // 256 x 192 + 128 x 120 <= 384 x 168 at launch
// (spilled: 4 bytes by the cluster instances of head size 64, 8 by attn_extend_flat_kernel, nothing by the others)

template <int D>
struct WideCfg {
  static constexpr int TILE_BYTES = kWideTile * D * 2;        // a K, V or Q tile
  static constexpr int SLOTS = D == 128 ? 5 : 10;             // K and V tiles in flight
  static constexpr int OFF_RING = 2 * TILE_BYTES;             // after the two Q tiles
  static constexpr int OFF_BAR = OFF_RING + SLOTS * TILE_BYTES;
  static constexpr int N_BARS = 1 + 2 * SLOTS + 8;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BARS * 8 + 16;
  static constexpr int O_COL = 256;
  static constexpr int PART_ROW = D * 4 + 16;                 // a row's partial O, then m and l
  static_assert(256 * PART_ROW <= OFF_BAR, "partial rows alias the operand tiles");
  static_assert(SMEM_BYTES <= 227 * 1024, "tiles exceed shared memory");
};

template <typename T, int D, bool SPLIT>
__global__ void __launch_bounds__(kWideThreads, 1)
attn_extend_wide_kernel(const ExtendParams p) {
  using C = WideCfg<D>;
  constexpr int SL = C::SLOTS;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  griddep_wait();
  const int b = blockIdx.z;
  const int S = SPLIT ? p.kv_splits : 1;           // cluster size; every CTA of a cluster has the same query tiles
  const int rank = S > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int ext = p.extend_lens[b];
  const int prefix = p.prefix_lens[b];
  const int tok_per_tile = 128 / p.pack;
  // the latest query tiles see the most keys: they start first
  const int tok0 = static_cast<int>((gridDim.x - 1 - blockIdx.x) / S) * 2 * tok_per_tile;
  if (tok0 >= ext) return;                         // uniform for the CTA and its cluster
  const int kvh = blockIdx.y / p.head_tiles;
  const int head_base = kvh * p.group + (blockIdx.y - kvh * p.head_tiles) * p.pack;
  const int kv_len = prefix + ext;
  const int tiles = tok0 + tok_per_tile < ext ? 2 : 1;          // query tiles with any row
  const int tok_last = min(tok0 + 2 * tok_per_tile, ext) - 1;
  const int n_all = ceil_div(p.causal ? prefix + tok_last + 1 : kv_len, kWideTile);
  const int per = ceil_div(n_all, S);
  const int j0 = min(n_all, rank * per);           // this CTA's key tiles: loop index j stands for tile j0 + j
  const int n_kv = min(n_all, j0 + per) - j0;      // 0: nothing left for this rank
  const int64_t q_row0 = p.extend_start[b];

  const uint32_t bars = sbase + C::OFF_BAR;
  const uint32_t bar_q = bars;
  auto bar_full = [&](int s) { return bars + 8u * (1 + s); };
  auto bar_empty = [&](int s) { return bars + 8u * (1 + SL + s); };
  auto bar_s = [&](int t) { return bars + 8u * (1 + 2 * SL + t); };        // scores of tile t are complete
  auto bar_p = [&](int t, int h) { return bars + 8u * (3 + 2 * SL + 2 * t + h); };  // half h of P of tile t is written
  auto bar_o = [&](int t) { return bars + 8u * (7 + 2 * SL + t); };        // PV of tile t is complete
  const uint32_t tmem_slot = bars + 8u * C::N_BARS, gave_up = tmem_slot + 4;
  bool dead = false;

  if (threadIdx.x == 0) {
    tc::mbar_init(bar_q, kWideLoaders);
    for (int s = 0; s < SL; ++s) {
      tc::mbar_init(bar_full(s), kWideLoaders);
      tc::mbar_init(bar_empty(s), 1);
    }
    for (int t = 0; t < 2; ++t) {
      tc::mbar_init(bar_s(t), 1);
      tc::mbar_init(bar_p(t, 0), 128);
      tc::mbar_init(bar_p(t, 1), 128);
      tc::mbar_init(bar_o(t), 1);
    }
    asm volatile("st.shared.u32 [%0], 0;\n" ::"r"(gave_up) : "memory");
    tc::fence_barrier_init();
  }
  if (warp == 8) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + C::OFF_BAR + 8 * C::N_BARS);

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kWideOtherRegs));
    if (warp > 8) {
      // ===================== gather =====================
      const int lt = static_cast<int>(threadIdx.x) - 9 * 32;
      constexpr int CPR = D / 8;                   // 16-byte chunks per row
      constexpr int RPP = kWideLoaders / CPR;      // rows per pass
      constexpr int PASSES = (kWideTile + RPP - 1) / RPP;
      const int lrow = lt / CPR, lcol = lt - lrow * CPR;
      const int32_t* rtt = p.req_to_token + p.req_pool_indices[b] * p.rtt_stride;
      const int64_t row_bytes = p.kv_row_stride * 2;
      const char* kbase = static_cast<const char*>(p.k_cache) + static_cast<int64_t>(kvh) * D * 2 + lcol * 16;
      const char* vbase = static_cast<const char*>(p.v_cache) + static_cast<int64_t>(kvh) * D * 2 + lcol * 16;
      int32_t slots[PASSES];
      auto load_slots = [&](int j) {
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
          const int r = lrow + RPP * i, pos = (j0 + j) * kWideTile + r;
          slots[i] = (r < kWideTile && pos < kv_len) ? __ldg(rtt + pos) : 0;   // 0 = the pool's dummy row
        }
      };
      if (n_kv > 0) load_slots(0);
      for (int c = lt; n_kv > 0 && c < tiles * 128 * CPR; c += kWideLoaders) {
        const int r = c / CPR, col = c - r * CPR, t = r >> 7, rr = r & 127;
        int tok = tok0 + r / p.pack;
        if (tok >= ext) tok = ext - 1;             // padding rows repeat the last token (never stored)
        const char* src = static_cast<const char*>(p.q) +
                          ((q_row0 + tok) * p.q_stride + (head_base + r % p.pack) * D) * 2 + col * 16;
        cp_async16(sbase + t * C::TILE_BYTES + swz_off<128>(rr, col), src);
      }
      // Unit u = 2 j + (0: K, 1: V) of key tile j goes to ring slot u % SL and is published LAG units later, when
      // its copies have landed.  Waiting for unit u - SL to be consumed cannot stall: the issuer needs no unit
      // past u - SL + 2 for that, and those up to u - 1 - LAG are published.
      constexpr int LAG = SL - 3;
      auto publish = [&](int u) {
        tc::fence_proxy_async_smem();
        if (u == 0) tc::mbar_arrive(bar_q);        // copied with unit 0
        tc::mbar_arrive(bar_full(u % SL));
      };
      int slot = 0;
      uint32_t phase = 0;
      for (int j = 0; j < n_kv; ++j) {
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          const int u = 2 * j + kv;
          if (u >= SL) tc::mbar_wait_bounded(bar_empty(slot), phase ^ 1u, dead, gave_up);
          const uint32_t dst = sbase + C::OFF_RING + slot * C::TILE_BYTES;
          const char* src = kv ? vbase : kbase;
#pragma unroll
          for (int i = 0; i < PASSES; ++i) {
            const int r = lrow + RPP * i;
            if (r < kWideTile) cp_async16(dst + swz_off<kWideTile>(r, lcol), src + static_cast<int64_t>(slots[i]) * row_bytes);
          }
          cp_async_commit();
          if (kv == 1 && j + 1 < n_kv) load_slots(j + 1);
          if (u >= LAG) {
            cp_async_wait<LAG>();
            publish(u - LAG);
          }
          if (++slot == SL) {
            slot = 0;
            phase ^= 1u;
          }
        }
      }
      cp_async_wait<0>();
      for (int u = max(0, 2 * n_kv - LAG); u < 2 * n_kv; ++u) publish(u);
    } else {
      // ===================== MMA issuer =====================
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc_qk = tc::make_idesc(fmt, fmt, 128, kWideTile, 0, 0);
      constexpr uint32_t idesc_pv = tc::make_idesc(fmt, fmt, 128, D, 0, 1);    // V: MN-major B
      const uint64_t qdesc = tc::make_smem_desc_sw128(sbase, 1024, 16);
      auto wait_unit = [&](int u) {
        tc::mbar_wait_bounded(bar_full(u % SL), (u / SL) & 1u, dead, gave_up);
        tc::tc_fence_after();
      };
      auto issue_qk = [&](int t, int j, bool last) {
        const int s = (2 * j) % SL;
        const uint64_t kdesc = tc::make_smem_desc_sw128(sbase + C::OFF_RING + s * C::TILE_BYTES, 1024, 16);
        if (tc::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = ((kk >> 2) * (128 * 128) + (kk & 3) * 32) >> 4;
            tc::mma_f16(tmem_base + t * 128, qdesc + t * (C::TILE_BYTES >> 4) + off, kdesc + off, idesc_qk, kk != 0 ? 1u : 0u);
          }
          tc::mma_commit(bar_s(t));
          if (last) tc::mma_commit(bar_empty(s));  // both tiles have used this K tile
        }
        __syncwarp();
      };
      if (n_kv > 0) {
        tc::mbar_wait_bounded(bar_q, 0, dead, gave_up);
        wait_unit(0);
        for (int t = 0; t < tiles; ++t) issue_qk(t, 0, t == tiles - 1);
      }
      for (int j = 0; j < n_kv; ++j) {
        const int s = (2 * j + 1) % SL;
        const uint64_t vdesc = tc::make_smem_desc_sw128(sbase + C::OFF_RING + s * C::TILE_BYTES, 1024, kWideTile * 128);
        wait_unit(2 * j + 1);
        for (int t = 0; t < tiles; ++t) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {            // the first 64 keys are multiplied while the others' P is made
            tc::mbar_wait_bounded(bar_p(t, h), j & 1u, dead, gave_up);
            tc::tc_fence_after();
            if (tc::elect_one()) {
#pragma unroll
              for (int kk = h * 4; kk < h * 4 + 4; ++kk)
                tc::mma_f16_ts(tmem_base + C::O_COL + t * D, tmem_base + t * 128 + kk * 8, vdesc + ((kk * 16 * 128) >> 4),
                               idesc_pv, (j | kk) != 0 ? 1u : 0u);
              if (h == 1) {
                tc::mma_commit(bar_o(t));
                if (t == tiles - 1) tc::mma_commit(bar_empty(s));
              }
            }
            __syncwarp();
          }
          if (j + 1 < n_kv) {
            if (t == 0) wait_unit(2 * j + 2);
            issue_qk(t, j + 1, t == tiles - 1);    // overwrites P(j) of this tile: MMAs run in issue order
          }
        }
      }
    }
  } else {
    // ===================== softmax / epilogue =====================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kWideSoftmaxRegs));
    const int t = warp >> 2;
    if (t < tiles) {
      const int r = (warp & 3) * 32 + lane;
      const int tok = tok0 + t * tok_per_tile + r / p.pack;
      const bool row_ok = tok < ext;
      const int limit = p.causal ? prefix + min(tok, ext - 1) : kv_len - 1;    // last visible key
      const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
      const uint32_t tmem_s = tmem_base + lane_addr + t * 128;
      const uint32_t tmem_o = tmem_base + lane_addr + C::O_COL + t * D;
      const float2 sc2 = make_float2(p.qk_scale, p.qk_scale), one2 = make_float2(1.f, 1.f);
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < n_kv; ++j) {
        tc::mbar_wait_bounded(bar_s(t), j & 1u, dead, gave_up);
        tc::tc_fence_after();
        __syncwarp();
        uint32_t v[4][32];
        tc::tmem_ld32(tmem_s, v[0]);
        tc::tmem_ld32(tmem_s + 32, v[1]);
        tc::tmem_ld_wait();
        tc::tmem_ld32(tmem_s + 64, v[2]);
        tc::tmem_ld32(tmem_s + 96, v[3]);
        const int k0 = (j0 + j) * kWideTile;
        float a[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        const bool edge = k0 + kWideTile - 1 > limit;
        if (!edge) {
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            a[0] = fmax3(a[0], __uint_as_float(v[0][e]), __uint_as_float(v[0][e + 1]));
            a[1] = fmax3(a[1], __uint_as_float(v[1][e]), __uint_as_float(v[1][e + 1]));
          }
        }
        tc::tmem_ld_wait();
        if (edge) {                                // the tile crosses the row's last key
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (k0 + c * 32 + e > limit) v[c][e] = 0xff800000u;              // -inf
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            a[0] = fmax3(a[0], __uint_as_float(v[0][e]), __uint_as_float(v[0][e + 1]));
            a[1] = fmax3(a[1], __uint_as_float(v[1][e]), __uint_as_float(v[1][e + 1]));
          }
        }
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          a[2] = fmax3(a[2], __uint_as_float(v[2][e]), __uint_as_float(v[2][e + 1]));
          a[3] = fmax3(a[3], __uint_as_float(v[3][e]), __uint_as_float(v[3][e + 1]));
        }
        const float mt = fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3])) * p.qk_scale;   // scale > 0: -inf stays
        const float m_new = fmaxf(m, mt);
        if (__any_sync(0xffffffffu, m_new > m + kRescaleThreshold)) {          // also the first finite maximum
          if (j > 0) {
            tc::mbar_wait_bounded(bar_o(t), (j - 1) & 1u, dead, gave_up);      // O holds tiles 0 .. j - 1
            tc::tc_fence_after();
            __syncwarp();
            const float alpha = (m == -INFINITY) ? 0.f : fast_exp2(m - m_new);
#pragma unroll 1
            for (int cc = 0; cc < D / 16; ++cc) {
              uint32_t o[16];
              tc::tmem_ld16(tmem_o + cc * 16, o);
              tc::tmem_ld_wait();
#pragma unroll
              for (int c = 0; c < 16; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
              tc::tmem_st16(tmem_o + cc * 16, o);
            }
            l *= alpha;
          }
          m = m_new;
        }
        const float m_use = (m == -INFINITY) ? 0.f : m;
        const float2 nm2 = make_float2(-m_use, -m_use);
        float2 lsum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t packed[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float2 x = ffma2(make_float2(__uint_as_float(v[c][2 * e]), __uint_as_float(v[c][2 * e + 1])), sc2, nm2);
            const float2 y = make_float2(fast_exp2(x.x), fast_exp2(x.y));
            lsum[e & 1] = ffma2(y, one2, lsum[e & 1]);
            packed[e] = pack16<T>(y.x, y.y);
          }
          tc::tmem_st16(tmem_s + c * 16, packed);  // over scores that are in registers by now
          if (c & 1) {
            tc::tmem_st_wait();
            tc::tc_fence_before();
            tc::mbar_arrive(bar_p(t, c >> 1));
          }
        }
        l += (lsum[0].x + lsum[0].y) + (lsum[1].x + lsum[1].y);
      }
      if (n_kv > 0) {
        tc::mbar_wait_bounded(bar_o(t), (n_kv - 1) & 1u, dead, gave_up);
        if (S > 1) tc::mbar_wait_bounded(bar_o(tiles - 1), (n_kv - 1) & 1u, dead, gave_up);  // the last reader
      }
      tc::tc_fence_after();
      __syncwarp();
      if (S > 1) {
        // this rank's O, m, l of the row; the operand tiles are idle (every MMA that read them is complete)
        const uint32_t row_at = sbase + (t * 128 + r) * C::PART_ROW;
#pragma unroll 1
        for (int cc = 0; cc < D / 32; ++cc) {
          uint32_t o[32];
          if (n_kv > 0) {
            tc::tmem_ld32(tmem_o + cc * 32, o);
            tc::tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(row_at + (cc * 32 + i * 4) * 4), "r"(o[4 * i]),
                         "r"(o[4 * i + 1]), "r"(o[4 * i + 2]), "r"(o[4 * i + 3])
                         : "memory");
        }
        asm volatile("st.shared.v2.f32 [%0], {%1,%2};\n" ::"r"(row_at + D * 4), "f"(m), "f"(l) : "memory");
      } else {
        // ---- O / l -> out
        const float inv_l = l > 0.f ? p.out_scale / l : 0.f;
        T* orow = static_cast<T*>(p.o) + (q_row0 + (row_ok ? tok : 0)) * p.o_stride +
                  static_cast<int64_t>(head_base + r % p.pack) * D;
#pragma unroll 1
        for (int cc = 0; cc < D / 32; ++cc) {
          uint32_t o[32];
          tc::tmem_ld32(tmem_o + cc * 32, o);
          tc::tmem_ld_wait();
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t w[4];
#pragma unroll
              for (int e = 0; e < 4; ++e)
                w[e] = pack16<T>(__uint_as_float(o[i * 8 + 2 * e]) * inv_l, __uint_as_float(o[i * 8 + 2 * e + 1]) * inv_l);
              *reinterpret_cast<uint4*>(orow + cc * 32 + i * 8) = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
    }
  }

  if (S > 1) {
    __syncwarp();
    cluster_sync_all();                            // every rank's rows are in its shared memory
    // rank r writes rows r, r + S, ..: a warp per row, four columns per lane, all ranks' pieces requested together
    // (4-byte reads with a row in every second lane took 60 us of remote accesses for 256 rows of 8 ranks)
    const int rows = tiles * 128 / S;              // S divides 128
    for (int i = warp; i < rows; i += kWideThreads / 32) {
      const int rr = i * S + rank, t = rr >> 7, r = rr & 127;
      const int tok = tok0 + t * tok_per_tile + r / p.pack;
      if (tok >= ext) continue;                    // uniform for the warp
      const uint32_t row_at = sbase + rr * C::PART_ROW;
      float x[8][4];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < S && lane * 4 < D)
          asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                       : "=f"(x[q][0]), "=f"(x[q][1]), "=f"(x[q][2]), "=f"(x[q][3])
                       : "r"(map_to_rank(row_at + lane * 16, q))
                       : "memory");
      float mq = -INFINITY, lq = 0.f;
      if (lane < S)
        asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];\n"
                     : "=f"(mq), "=f"(lq) : "r"(map_to_rank(row_at + D * 4, lane)) : "memory");
      float M = mq;
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
      M = __shfl_sync(0xffffffffu, M, 0);
      const float wq = mq == -INFINITY ? 0.f : fast_exp2(mq - M);
      float den = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= S) break;
        const float w = __shfl_sync(0xffffffffu, wq, q);
        den = fmaf(w, __shfl_sync(0xffffffffu, lq, q), den);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[e] = fmaf(w, x[q][e], acc[e]);
      }
      const float inv = den > 0.f ? p.out_scale / den : 0.f;
      if (lane * 4 < D)
        *reinterpret_cast<uint2*>(static_cast<T*>(p.o) + (q_row0 + tok) * p.o_stride +
                                  static_cast<int64_t>(head_base + r % p.pack) * D + lane * 4) =
            make_uint2(pack16<T>(acc[0] * inv, acc[1] * inv), pack16<T>(acc[2] * inv, acc[3] * inv));
    }
    __syncwarp();
    cluster_sync_all();                            // the peers have read this rank's rows
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc::report_gave_up(gave_up, p.wait_error);
    tc::tmem_dealloc(tmem_base, 512);
  }
}

// Clusters of S CTAs that are resident at once on the current device (0: none).
template <typename T, int D>
static int wide_clusters(int S) {
  static std::atomic<int> cached[64][9];
  auto kern = attn_extend_wide_kernel<T, D, true>;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = cached[dev][S].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S * 8);
    cfg.blockDim = dim3(kWideThreads);
    cfg.dynamicSmemBytes = WideCfg<D>::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WideCfg<D>::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = -1;
    }
    cached[dev][S].store(n, std::memory_order_relaxed);
  }
  return n > 0 ? n : 0;
}

// CTAs of a call before its keys are split, and the split: the longest request's keys are cut while whole clusters still
// fit the idle SMs and a CTA keeps three key tiles (~1.8 us each; launch and merge of a cluster cost ~3).  us, one CTA ->
// split: 64 tokens behind 8192, two kv heads 117 -> 36; 128 behind 4000, eight 68 -> 36; 30 behind 2000 47 -> 22.
template <typename T, int D>
static int64_t wide_ctas(const ExtendParams& p, int bs, int max_extend_len, int max_kv_len, int* splits) {
  const int64_t ctas = static_cast<int64_t>(ceil_div(max_extend_len, 256 / p.pack)) * p.Hkv * p.head_tiles * bs;
  *splits = 1;
  for (int S = 8; S > 1 && ctas < device_sm_count(); S /= 2)   // (the occupancy answer also raises the shared memory limit)
    if (max_kv_len >= 3 * S * kWideTile && wide_clusters<T, D>(S) >= ctas) {
      *splits = S;
      break;
    }
  return ctas;
}

template <typename T, int D>
static int launch_extend_wide(const ExtendParams& p_in, int bs, int max_extend_len, int splits, cudaStream_t st) {
  using C = WideCfg<D>;
  ExtendParams p = p_in;
  if (const int rc = wait_error_arm("attn_extend", &p.wait_error)) return rc;
  B200_CUDA_OK(cudaFuncSetAttribute(attn_extend_wide_kernel<T, D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    C::SMEM_BYTES));
  p.kv_splits = splits;
  const dim3 grid(ceil_div(max_extend_len, 256 / p.pack) * p.kv_splits, p.Hkv * p.head_tiles, bs);
  note_variant("attn_extend_wide d=%d splits=%d", D, p.kv_splits);
  {
    ScopedKernelTimer timer("attn_extend", st);
    if (p.kv_splits > 1)
      B200_CUDA_OK(launch_kernel(attn_extend_wide_kernel<T, D, true>, grid, dim3(kWideThreads), C::SMEM_BYTES, st, p.kv_splits, extend_pdl(), p));
    else
      B200_CUDA_OK(launch_kernel(attn_extend_wide_kernel<T, D, false>, grid, dim3(kWideThreads), C::SMEM_BYTES, st, 1, extend_pdl(), p));
  }
  B200_CHECK_LAUNCH("attn_extend_wide_kernel");
  return 0;
}

}  // namespace b200
