// The two-tile extend attention of attn_extend_wide.cuh as a persistent kernel: one CTA per SM, each an equal share of all
// key tiles of the batch.
//
// Why: a CTA per pair of query tiles leaves SMs idle in the last wave (8 turns of up to 512 tokens behind 1536: 320 CTAs
// of unequal length on 148 SMs, 2.2 waves that take three) and spends ~8 us around its tiles (parameters, slots, first loads,
// first scores, last product, store) with idle tensor cores.  Here the items (request, head, pair of query tiles) stand
// in a row, an item as long as its key tiles plus kFlatItem for what comes once per item; CTA c takes positions
// [c, c + 1) * total / CTAs of that row, so ranges begin and end inside items.  The next item's K, V and Q are requested
// while the last products and the store of the one before run.  The plan is made on the device from the request lengths
// (a scan of at most kFlatMaxBs requests in every CTA), so nothing depends on the host's knowledge of them.
//
// A range of an item's keys leaves its unnormalised O, maximum and sum in the workspace: slot 2 c + 1 of a CTA that begins
// the item, 2 c of one that goes on with it.  attn_extend_flat_merge_kernel adds them in the order of the keys
// (deterministic); who begins an item writes how many go on with it.
//
// Bound by the softmax chain of a key tile as that kernel is (2.0 us a pair of tiles), by ~8 us an item that the next item's
// loads hide in part, and ~28 us once (plan, first loads, partial results through L2, merge).  us, other kernels / this (in rows
// of 8 calls, profiles/extend_flat_calls.json): groups of 4, 8 x up to 512 behind 1536 121 / 114, 2 x up to 390 behind 4192 84 /
// 70; groups of 5, 4 x 512 behind 8000 290 / 202; head size 64, 4 x up to 1000 behind 6000 205 / 150; but fresh 2 x 8192 972 /
// 1155: flat_pays in attn_extend.cu chooses.  Counters (the first of these): tensor pipe 40 %, exponential unit 41 % of the
// active clocks, 0.34 instructions a clock; the merge 12 us of 111, bound by reading its 39 MB.
//
// Warps, shared and tensor memory as in attn_extend_wide.cuh; three barriers more: Q is free, O of a tile is free.
#pragma once

namespace b200 {

constexpr int kFlatMaxBs = 512;
constexpr int kFlatItem = 2;        // weight of an item beside its key tiles
constexpr int kFlatMinCut = 2;      // no range of fewer key tiles at either end of an item
constexpr int kFlatMinShare = 8;    // least weight of a CTA

// What every warp of a CTA walks through: the items of its range of the row.  In shared memory, a copy per warp: the softmax
// warps have no registers to spare.
struct FlatWalk {
  int b, head, qb, off, rem;        // the next item, the position in it, what is left of the range
  int cb, chead, cqb, j0, j1, n, ext, prefix;   // the current item and its range of keys
  int64_t item0, citem0;            // positions of the next and of the current item
};

template <int D>
struct FlatCfg {
  using W = WideCfg<D>;
  static constexpr int N_BARS = W::N_BARS + 3;                       // + Q free, O free of both tiles
  static constexpr int OFF_WALK = W::OFF_BAR + N_BARS * 8 + 32;      // after tmem slot, gave up, CTAs, total
  static constexpr int SMEM_BYTES = OFF_WALK + (kWideThreads / 32) * static_cast<int>(sizeof(FlatWalk));
  static constexpr int SLOT_FLOATS = 256 * D + 512;                  // O as [D / 4][256 rows] float4, (m, l) of 256 rows
  static_assert(OFF_WALK % 8 == 0 && sizeof(FlatWalk) % 8 == 0, "walks");
  static_assert(kFlatMaxBs * 8 + 128 <= W::OFF_BAR, "the plan's scan aliases the operand tiles");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};
template <int D>
static size_t flat_workspace_bytes(int ctas) {
  return static_cast<size_t>(ctas) * (2 * FlatCfg<D>::SLOT_FLOATS * sizeof(float) + sizeof(int4));
}

// Key tiles of the item of query tiles qb, and where a cut at position p of the item falls
__host__ __device__ inline int flat_tiles(int prefix, int ext, int qb, int tok_cta, int causal) {
  const int last = min((qb + 1) * tok_cta, ext);
  return ceil_div(causal ? prefix + last : prefix + ext, kWideTile);
}
__host__ __device__ inline int flat_cut(int p, int n) {
  const int q = p - kFlatItem;
  if (p >= n + kFlatItem || n - q < kFlatMinCut) return n;
  return q < kFlatMinCut ? 0 : q;
}

__device__ __forceinline__ bool flat_next(volatile FlatWalk* s, const ExtendParams& p, int lane) {
  const int heads = p.Hkv * p.head_tiles, tok_cta = 256 / p.pack;
  int b = s->b, head = s->head, qb = s->qb, off = s->off, rem = s->rem;
  int64_t item0 = s->item0;
  bool found = false;
  __syncwarp();
  while (rem > 0 && !found) {
    const int ext = p.extend_lens[b], prefix = p.prefix_lens[b];
    if (ext <= 0) {
      ++b;
      continue;
    }
    const int n = flat_tiles(prefix, ext, qb, tok_cta, p.causal), w = n + kFlatItem;
    const int p1 = min(w, off + rem), j0 = flat_cut(off, n), j1 = flat_cut(p1, n);
    found = j0 < j1;
    if (found && lane == 0) {
      s->cb = b;
      s->chead = head;
      s->cqb = qb;
      s->j0 = j0;
      s->j1 = j1;
      s->n = n;
      s->ext = ext;
      s->prefix = prefix;
      s->citem0 = item0;
    }
    rem -= p1 - off;
    item0 += w;
    off = 0;
    if (++qb * tok_cta >= ext) {
      qb = 0;
      if (++head == heads) {
        head = 0;
        ++b;
      }
    }
  }
  if (lane == 0) {
    s->b = b;
    s->head = head;
    s->qb = qb;
    s->off = off;
    s->rem = rem;
    s->item0 = item0;
  }
  __syncwarp();
  return found;
}

template <typename T, int D>
__global__ void __launch_bounds__(kWideThreads, 1)
attn_extend_flat_kernel(const ExtendParams p, int bs, float* ws) {
  using C = WideCfg<D>;
  using F = FlatCfg<D>;
  constexpr int SL = C::SLOTS;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int tok_per_tile = 128 / p.pack;
  const int heads = p.Hkv * p.head_tiles, tok_cta = 2 * tok_per_tile;
  int4* desc = reinterpret_cast<int4*>(ws + static_cast<size_t>(gridDim.x) * 2 * F::SLOT_FLOATS);

  const uint32_t bars = sbase + C::OFF_BAR;
  const uint32_t bar_q = bars;
  auto bar_full = [&](int s) { return bars + 8u * (1 + s); };
  auto bar_empty = [&](int s) { return bars + 8u * (1 + SL + s); };
  auto bar_s = [&](int t) { return bars + 8u * (1 + 2 * SL + t); };        // scores of tile t are complete
  auto bar_p = [&](int t, int h) { return bars + 8u * (3 + 2 * SL + 2 * t + h); };  // half h of P of tile t is written
  auto bar_o = [&](int t) { return bars + 8u * (7 + 2 * SL + t); };        // PV of tile t is complete
  const uint32_t bar_qfree = bars + 8u * C::N_BARS;                        // every QK of the item is complete
  auto bar_ofree = [&](int t) { return bars + 8u * (C::N_BARS + 1 + t); }; // O of tile t has been read
  const uint32_t tmem_slot = bars + 8u * F::N_BARS, gave_up = tmem_slot + 4;
  volatile int* plan_ctas = reinterpret_cast<volatile int*>(smem + C::OFF_BAR + 8 * F::N_BARS + 8);
  volatile int64_t* plan_total = reinterpret_cast<volatile int64_t*>(smem + C::OFF_BAR + 8 * F::N_BARS + 16);
  volatile FlatWalk* walks = reinterpret_cast<volatile FlatWalk*>(smem + F::OFF_WALK);
  volatile FlatWalk& it = walks[warp];
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
      tc::mbar_init(bar_ofree(t), 128);
    }
    tc::mbar_init(bar_qfree, 1);
    asm volatile("st.shared.u32 [%0], 0;\n" ::"r"(gave_up) : "memory");
    tc::fence_barrier_init();
  }
  if (warp == 8) {
    tc::tmem_alloc(tmem_slot, 512);
    tc::tmem_relinquish();
  }
  griddep_wait();                                  // lengths, pages, new rows and the workspace are the launch's before
  // ---- the plan: weight of one head of every request, then this CTA's first position
  {
    int64_t* wsum = reinterpret_cast<int64_t*>(smem);
    for (int b = warp; b < bs; b += kWideThreads / 32) {
      const int ext = p.extend_lens[b], prefix = p.prefix_lens[b], nqb = ceil_div(max(ext, 0), tok_cta);
      int sum = 0;
      for (int i = lane; i < nqb; i += 32) sum += flat_tiles(prefix, ext, i, tok_cta, p.causal) + kFlatItem;
      sum = __reduce_add_sync(0xffffffffu, sum);
      if (lane == 0) wsum[b] = sum;
    }
    __syncthreads();
    if (warp == 0) {
      int64_t total = 0;
      for (int b0 = 0; b0 < bs; b0 += 32) {
        int64_t v = b0 + lane < bs ? wsum[b0 + lane] : 0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        total += v;
      }
      total *= heads;
      const int64_t share = total / kFlatMinShare;
      const int ctas = share < 1 ? 1 : share < static_cast<int64_t>(gridDim.x) ? static_cast<int>(share) : static_cast<int>(gridDim.x);
      const int c = blockIdx.x;
      const int64_t x0 = c < ctas ? total * c / ctas : 0, x1 = c < ctas ? total * (c + 1) / ctas : 0;
      // request of x0: a scan 32 requests at a time
      int64_t base = 0;
      int b = 0;
      for (int b0 = 0; b0 < bs; b0 += 32) {
        int64_t v = (b0 + lane < bs ? wsum[b0 + lane] : 0) * heads;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int64_t u = __shfl_up_sync(0xffffffffu, v, off);
          if (lane >= off) v += u;
        }
        const unsigned past = __ballot_sync(0xffffffffu, base + v > x0);
        if (past) {
          const int k = __ffs(past) - 1;
          const int64_t before = __shfl_sync(0xffffffffu, v, k > 0 ? k - 1 : 0);
          b = b0 + k;
          base += k > 0 ? before : 0;
          break;
        }
        base += __shfl_sync(0xffffffffu, v, 31);
      }
      int head = 0, qb = 0, off0 = 0;
      int64_t item0 = base;
      if (x1 > x0) {
        const int64_t w1 = wsum[b];
        head = static_cast<int>((x0 - base) / w1);
        item0 = base + head * w1;
        const int ext = p.extend_lens[b], prefix = p.prefix_lens[b], nqb = ceil_div(ext, tok_cta);
        for (int i0 = 0; i0 < nqb; i0 += 32) {
          int v = i0 + lane < nqb ? flat_tiles(prefix, ext, i0 + lane, tok_cta, p.causal) + kFlatItem : 0;
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, off);
            if (lane >= off) v += u;
          }
          const unsigned past = __ballot_sync(0xffffffffu, item0 + v > x0);
          if (past) {
            const int k = __ffs(past) - 1;
            const int before = __shfl_sync(0xffffffffu, v, k > 0 ? k - 1 : 0);
            qb = i0 + k;
            item0 += k > 0 ? before : 0;
            break;
          }
          item0 += __shfl_sync(0xffffffffu, v, 31);
        }
        off0 = static_cast<int>(x0 - item0);
      }
      if (lane < kWideThreads / 32) {
        volatile FlatWalk& f = walks[lane];
        f.b = b;
        f.head = head;
        f.qb = qb;
        f.off = off0;
        f.rem = static_cast<int>(x1 - x0);
        f.item0 = item0;
      }
      if (lane == 0) {
        *plan_ctas = ctas;
        *plan_total = total;
        desc[c] = make_int4(0, 0, 0, 0);
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem + C::OFF_BAR + 8 * F::N_BARS);

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kWideOtherRegs));
    if (warp > 8) {
      // ===================== gather =====================
      const int lt = static_cast<int>(threadIdx.x) - 9 * 32;
      constexpr int CPR = D / 8;                   // 16-byte chunks per row
      constexpr int RPP = kWideLoaders / CPR;      // rows per pass
      constexpr int PASSES = (kWideTile + RPP - 1) / RPP;
      const int lrow = lt / CPR, lcol = lt - lrow * CPR;
      const int64_t row_bytes = p.kv_row_stride * 2;
      // Unit u = a K or V tile goes to ring slot u % SL and is published up to LAG units later, when its copies have
      // landed (attn_extend_wide.cuh).
      constexpr int LAG = SL - 3;
      int u = 0, pub = 0, slot = 0, item = 0;
      uint32_t phase = 0;
      int pub_slot = 0;
      auto publish = [&]() {
        tc::fence_proxy_async_smem();
        if (pub == 0) tc::mbar_arrive(bar_q);      // the first item's Q came with unit 0
        tc::mbar_arrive(bar_full(pub_slot));
        if (++pub_slot == SL) pub_slot = 0;
        ++pub;
      };
      while (flat_next(&it, p, lane)) {
        const int ext = it.ext, j0 = it.j0, n_kv = it.j1 - j0, kv_len = it.prefix + ext;
        const int tok0 = it.cqb * tok_cta;
        const int tiles = tok0 + tok_per_tile < ext ? 2 : 1;
        const int kvh = it.chead / p.head_tiles;
        const int32_t* rtt = p.req_to_token + p.req_pool_indices[it.cb] * p.rtt_stride;
        const char* kbase = static_cast<const char*>(p.k_cache) + static_cast<int64_t>(kvh) * D * 2 + lcol * 16;
        const char* vbase = static_cast<const char*>(p.v_cache) + static_cast<int64_t>(kvh) * D * 2 + lcol * 16;
        int32_t slots[PASSES];
        auto load_slots = [&](int j) {
#pragma unroll
          for (int i = 0; i < PASSES; ++i) {
            const int r = lrow + RPP * i, pos = j * kWideTile + r;
            slots[i] = (r < kWideTile && pos < kv_len) ? __ldg(rtt + pos) : 0;   // 0 = the pool's dummy row
          }
        };
        auto load_q = [&]() {
          const int64_t q_row0 = p.extend_start[it.cb];
          const int head_base = kvh * p.group + (it.chead - kvh * p.head_tiles) * p.pack;
          for (int c = lt; c < tiles * 128 * CPR; c += kWideLoaders) {
            const int r = c / CPR, col = c - r * CPR, t = r >> 7, rr = r & 127;
            int tok = tok0 + r / p.pack;
            if (tok >= ext) tok = ext - 1;         // padding rows repeat the last token (never stored)
            const char* src = static_cast<const char*>(p.q) +
                              ((q_row0 + tok) * p.q_stride + (head_base + r % p.pack) * D) * 2 + col * 16;
            cp_async16(sbase + t * C::TILE_BYTES + swz_off<128>(rr, col), src);
          }
        };
        load_slots(j0);
        if (item == 0) load_q();                   // in the group of the first unit
        for (int j = 0; j < n_kv; ++j) {
#pragma unroll
          for (int kv = 0; kv < 2; ++kv) {
            if (u >= SL) tc::mbar_wait_bounded(bar_empty(slot), phase ^ 1u, dead, gave_up);
            const uint32_t dst = sbase + C::OFF_RING + slot * C::TILE_BYTES;
            const char* src = kv ? vbase : kbase;
#pragma unroll
            for (int i = 0; i < PASSES; ++i) {
              const int r = lrow + RPP * i;
              if (r < kWideTile) cp_async16(dst + swz_off<kWideTile>(r, lcol), src + static_cast<int64_t>(slots[i]) * row_bytes);
            }
            cp_async_commit();
            if (kv == 1 && j + 1 < n_kv) load_slots(j0 + j + 1);
            if (u - pub >= LAG) {
              cp_async_wait<LAG>();
              publish();
            }
            ++u;
            if (++slot == SL) {
              slot = 0;
              phase ^= 1u;
            }
          }
          if (j == 0 && item > 0) {
            // Q of this item behind its first K and V.  What the item before still needs is published before its last
            // QK is waited for.
            cp_async_wait<2>();
            while (pub < u - 2) publish();
            tc::mbar_wait_bounded(bar_qfree, (item - 1) & 1u, dead, gave_up);
            load_q();
            cp_async_commit();
            cp_async_wait<0>();
            tc::fence_proxy_async_smem();
            tc::mbar_arrive(bar_q);
            while (pub < u) publish();
          }
        }
        ++item;
      }
      cp_async_wait<0>();
      while (pub < u) publish();
    } else {
      // ===================== MMA issuer =====================
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc_qk = tc::make_idesc(fmt, fmt, 128, kWideTile, 0, 0);
      constexpr uint32_t idesc_pv = tc::make_idesc(fmt, fmt, 128, D, 0, 1);    // V: MN-major B
      const uint64_t qdesc = tc::make_smem_desc_sw128(sbase, 1024, 16);
      int slot = 0, item = 0;                      // ring slot of the next unit to wait for
      uint32_t phase = 0;
      uint32_t cnt[2] = {0u, 0u}, osub[2] = {0u, 0u};   // key tiles and items that a query tile has had
      auto wait_unit = [&]() {                     // -> its slot
        const int s = slot;
        tc::mbar_wait_bounded(bar_full(s), phase, dead, gave_up);
        tc::tc_fence_after();
        if (++slot == SL) {
          slot = 0;
          phase ^= 1u;
        }
        return s;
      };
      auto issue_qk = [&](int t, int s, bool last, bool item_last) {
        const uint64_t kdesc = tc::make_smem_desc_sw128(sbase + C::OFF_RING + s * C::TILE_BYTES, 1024, 16);
        if (tc::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = ((kk >> 2) * (128 * 128) + (kk & 3) * 32) >> 4;
            tc::mma_f16(tmem_base + t * 128, qdesc + t * (C::TILE_BYTES >> 4) + off, kdesc + off, idesc_qk, kk != 0 ? 1u : 0u);
          }
          tc::mma_commit(bar_s(t));
          if (last) tc::mma_commit(bar_empty(s));  // both tiles have used this K tile
          if (last && item_last) tc::mma_commit(bar_qfree);
        }
        __syncwarp();
      };
      while (flat_next(&it, p, lane)) {
        const int tiles = it.cqb * tok_cta + tok_per_tile < it.ext ? 2 : 1;
        const int n_kv = it.j1 - it.j0;
        tc::mbar_wait_bounded(bar_q, item & 1u, dead, gave_up);
        int ks = wait_unit();
        for (int t = 0; t < tiles; ++t) issue_qk(t, ks, t == tiles - 1, n_kv == 1);
        for (int j = 0; j < n_kv; ++j) {
          const int s = wait_unit();
          const uint64_t vdesc = tc::make_smem_desc_sw128(sbase + C::OFF_RING + s * C::TILE_BYTES, 1024, kWideTile * 128);
          for (int t = 0; t < tiles; ++t) {
            if (j == 0 && osub[t] > 0) {           // O of the item before has been read
              tc::mbar_wait_bounded(bar_ofree(t), (osub[t] - 1) & 1u, dead, gave_up);
              tc::tc_fence_after();
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {          // the first 64 keys are multiplied while the others' P is made
              tc::mbar_wait_bounded(bar_p(t, h), cnt[t] & 1u, dead, gave_up);
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
            ++cnt[t];
            if (j + 1 < n_kv) {
              if (t == 0) ks = wait_unit();
              issue_qk(t, ks, t == tiles - 1, j + 2 == n_kv);    // overwrites P(j) of this tile: MMAs run in issue order
            }
          }
        }
        for (int t = 0; t < tiles; ++t) ++osub[t];
        ++item;
      }
    }
  } else {
    // ===================== softmax / epilogue =====================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kWideSoftmaxRegs));
    const int t = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tmem_s = tmem_base + lane_addr + t * 128;
    const uint32_t tmem_o = tmem_base + lane_addr + C::O_COL + t * D;
    const float2 sc2 = make_float2(p.qk_scale, p.qk_scale), one2 = make_float2(1.f, 1.f);
    uint32_t cnt = 0;                              // key tiles that this query tile has had
    while (flat_next(&it, p, lane)) {
      const int tok0 = it.cqb * tok_cta;
      if (t > 0 && tok0 + tok_per_tile >= it.ext) continue;
      const int tok = tok0 + t * tok_per_tile + r / p.pack;
      const int limit = p.causal ? it.prefix + min(tok, it.ext - 1) : it.prefix + it.ext - 1;    // last visible key
      const int j0 = it.j0, j1 = it.j1;
      float m = -INFINITY, l = 0.f;
      for (int j = j0; j < j1; ++j, ++cnt) {
        tc::mbar_wait_bounded(bar_s(t), cnt & 1u, dead, gave_up);
        tc::tc_fence_after();
        __syncwarp();
        uint32_t v[4][32];
        tc::tmem_ld32(tmem_s, v[0]);
        tc::tmem_ld32(tmem_s + 32, v[1]);
        tc::tmem_ld_wait();
        tc::tmem_ld32(tmem_s + 64, v[2]);
        tc::tmem_ld32(tmem_s + 96, v[3]);
        const int k0 = j * kWideTile;
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
          if (j > j0) {
            tc::mbar_wait_bounded(bar_o(t), (cnt - 1) & 1u, dead, gave_up);    // O holds the range's tiles before j
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
      tc::mbar_wait_bounded(bar_o(t), (cnt - 1) & 1u, dead, gave_up);
      tc::tc_fence_after();
      __syncwarp();
      if (j0 > 0 || j1 < it.n) {
        // a part of the item's keys: unnormalised O, maximum and sum
        float* part = ws + (static_cast<size_t>(blockIdx.x) * 2 + (j0 == 0 ? 1 : 0)) * F::SLOT_FLOATS;
        float4* po = reinterpret_cast<float4*>(part) + t * 128 + r;
#pragma unroll 1
        for (int cc = 0; cc < D / 16; ++cc) {
          uint32_t o[16];
          tc::tmem_ld16(tmem_o + cc * 16, o);
          tc::tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i)
            __stcg(po + (cc * 4 + i) * 256, make_float4(__uint_as_float(o[4 * i]), __uint_as_float(o[4 * i + 1]),
                                                        __uint_as_float(o[4 * i + 2]), __uint_as_float(o[4 * i + 3])));
        }
        __stcg(reinterpret_cast<float2*>(part + 256 * D) + t * 128 + r, make_float2(m, l));
        if (threadIdx.x == 0 && j0 == 0) {         // this CTA begins the item: how many go on with it
          const int ctas = *plan_ctas;
          const int64_t total = *plan_total;
          int more = 0;
          for (int c = blockIdx.x + 1; c < ctas; ++c) {
            const int64_t at = total * c / ctas - it.citem0;
            if (at >= it.n + kFlatItem || flat_cut(static_cast<int>(at), it.n) >= it.n) break;
            ++more;
          }
          desc[blockIdx.x] = make_int4(it.cb, it.chead, it.cqb, more);
        }
      } else {
        // ---- O / l -> out
        const bool row_ok = tok < it.ext;
        const int kvh = it.chead / p.head_tiles;
        const int head_base = kvh * p.group + (it.chead - kvh * p.head_tiles) * p.pack;
        const float inv_l = l > 0.f ? p.out_scale / l : 0.f;
        T* orow = static_cast<T*>(p.o) + (p.extend_start[it.cb] + static_cast<int64_t>(row_ok ? tok : 0)) * p.o_stride +
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
      tc::tc_fence_before();
      tc::mbar_arrive(bar_ofree(t));
    }
  }
  griddep_launch_dependents();
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc::report_gave_up(gave_up, p.wait_error);
    tc::tmem_dealloc(tmem_base, 512);
  }
}

// Adds the parts of the items that more than one CTA worked on.  Block (c, g): 16 columns (g) of the 256 rows of the item
// that CTA c began; a thread has a row, so that reads are coalesced and a store is a whole sector.
template <typename T, int D>
__global__ void __launch_bounds__(256)
attn_extend_flat_merge_kernel(const ExtendParams p, const float* ws, int ctas) {
  using F = FlatCfg<D>;
  griddep_wait();
  const int c0 = blockIdx.x;
  const int4 d = __ldcg(reinterpret_cast<const int4*>(ws + static_cast<size_t>(ctas) * 2 * F::SLOT_FLOATS) + c0);
  if (d.w == 0) return;
  const int r = threadIdx.x, ext = p.extend_lens[d.x];
  const int tok = d.z * (256 / p.pack) + r / p.pack;   // row r of the two tiles
  if (tok >= ext) return;
  float M = -INFINITY, den = 0.f;
  float acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.f;
  for (int k = 0; k <= d.w; ++k) {
    const float* part = ws + (static_cast<size_t>(c0 + k) * 2 + (k == 0 ? 1 : 0)) * F::SLOT_FLOATS;
    const float2 ml = __ldcg(reinterpret_cast<const float2*>(part + 256 * D) + r);
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = __ldcg(reinterpret_cast<const float4*>(part) + (blockIdx.y * 4 + i) * 256 + r);
    const float Mn = fmaxf(M, ml.x);
    const float wo = M == -INFINITY ? 0.f : fast_exp2(M - Mn), wn = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - Mn);
    M = Mn;
    den = den * wo + ml.y * wn;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[4 * i] = acc[4 * i] * wo + x[i].x * wn;
      acc[4 * i + 1] = acc[4 * i + 1] * wo + x[i].y * wn;
      acc[4 * i + 2] = acc[4 * i + 2] * wo + x[i].z * wn;
      acc[4 * i + 3] = acc[4 * i + 3] * wo + x[i].w * wn;
    }
  }
  const float inv = den > 0.f ? p.out_scale / den : 0.f;
  const int kvh = d.y / p.head_tiles;
  const int head = kvh * p.group + (d.y - kvh * p.head_tiles) * p.pack + r % p.pack;
  T* dst = static_cast<T*>(p.o) + (p.extend_start[d.x] + static_cast<int64_t>(tok)) * p.o_stride +
           static_cast<int64_t>(head) * D + blockIdx.y * 16;
  uint32_t w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = pack16<T>(acc[2 * e] * inv, acc[2 * e + 1] * inv);
  *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
  *reinterpret_cast<uint4*>(dst + 8) = make_uint4(w[4], w[5], w[6], w[7]);
}

template <typename T, int D>
static int launch_extend_flat(const ExtendParams& p_in, int bs, float* ws, size_t ws_bytes, cudaStream_t st) {
  const int ctas = device_sm_count();
  B200_REQUIRE(bs <= kFlatMaxBs && ws && aligned16(ws) && ws_bytes >= flat_workspace_bytes<D>(ctas),
               "attn_extend_flat: %d requests, workspace of %zu bytes (needs %zu)", bs, ws_bytes, flat_workspace_bytes<D>(ctas));
  ExtendParams p = p_in;
  if (const int rc = wait_error_arm("attn_extend", &p.wait_error)) return rc;
  constexpr int SMEM = FlatCfg<D>::SMEM_BYTES;
  B200_CUDA_OK(cudaFuncSetAttribute(attn_extend_flat_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
  note_variant("attn_extend_wide flat d=%d ctas=%d", D, ctas);
  {
    ScopedKernelTimer timer("attn_extend", st);
    B200_CUDA_OK(launch_kernel(attn_extend_flat_kernel<T, D>, dim3(ctas), dim3(kWideThreads), SMEM, st, 1, extend_pdl(), p, bs, ws));
    B200_CHECK_LAUNCH("attn_extend_flat_kernel");
    B200_CUDA_OK(launch_kernel(attn_extend_flat_merge_kernel<T, D>, dim3(ctas, D / 16), dim3(256), 0, st, 1, kPdlMerge, p,
                               static_cast<const float*>(ws), ctas));
  }
  B200_CHECK_LAUNCH("attn_extend_flat_merge_kernel");
  return 0;
}

}  // namespace b200
