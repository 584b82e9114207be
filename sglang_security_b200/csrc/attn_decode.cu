// Paged split-KV decode attention for sm_100a.
//
// Path replaced: AttentionBackend.forward_decode (numerical oracle
// torch_native_backend.py:112-180; GPU reference triton_ops/decode_attention.py:50-557).
//
// Work decomposition
//   grid = (num_splits, Hkv * head_tiles, bs).  One CTA owns one (request, kv head, KV split) and
//   ALL query heads of that kv head's GQA group (up to 16 per head tile), so every K/V row is
//   fetched from HBM exactly once per group.  The KV pool is token-granular (page_size 1): row
//   `slot = req_to_token[req, t]` of k_cache/v_cache, D contiguous elements per kv head.
//   The kernel reads req_to_token directly — no flat kv_indices round trip.
//
// Data movement (the HBM-bound part)
//   Each warp runs its own STAGES-deep cp.async ring (16-byte LDGSTS, L2-only) over NT-token
//   tiles of gathered K and V rows; slot ids are fetched one tile ahead with 16-byte loads.
//   No CTA-wide barrier in the main loop.
//
// Math
//   Q.K^T and P.V of the whole GQA group on mma.sync m16n8k16 (rows = query heads), fp32
//   accumulators and fp32 online softmax in registers (exp2 domain, scale*log2e folded in).
//   Warps are merged once through shared memory; partials (normalised O, log2-domain LSE) go to
//   the workspace and are merged by attn_merge_kernel.
#include <cstdlib>
#include <type_traits>

#include "common.cuh"

namespace b200 {

struct DecodeParams {
  const void* q;
  int64_t q_stride;
  const void* k_cache;
  const void* v_cache;
  int64_t kv_row_stride;
  void* o;
  int64_t o_stride;
  const int32_t* req_to_token;
  int64_t rtt_stride;
  const int64_t* req_pool_indices;
  const int64_t* seq_lens;
  float* part_o;
  float* part_lse;
  int bs, Hq, Hkv, group, head_tiles;
  int num_splits;
  float qk_scale;   // scale*log2e, or plain scale when logit_cap > 0
  float logit_cap;  // <= 0: disabled
  float v_scale;    // FP8 KV pool only: output multiplier (k_scale is folded into qk_scale)
  int pdl_late;
  // Fused tail (b200_attn_decode*_fused, see decode_fused_tail): split partials are merged and,
  // optionally, the output row is quantised to e4m3 per token inside this kernel — the merge kernel
  // and the o_proj input quantiser disappear from the step.
  unsigned* tickets;     // [bs * (1 + gridDim.y)], zero before the first launch, self-resetting
  uint8_t* q_out;        // [bs, q_out_stride] e4m3 or null
  int64_t q_out_stride;
  float* q_scales;       // [bs]
  // rows of a mixed step (b200_attn_decode_rows): entry b is row row_list[b] of q and o (NULL: row b)
  const int32_t* row_list;
  // optional output gate [rows, gate_stride] in T: o is multiplied by sigmoid(gate[row, head * D + d])
  const void* gate;
  int64_t gate_stride;
  // PIECES instances: the batch is cut into this many pieces at most (decode_piece); grid.x is the piece
  int pieces;
  int2* plan;                   // [bs] first partial row and count of a request, for the merge
};

// b200_attn_decode_layer: entry b's new K/V row [Hkv, D] in T, stored to slot loc[b] of the pool before it is read (null: the
// pool holds it already); new_all: every CTA stores the rows of all entries (see store_new_rows).  Kernels that take these
// parameters are instances of their own: with the stores in them, the others were slower by up to 7 % on short requests (us,
// behind a write launch, 41 x 105 tokens of head size 64 5.06 -> 4.71, 6 x up to 92 4.75 -> 4.65, 64 x 600 30.4 -> 30.2).
struct DecodeParamsNew : DecodeParams {
  const void* new_k;
  const void* new_v;
  int64_t new_k_stride, new_v_stride;
  const int64_t* loc;
  float k_scale_w, v_scale_w;   // FP8 pool: divisors of the stored rows, where scale_new
  int scale_new, new_all;
};

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kNegBig = -1.0e30f;

// Tokens per split for a request of `len` tokens: equal parts rounded up to `align` tokens so
// that decode and merge agree on which splits are non-empty.
__host__ __device__ inline int split_chunk(int len, int num_splits, int align) {
  int c = ceil_div(len, num_splits);
  c = ceil_div(c, align) * align;
  return c < align ? align : c;
}

// ------------------------------------------------------------------------------------------------
// The dot products of a GQA group run on mma.sync m16n8k16 (rows = query heads of the group,
// padded to 16), so the per-token instruction count does not scale with the group size and the
// SM front end stays far below the HBM-bound gather stream (a CUDA-core FFMA version of this
// kernel was issue-bound at 78 % of the HBM peak).
//
//   S[16 heads, NT tokens] = Q[16, D] . K^T   (K rows from swizzled smem via ldmatrix)
//   P = exp2(S*scale - m)  (fp32 registers; the accumulator layout of S is the A layout of P)
//   O[16, D] += P[16, NT] . V[NT, D]          (V via ldmatrix.trans)
//
// Each warp still owns its private STAGES-deep cp.async ring of NT-token tiles.  Every lane copies
// column (lane % CPR) of RPG consecutive rows, so its slot ids are RPG consecutive int32 of
// req_to_token: fetched one tile ahead with 16-byte loads, no shuffles in the issue loop.
// 16-byte chunk c of row r is stored at chunk (c ^ (r & 7)) => ldmatrix is bank-conflict free.
template <int D, int NT, int STAGES, int NW>
struct MmaCfg {
  static constexpr int CPR = D / 8;            // 16-byte chunks per row
  static constexpr int RG = 32 / CPR;          // row groups copied concurrently by a warp
  static constexpr int RPG = NT / RG;          // consecutive rows per lane
  static constexpr int ROW_BYTES = D * 2;
  static constexpr int STAGE_BYTES = NT * ROW_BYTES * 2;  // K rows then V rows
  static constexpr int THREADS = NW * 32;
  static constexpr int ALIGN = NW * NT;
  static constexpr int RING_BYTES = NW * STAGES * STAGE_BYTES;
  static constexpr int FINAL_BYTES = NW * 16 * (D + 2) * 4;
  static constexpr int SMEM_BYTES = RING_BYTES > FINAL_BYTES ? RING_BYTES : FINAL_BYTES;
  static_assert(RPG % 4 == 0, "slot ids are fetched as int4");
  static_assert(NT % 16 == 0, "PV k-step is 16 tokens");
};

template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1);
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4],
                                                        uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma16816<__half>(float (&c)[4], const uint32_t (&a)[4],
                                                 uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}


// ---- pieces of equal length, for batches of unequal requests --------------------------------------------------------
// A split count for all requests cuts the long ones into long pieces and the short ones into short ones, and the long
// pieces run alone at the end.  Here the batch is cut into at most `pieces` pieces of about equal length, one wave of CTAs:
// the least length T (in ALIGN tokens) that gives no more than that, found by bisection over the lengths in the warp's
// registers, then a prefix sum over the requests' piece counts.  Every warp of every CTA does it for itself (~0.5 us) from
// the lengths on the device, so a captured launch follows them.  us, splits / pieces (random lengths, 32 / 8 heads of 128):
// bf16 16 x up to 6000 51.2 -> 43.0, 32 x up to 1000 20.2 -> 16.0; e4m3 27 x up to 6000 46.8 -> 42.8, 32 x up to 3000 35.2
// -> 28.7.  Tried: exact equal pieces, ranges that begin and end inside requests; a CTA then starts on up to two requests,
// which costs what the even end gives below ~1000 tokens a CTA (e4m3 48 x up to 1500: splits 27.2, pieces 21.3, shares 25.0).
constexpr int kPieceMaxBatch = 128;
struct DecodePiece {
  int b, start, end, len, count;   // b < 0: no such piece
  unsigned empty[kPieceMaxBatch / 32];   // entries without tokens
};
__device__ __forceinline__ DecodePiece decode_piece(const int64_t* seq_lens, int bs, int pieces, int x, int align, int lane) {
  constexpr int R = kPieceMaxBatch / 32;
  int u[R];
  int total = 0, longest = 1;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = r * 32 + lane;
    const int len = i < bs ? static_cast<int>(seq_lens[i]) : 0;
    u[r] = len > 0 ? (len + align - 1) / align : 0;
    total += u[r];
    longest = max(longest, u[r]);
  }
  total = __reduce_add_sync(0xffffffffu, total);
  longest = __reduce_max_sync(0xffffffffu, longest);
  // ceil(a / T) for a >= 1: (a - 0.5) / T never rounds across a whole number below 2^22
  auto count_of = [](int a, float inv) { return a ? static_cast<int>((static_cast<float>(a) - 0.5f) * inv) + 1 : 0; };
  int lo = max(1, total / pieces), hi = longest;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const float inv = 1.0f / static_cast<float>(mid);
    int n = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) n += count_of(u[r], inv);
    if (__reduce_add_sync(0xffffffffu, n) <= pieces) hi = mid;
    else lo = mid + 1;
  }
  const float inv = 1.0f / static_cast<float>(lo);
  DecodePiece out = {-1, 0, 0, 0, 0, {}};
  int before = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (r * 32 >= bs) break;
    out.empty[r] = __ballot_sync(0xffffffffu, r * 32 + lane < bs && u[r] == 0);
    const int n = count_of(u[r], inv);
    int incl = n;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, x < before + incl);
    if (out.b < 0 && hit) {
      const int src = __ffs(hit) - 1;
      const int units = __shfl_sync(0xffffffffu, u[r], src);
      out.count = __shfl_sync(0xffffffffu, n, src);
      const int j = x - before - (__shfl_sync(0xffffffffu, incl, src) - out.count);
      out.b = r * 32 + src;
      out.len = static_cast<int>(seq_lens[out.b]);
      const int chunk = (units + out.count - 1) / out.count * align;   // gives `count` pieces again, none empty
      out.start = j * chunk;
      out.end = min(out.len, out.start + chunk);
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
  return out;
}

// One warp stores entry b's new K and V rows of one kv head to the pool, 16 bytes of the source a lane and pass.  A KV write
// launch of its own costs 0.5 to 1.5 us in front of every layer's attention; the store's latency hides beside the page
// table's.  Two forms, and who may read a new slot in the same launch differs:
//  own slots   (the caller says so): entry b's page table names loc[b] at position seq_lens[b] - 1 or nowhere, and no other
//              entry's new slot.  The warp whose last tile holds the new token stores the row, nothing else reads it.
//  new_all     any page table (two positions of one request as two entries, a fork of a request beside it): the warps of
//              every CTA store the rows of all entries, and the CTA synchronises before it reads the pool.  CTAs store the
//              same bytes, so what a CTA reads behind its own store does not depend on the others.  Up to kNewRowsAll
//              entries; beyond, the stores cost what the write launch does or more.
// us, calls in a graph, own slots / new_all / write launch, bf16, 32 / 8 heads of 128: 1 x 1500 6.48 / 6.34 / 7.18, 2 x 1500
// 7.57 / 7.93 / 8.47, 2 x 8000 14.1 / 14.6 / 15.5, 3 x 8000 17.7 / 18.4 / 17.4, 4 x 8000 28.0 / 29.1 / 29.4, 16 x 1024 13.0 /
// 15.1 / 14.2, 64 x 4096 160.3 / 169.8 / 161.9; e4m3 2 x 8000 11.5 / 11.9 / 12.3, 27 x up to 6000 42.1 / 46.9 / 43.6, 8 / 2
// heads 4 x 8000 10.5 / 11.1 / 10.5.
constexpr int kNewRowsAll = 2;
template <typename T, int D, bool FP8, bool E5M2>
__device__ __forceinline__ void store_new_rows(const DecodeParamsNew& p, int b, int kvh, int lane) {
  constexpr int CPR = D / 8;
  const int64_t slot = p.loc[b];
#pragma unroll
  for (int i = lane; i < 2 * CPR; i += 32) {
    const bool is_v = i >= CPR;
    const int c = i - (is_v ? CPR : 0);
    const T* src = static_cast<const T*>(is_v ? p.new_v : p.new_k) + b * (is_v ? p.new_v_stride : p.new_k_stride) + kvh * D + c * 8;
    char* dst = const_cast<char*>(static_cast<const char*>(is_v ? p.v_cache : p.k_cache));
    const uint4 raw = *reinterpret_cast<const uint4*>(src);
    if (FP8) {
      const T* e = reinterpret_cast<const T*>(&raw);
      const float scale = is_v ? p.v_scale_w : p.k_scale_w;
      uint32_t lo = 0, hi = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lo |= to_fp8_torch<T>(e[j], scale, p.scale_new != 0, E5M2) << (8 * j);
        hi |= to_fp8_torch<T>(e[4 + j], scale, p.scale_new != 0, E5M2) << (8 * j);
      }
      *reinterpret_cast<uint2*>(dst + slot * p.kv_row_stride + kvh * D + c * 8) = make_uint2(lo, hi);
    } else {
      *reinterpret_cast<uint4*>(dst + (slot * p.kv_row_stride + kvh * D + c * 8) * 2) = raw;
    }
  }
}

// ---- fused tail: merge of the split partials (+ per-token FP8 quantisation) inside the kernel ----
// Two levels of ticket counters (threadFenceReduction pattern; bar.sync + one gpu-scope acq_rel
// atomic by thread 0 orders the CTA's stores before the draw and the winner's loads after it):
//   level 1, one counter per (request, kv-head tile): the LAST of the nvalid split CTAs of that tile
//            merges the partials of its own query heads — same arithmetic as attn_merge_kernel
//            (num * 1/den, one rounding to T) — and writes them to the 16-bit output row;
//   level 2, one counter per request (only when q_out is requested): the last tile to finish
//            quantises the whole row exactly as fp8_quant_per_token_kernel would (scale = amax / 448,
//            q = sat(x * (1/scale)) on the rounded 16-bit values).
// The merge work is spread over all (request, tile) pairs instead of one CTA per request; counters
// re-arm themselves, so CUDA-graph replays need no memset.
// Ticket words: [0, bs) level 2, bs + b * gridDim.y + blockIdx.y level 1.
struct TailDev {
  unsigned* tickets;
  uint8_t* q_out;
  int64_t q_out_stride;
  float* q_scales;
  void* o;
  int64_t o_stride;
  const float* part_o;
  const float* part_lse;
  int Hq, num_splits, bs;
};
__device__ __forceinline__ TailDev tail_of(const DecodeParams& p) {
  TailDev t;
  t.tickets = p.tickets;
  t.q_out = p.q_out;
  t.q_out_stride = p.q_out_stride;
  t.q_scales = p.q_scales;
  t.o = p.o;
  t.o_stride = p.o_stride;
  t.part_o = p.part_o;
  t.part_lse = p.part_lse;
  t.Hq = p.Hq;
  t.num_splits = p.num_splits;
  t.bs = p.bs;
  return t;
}

// true on every thread of the CTA that drew the last of `total` tickets (and re-arms the counter)
__device__ __forceinline__ bool draw_last_ticket(unsigned* ticket, unsigned total, unsigned* s_flag) {
  __syncthreads();  // every thread's stores are ordered before thread 0's release
  if (threadIdx.x == 0) {
    unsigned prev;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n"
                 : "=r"(prev) : "l"(ticket) : "memory");
    const bool last = prev + 1 == total;
    if (last) *ticket = 0u;  // every other participant has drawn: safe to re-arm
    *s_flag = last ? 1u : 0u;
  }
  __syncthreads();
  return *s_flag != 0u;
}

template <typename T, int THREADS>
__device__ __noinline__ void decode_fused_tail(const TailDev p, int b, int hq0, int heads_here,
                                               int nvalid, int D) {
  __shared__ unsigned s_flag;
  __shared__ float s_red[THREADS / 32];
  const int NS = p.num_splits;
  T* orow = static_cast<T*>(p.o) + static_cast<int64_t>(b) * p.o_stride;
  if (NS > 1) {
    if (!draw_last_ticket(p.tickets + p.bs + b * gridDim.y + blockIdx.y,
                          static_cast<unsigned>(nvalid), &s_flag))
      return;
    for (int it = threadIdx.x; it < heads_here * D / 4; it += THREADS) {
      const int e0 = it * 4, h = e0 / D, d = e0 - h * D;
      const int hq = hq0 + h;
      const int64_t base = (static_cast<int64_t>(b) * p.Hq + hq) * NS;
      float M = -INFINITY;
      for (int s = 0; s < nvalid; ++s) M = fmaxf(M, __ldcg(p.part_lse + base + s));
      float den = 0.f, num[4] = {0.f, 0.f, 0.f, 0.f};
      for (int s = 0; s < nvalid; ++s) {
        const float w = fast_exp2(__ldcg(p.part_lse + base + s) - M);
        const float4 x = __ldcg(reinterpret_cast<const float4*>(p.part_o + (base + s) * D + d));
        den += w;
        num[0] += w * x.x;
        num[1] += w * x.y;
        num[2] += w * x.z;
        num[3] += w * x.w;
      }
      const float inv = 1.f / den;
      uint2 pk;
      pk.x = pack2<T>(num[0] * inv, num[1] * inv);
      pk.y = pack2<T>(num[2] * inv, num[3] * inv);
      *reinterpret_cast<uint2*>(orow + hq * D + d) = pk;
    }
  }
  if (!p.q_out) return;
  if (!draw_last_ticket(p.tickets + b, gridDim.y, &s_flag)) return;
  // the whole 16-bit row of request b is final: per-token quantisation (two passes over 8 KiB of L2)
  const int n8 = p.Hq * D / 8;
  float amax = 0.f;
  for (int it = threadIdx.x; it < n8; it += THREADS) {
    const uint4 pk = __ldcg(reinterpret_cast<const uint4*>(orow) + it);
    const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 v = unpack2<T>(w[e]);
      amax = fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y)));
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = s_red[0];
#pragma unroll
  for (int w = 1; w < THREADS / 32; ++w) amax = fmaxf(amax, s_red[w]);
  const float scale = amax / 448.0f;
  if (threadIdx.x == 0) p.q_scales[b] = scale;
  const float inv = scale > 0.f ? 1.0f / scale : 0.f;
  uint8_t* qrow = p.q_out + static_cast<int64_t>(b) * p.q_out_stride;
  for (int it = threadIdx.x; it < n8; it += THREADS) {
    const uint4 pk = __ldcg(reinterpret_cast<const uint4*>(orow) + it);
    const uint32_t w[4] = {pk.x, pk.y, pk.z, pk.w};
    uint32_t q[2] = {0u, 0u};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 v = unpack2<T>(w[e]);
      const float x0 = fmaxf(fminf(v.x * inv, 448.0f), -448.0f);
      const float x1 = fmaxf(fminf(v.y * inv, 448.0f), -448.0f);
      uint16_t r;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;\n" : "=h"(r) : "f"(x1), "f"(x0));
      q[e >> 1] |= static_cast<uint32_t>(r) << (16 * (e & 1));
    }
    *reinterpret_cast<uint2*>(qrow + it * 8) = make_uint2(q[0], q[1]);
  }
}

}  // namespace b200
#include "attn_decode_fp8.cuh"
namespace b200 {

// HI: the tile holds more than 8 heads (rows 8..15 of the MMA are live).  ROWS: the row list and the output gate
// of b200_attn_decode_rows (an instance of its own: the others stay at their register limit without spills).
template <typename P, typename T, int D, int NT, int STAGES, int NW, bool HI, bool TAIL, bool ROWS = false, bool PIECES = false>
__global__ void __launch_bounds__(NW * 32, TAIL ? 4 : 0)
attn_decode_mma_kernel(const P p) {
  using C = MmaCfg<D, NT, STAGES, NW>;
  constexpr int CPR = C::CPR, RPG = C::RPG, ROW_BYTES = C::ROW_BYTES;
  constexpr int STAGE_BYTES = C::STAGE_BYTES;
  constexpr int KS = D / 16;   // k-steps of Q.K^T
  constexpr int NS = NT / 8;   // n-tiles (8 tokens) of S
  constexpr int NO = D / 8;    // n-tiles (8 dims) of O
  constexpr int GT = HI ? 16 : 8;

  extern __shared__ __align__(128) uint8_t smem[];
  griddep_wait();  // q, the new KV rows and seq_lens are written by the kernels before this one
  if (!p.pdl_late) griddep_launch_dependents();

  const int split = blockIdx.x;
  const int kvh = blockIdx.y / p.head_tiles;
  const int ht = blockIdx.y - kvh * p.head_tiles;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  constexpr bool NEW = std::is_same<P, DecodeParamsNew>::value;
  static_assert(!NEW || !(TAIL || ROWS), "new rows are written before these");
  int b = blockIdx.z, len, chunk = 0, start, end;
  bool whole = false;                    // PIECES: writes the output row, not a partial one
  if constexpr (PIECES) {
    const DecodePiece piece = decode_piece(p.seq_lens, p.bs, p.pieces, split, C::ALIGN, lane);
    if (split == 0 && warp == 0) {       // entries without tokens
#pragma unroll
      for (int r = 0; r < kPieceMaxBatch / 32; ++r)
        for (unsigned z = piece.empty[r]; z; z &= z - 1) {
          const int i = r * 32 + __ffs(z) - 1;
          if constexpr (NEW) store_new_rows<T, D, false, false>(p, i, kvh, lane);
          if (blockIdx.y == 0 && lane == 0) p.plan[i] = make_int2(0, 0);
        }
    }
    if (piece.b < 0) return;
    b = piece.b;
    len = piece.len;
    start = piece.start;
    end = piece.end;
    whole = piece.count == 1;
    if (start == 0 && blockIdx.y == 0 && threadIdx.x == 0) p.plan[b] = make_int2(split, piece.count);
  } else {
    len = static_cast<int>(p.seq_lens[b]);
    chunk = split_chunk(len, p.num_splits, C::ALIGN);
    start = split * chunk;
    if (start >= len) {
      if constexpr (NEW) {
        if (len <= 0 && split == 0 && warp == 0) store_new_rows<T, D, false, false>(p, b, kvh, lane);
      }
      return;
    }
    end = min(len, start + chunk);
  }
  const int ntiles = ceil_div(end - start, NT);
  const int n_my = warp < ntiles ? (ntiles - warp + NW - 1) / NW : 0;

  const int32_t* __restrict__ rtt = p.req_to_token + p.req_pool_indices[b] * p.rtt_stride;
  const int64_t row_stride_bytes = p.kv_row_stride * 2;
  const int head0 = ht * GT;
  const int heads_here = min(GT, p.group - head0);

  // ---- Q fragments (A operand, rows = heads) -------------------------------------------------
  uint32_t qa[KS][4];
  {
    const int r_lo = lane >> 2, r_hi = r_lo + 8;
    const T* qb = static_cast<const T*>(p.q) + static_cast<int64_t>(ROWS && p.row_list ? p.row_list[b] : b) * p.q_stride +
                  static_cast<int64_t>(kvh * p.group + head0) * D + (lane & 3) * 2;
    const bool v_lo = r_lo < heads_here, v_hi = HI && r_hi < heads_here;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      qa[ks][0] = v_lo ? *reinterpret_cast<const uint32_t*>(qb + r_lo * D + ks * 16) : 0u;
      qa[ks][2] = v_lo ? *reinterpret_cast<const uint32_t*>(qb + r_lo * D + ks * 16 + 8) : 0u;
      qa[ks][1] = v_hi ? *reinterpret_cast<const uint32_t*>(qb + r_hi * D + ks * 16) : 0u;
      qa[ks][3] = v_hi ? *reinterpret_cast<const uint32_t*>(qb + r_hi * D + ks * 16 + 8) : 0u;
    }
  }

  float o[NO][4];
#pragma unroll
  for (int i = 0; i < NO; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_lo = kNegBig, m_hi = kNegBig, l_lo = 0.f, l_hi = 0.f;

  // ---- copy-issue geometry ---------------------------------------------------------------------
  const int ccol = lane % CPR;         // 16-byte column this lane copies
  const int crow0 = (lane / CPR) * RPG;  // first of its RPG consecutive rows
  const char* kcol = static_cast<const char*>(p.k_cache) + static_cast<int64_t>(kvh) * ROW_BYTES +
                     ccol * 16;
  const char* vcol = static_cast<const char*>(p.v_cache) + static_cast<int64_t>(kvh) * ROW_BYTES +
                     ccol * 16;
  const uint32_t ring = smem_u32(smem) + warp * (STAGES * STAGE_BYTES);
  const bool rtt_vec = (p.rtt_stride & 3) == 0 && (reinterpret_cast<uintptr_t>(p.req_to_token) & 15) == 0;

  int slot[RPG];
  // SAFE: tile k exists and is a whole one, and the page table takes 16-byte loads
  auto load_slots = [&](int k, auto safe) {
    if (!safe.value && k >= n_my) return;
    const int pos = start + (warp + k * NW) * NT + crow0;
    if (safe.value || (rtt_vec && pos + RPG <= end)) {
#pragma unroll
      for (int i = 0; i < RPG / 4; ++i) {
        const int4 v = __ldg(reinterpret_cast<const int4*>(rtt + pos) + i);
        slot[4 * i + 0] = v.x; slot[4 * i + 1] = v.y; slot[4 * i + 2] = v.z; slot[4 * i + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < RPG; ++i) slot[i] = pos + i < end ? __ldg(rtt + pos + i) : 0;
    }
  };
  auto issue_tile = [&](int k, auto safe) {
    if (safe.value || k < n_my) {
      const uint32_t sk = ring + (k % STAGES) * STAGE_BYTES;
#pragma unroll
      for (int i = 0; i < RPG; ++i) {
        const int row = crow0 + i;
        const int64_t off = static_cast<int64_t>(slot[i]) * row_stride_bytes;
        const uint32_t dst = sk + row * ROW_BYTES + ((ccol ^ (row & 7)) << 4);
        cp_async16(dst, kcol + off);
        cp_async16(dst + NT * ROW_BYTES, vcol + off);
      }
    }
    cp_async_commit();
  };

  load_slots(0, std::false_type{});
  if constexpr (NEW) {
    if (p.new_all) {
      for (int i = warp; i < p.bs; i += NW) store_new_rows<T, D, false, false>(p, i, kvh, lane);
      __syncthreads();
    } else if (end == len && warp == (ntiles - 1) % NW) {   // this warp's last tile holds the new token
      store_new_rows<T, D, false, false>(p, b, kvh, lane);
      __syncwarp();
    }
  }
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    issue_tile(s, std::false_type{});
    load_slots(s + 1, std::false_type{});
  }

  const bool capped = p.logit_cap > 0.f;
  // qk_scale = plain scale if capped; in the units of exact_tanh_log2
  const float inv_cap = capped ? p.qk_scale / p.logit_cap * (2.0f * kLog2e) : 0.f;
  const float cap_log2 = p.logit_cap * kLog2e;
  const float sc_mul = capped ? 1.f : p.qk_scale;

  // ldmatrix lane geometry
  const int lx = lane & 7;
  const uint32_t k_row_off = lx * ROW_BYTES;                 // + nt * 8 * ROW_BYTES
  const int k_y = (lane >> 3) ^ lx;                          // chunk xor term (QK)
  const uint32_t v_row_off = (((lane >> 3) & 1) * 8 + lx) * ROW_BYTES;  // + kt * 16 * ROW_BYTES
  const int v_y = (lane >> 4) ^ lx;

  auto step = [&](int it, auto safe) {
    issue_tile(it + STAGES - 1, safe);
    load_slots(it + STAGES, safe);
    cp_async_wait<STAGES - 1>();
    __syncwarp();

    const uint32_t sk = ring + (it % STAGES) * STAGE_BYTES;
    const uint32_t sv = sk + NT * ROW_BYTES;
    const int tok0 = start + (warp + it * NW) * NT;

    // ---- S = Q . K^T ---------------------------------------------------------------------------
    float s[NS][4];
#pragma unroll
    for (int nt = 0; nt < NS; ++nt) {
      s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < KS; ks += 2) {
        uint32_t kb[4];
        ldsm_x4(kb, sk + nt * 8 * ROW_BYTES + k_row_off + (((2 * ks) ^ k_y) << 4));
        mma16816<T>(s[nt], qa[ks], kb[0], kb[1]);
        mma16816<T>(s[nt], qa[ks + 1], kb[2], kb[3]);
      }
    }
    if (capped) {
#pragma unroll
      for (int nt = 0; nt < NS; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[nt][e] = cap_log2 * exact_tanh_log2(s[nt][e] * inv_cap);
    }
    if (!safe.value && tok0 + NT > end) {  // tail tile: mask tokens past the end (warp-uniform branch)
#pragma unroll
      for (int nt = 0; nt < NS; ++nt) {
        const int t = tok0 + nt * 8 + (lane & 3) * 2;
        if (t >= end) s[nt][0] = s[nt][2] = -INFINITY;
        if (t + 1 >= end) s[nt][1] = s[nt][3] = -INFINITY;
      }
    }

    // ---- online softmax ----------------------------------------------------------------------
    float mt_lo = fmaxf(s[0][0], s[0][1]), mt_hi = fmaxf(s[0][2], s[0][3]);
#pragma unroll
    for (int nt = 1; nt < NS; ++nt) {
      mt_lo = fmaxf(mt_lo, fmaxf(s[nt][0], s[nt][1]));
      if (HI) mt_hi = fmaxf(mt_hi, fmaxf(s[nt][2], s[nt][3]));
    }
    mt_lo = fmaxf(mt_lo, __shfl_xor_sync(0xffffffffu, mt_lo, 1));
    mt_lo = fmaxf(mt_lo, __shfl_xor_sync(0xffffffffu, mt_lo, 2));
    const float mn_lo = fmaxf(m_lo, mt_lo * sc_mul);
    float mn_hi = m_hi;
    if (HI) {
      mt_hi = fmaxf(mt_hi, __shfl_xor_sync(0xffffffffu, mt_hi, 1));
      mt_hi = fmaxf(mt_hi, __shfl_xor_sync(0xffffffffu, mt_hi, 2));
      mn_hi = fmaxf(m_hi, mt_hi * sc_mul);
    }
    if (__any_sync(0xffffffffu, mn_lo > m_lo || (HI && mn_hi > m_hi))) {
      const float a_lo = fast_exp2(m_lo - mn_lo);
      const float a_hi = HI ? fast_exp2(m_hi - mn_hi) : 1.f;
      l_lo *= a_lo;
      l_hi *= a_hi;
#pragma unroll
      for (int i = 0; i < NO; ++i) {
        o[i][0] *= a_lo;
        o[i][1] *= a_lo;
        if (HI) {
          o[i][2] *= a_hi;
          o[i][3] *= a_hi;
        }
      }
      m_lo = mn_lo;
      m_hi = mn_hi;
    }
    uint32_t pa[NT / 16][4];
#pragma unroll
    for (int nt = 0; nt < NS; ++nt) {
      const float p0 = fast_exp2(fmaf(s[nt][0], sc_mul, -m_lo));
      const float p1 = fast_exp2(fmaf(s[nt][1], sc_mul, -m_lo));
      l_lo += p0 + p1;
      pa[nt >> 1][(nt & 1) * 2] = pack2<T>(p0, p1);
      if (HI) {
        const float p2 = fast_exp2(fmaf(s[nt][2], sc_mul, -m_hi));
        const float p3 = fast_exp2(fmaf(s[nt][3], sc_mul, -m_hi));
        l_hi += p2 + p3;
        pa[nt >> 1][(nt & 1) * 2 + 1] = pack2<T>(p2, p3);
      } else {
        pa[nt >> 1][(nt & 1) * 2 + 1] = 0u;
      }
    }

    // ---- O += P . V --------------------------------------------------------------------------
#pragma unroll
    for (int kt = 0; kt < NT / 16; ++kt) {
#pragma unroll
      for (int np = 0; np < NO / 2; ++np) {
        uint32_t vb[4];
        ldsm_x4_t(vb, sv + kt * 16 * ROW_BYTES + v_row_off + (((2 * np) ^ v_y) << 4));
        mma16816<T>(o[2 * np], pa[kt], vb[0], vb[1]);
        mma16816<T>(o[2 * np + 1], pa[kt], vb[2], vb[3]);
      }
    }
    __syncwarp();  // stage may be refilled by the next iteration's issue
  };
  // Tiles whose successors are whole ones run a copy of the step without their checks (us: 64 x 4096 bf16 166.8 -> 160.9,
  // 32 x up to 4000 of head size 64 15.6 -> 13.9, 1 x 1500 7.0 -> 6.6; e4m3 64 x 4096 100.3 -> 99.1).
  int it = 0;
  if (rtt_vec)
    for (; it + STAGES + 1 < n_my; ++it) step(it, std::true_type{});
  for (; it < n_my; ++it) step(it, std::false_type{});
  cp_async_wait<0>();
  if (p.pdl_late) griddep_launch_dependents();

  // ---- quad-reduce the row sums, merge warps through shared memory ---------------------------
  l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1);
  l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
  if (HI) {
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
  }
  __syncthreads();
  float* fin = reinterpret_cast<float*>(smem);   // [NW][16][D]
  float* fin_m = fin + NW * 16 * D;               // [NW][16]
  float* fin_l = fin_m + NW * 16;                 // [NW][16]
  {
    const int r_lo = lane >> 2, c0 = (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < NO; ++i) {
      *reinterpret_cast<float2*>(fin + (warp * 16 + r_lo) * D + i * 8 + c0) =
          make_float2(o[i][0], o[i][1]);
      if (HI)
        *reinterpret_cast<float2*>(fin + (warp * 16 + r_lo + 8) * D + i * 8 + c0) =
            make_float2(o[i][2], o[i][3]);
    }
    if ((lane & 3) == 0) {
      fin_m[warp * 16 + r_lo] = m_lo;
      fin_l[warp * 16 + r_lo] = l_lo;
      if (HI) {
        fin_m[warp * 16 + r_lo + 8] = m_hi;
        fin_l[warp * 16 + r_lo + 8] = l_hi;
      }
    }
  }
  __syncthreads();

  for (int idx = threadIdx.x; idx < heads_here * D; idx += NW * 32) {
    const int h = idx / D, d = idx - h * D;
    float M = fin_m[h];
#pragma unroll
    for (int w = 1; w < NW; ++w) M = fmaxf(M, fin_m[w * 16 + h]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float f = fast_exp2(fin_m[w * 16 + h] - M);  // idle warps: m = -1e30, l = 0 -> f = 0
      num += fin[(w * 16 + h) * D + d] * f;
      den += fin_l[w * 16 + h] * f;
    }
    float out = num / den;
    const int hq = kvh * p.group + head0 + h;
    if (PIECES ? whole : p.num_splits == 1) {
      const int64_t row = ROWS && p.row_list ? p.row_list[b] : b;
      if (ROWS && p.gate) out *= sigmoid_f(to_float<T>(static_cast<const T*>(p.gate)[row * p.gate_stride + hq * D + d]));
      static_cast<T*>(p.o)[row * p.o_stride + hq * D + d] = from_float<T>(out);
    } else {
      const int64_t pidx = PIECES ? static_cast<int64_t>(split) * p.Hq + hq
                                  : (static_cast<int64_t>(b) * p.Hq + hq) * p.num_splits + split;
      p.part_o[pidx * D + d] = out;
      if (d == 0) p.part_lse[pidx] = M + log2f(den);
    }
  }
  if constexpr (TAIL)
    decode_fused_tail<T, NW * 32>(tail_of(p), b, kvh * p.group + head0, heads_here, ceil_div(len, chunk), D);
}

// Merge of split partials: one warp per (query head, request), four columns per lane.  Latency-bound (a few hundred
// KB): the split sums are read by all lanes at once and the first partial rows are requested before the sequence length
// is known, so the chain is one round trip to L2, not one per split (1 request of 1500 tokens in 7 splits: 5.2 us, now
// 3.8).  BYCOLS, for more splits than the rows requested ahead and few heads: the four warps of a CTA share the columns
// of a head, one column per lane, so that 32 rows are requested together (64 splits are two round trips, not eight).
// Sums run over the splits in order, as in attn_merge_quant_kernel: same bytes.
constexpr int kMergeWarps = 4;

// V columns per lane: 4 (2: half-width rows), or 1 for rows that 16-byte loads do not fit
template <int V>
__device__ __forceinline__ void merge_load(float (&x)[V], const float* p) {
  if constexpr (V == 4) {
    const float4 f = __ldcg(reinterpret_cast<const float4*>(p));
    x[0] = f.x;
    x[1] = f.y;
    x[2] = f.z;
    x[3] = f.w;
  } else if constexpr (V == 2) {
    const float2 f = __ldcg(reinterpret_cast<const float2*>(p));
    x[0] = f.x;
    x[1] = f.y;
  } else {
    x[0] = __ldcg(p);
  }
}

template <typename T, int V, bool BYCOLS>
__global__ void __launch_bounds__(kMergeWarps * 32)
attn_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse, T* __restrict__ o,
                  int64_t o_stride, const int64_t* __restrict__ seq_lens, int Hq, int Dv, int num_splits, int align,
                  const int32_t* __restrict__ row_list, const T* __restrict__ gate, int64_t gate_stride) {
  griddep_wait();
  griddep_launch_dependents();
  constexpr int AHEAD = BYCOLS ? 32 : 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int hq = BYCOLS ? blockIdx.x : blockIdx.x * kMergeWarps + warp, b = blockIdx.y;
  if (hq >= Hq) return;
  const int64_t base = (static_cast<int64_t>(b) * Hq + hq) * num_splits;
  const float* po = part_o + base * Dv;
  // splits past the sequence are allocated but hold nothing: their values are not used
  float x[AHEAD][V];
  const int dd0 = BYCOLS ? warp * 32 * V : 0, step = BYCOLS ? kMergeWarps * 32 * V : 32 * V;
  const int d0 = dd0 + lane * V;
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < num_splits && d0 < Dv) merge_load<V>(x[i], po + static_cast<int64_t>(i) * Dv + d0);
  const float lse0 = lane < num_splits ? __ldcg(part_lse + base + lane) : 0.f;
  const int len = static_cast<int>(seq_lens[b]);
  if (len <= 0) return;
  const int nvalid = ceil_div(len, split_chunk(len, num_splits, align));
  float M = lane < nvalid ? lse0 : -INFINITY;
  for (int s = 32 + lane; s < nvalid; s += 32) M = fmaxf(M, __ldcg(part_lse + base + s));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
  const int64_t row = row_list ? row_list[b] : b;
  for (int dd = dd0; dd < Dv; dd += step) {
    const int d = dd + lane * V;
    float den = 0.f, num[V];
#pragma unroll
    for (int e = 0; e < V; ++e) num[e] = 0.f;
    for (int s0 = 0; s0 < nvalid; s0 += 32) {
      const float lse = s0 == 0 ? lse0 : (s0 + lane < nvalid ? __ldcg(part_lse + base + s0 + lane) : 0.f);
      const float w_lane = s0 + lane < nvalid ? fast_exp2(lse - M) : 0.f;
      for (int s1 = s0; s1 < min(nvalid, s0 + 32); s1 += AHEAD) {
        if (s1 > 0 || dd > dd0) {
#pragma unroll
          for (int i = 0; i < AHEAD; ++i)
            if (s1 + i < nvalid && d < Dv) merge_load<V>(x[i], po + static_cast<int64_t>(s1 + i) * Dv + d);
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
          const float w = __shfl_sync(0xffffffffu, w_lane, (s1 + i) & 31);
          if (s1 + i < nvalid) {
            den += w;
#pragma unroll
            for (int e = 0; e < V; ++e) num[e] += w * x[i][e];
          }
        }
      }
    }
    if (d >= Dv) continue;
    const float inv = 1.f / den;
    T* dst = o + row * o_stride + hq * Dv + d;
#pragma unroll
    for (int e = 0; e < V; ++e) {
      float y = num[e] * inv;
      if (gate) y *= sigmoid_f(to_float<T>(gate[row * gate_stride + hq * Dv + d + e]));
      dst[e] = from_float<T>(y);
    }
  }
}

// Merge behind the PIECES instances: one warp per head, piece s of request b in row first + s of the partials.  A request
// in one piece was written by the split kernel.  Sums run over the pieces in order.
template <typename T, int D>
__global__ void __launch_bounds__(kMergeWarps * 32)
attn_merge_pieces_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse, T* __restrict__ o,
                         int64_t o_stride, const int2* __restrict__ plan, int Hq) {
  constexpr int V = D / 32, AHEAD = 8;
  griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 31, b = blockIdx.y;
  const int hq = blockIdx.x * kMergeWarps + (threadIdx.x >> 5);
  if (hq >= Hq) return;
  const int2 pc = __ldcg(plan + b);
  const int count = pc.y;
  if (count <= 1) return;
  const float* lse = part_lse + static_cast<int64_t>(pc.x) * Hq + hq;
  const float* po = part_o + (static_cast<int64_t>(pc.x) * Hq + hq) * D + lane * V;
  const int64_t step = static_cast<int64_t>(Hq) * D;
  float x[AHEAD][V];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < count) merge_load<V>(x[i], po + i * step);
  const float lse0 = lane < count ? __ldcg(lse + static_cast<int64_t>(lane) * Hq) : -INFINITY;
  float M = lse0;
  for (int s = 32 + lane; s < count; s += 32) M = fmaxf(M, __ldcg(lse + static_cast<int64_t>(s) * Hq));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
  float den = 0.f, num[V];
#pragma unroll
  for (int e = 0; e < V; ++e) num[e] = 0.f;
  for (int s0 = 0; s0 < count; s0 += 32) {
    const float l = s0 == 0 ? lse0 : (s0 + lane < count ? __ldcg(lse + static_cast<int64_t>(s0 + lane) * Hq) : -INFINITY);
    const float w_lane = s0 + lane < count ? fast_exp2(l - M) : 0.f;
    for (int s1 = s0; s1 < min(count, s0 + 32); s1 += AHEAD) {
      if (s1 > 0) {
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
          if (s1 + i < count) merge_load<V>(x[i], po + (s1 + i) * step);
      }
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) {
        const float w = __shfl_sync(0xffffffffu, w_lane, (s1 + i) & 31);
        if (s1 + i < count) {
          den += w;
#pragma unroll
          for (int e = 0; e < V; ++e) num[e] += w * x[i][e];
        }
      }
    }
  }
  const float inv = 1.f / den;
  T* dst = o + static_cast<int64_t>(b) * o_stride + hq * D + lane * V;
#pragma unroll
  for (int e = 0; e < V; ++e) dst[e] = from_float<T>(num[e] * inv);
}

// Merge of split partials for ALL heads of a request + per-token FP8 quantisation of the merged
// row in one launch.  Replaces attn_merge_kernel followed by fp8_quant_per_token_kernel (same
// arithmetic in the same order, so the bytes are identical); with num_splits == 1 it only quantises
// the row the split kernel wrote.  A request is spread over a CLUSTER of S CTAs (128 threads, one
// 4-element item per thread and pass), the per-token amax is combined through distributed shared
// memory (a maximum, so the result does not depend on the split), every value stays in registers
// between the amax and the quantising pass.
constexpr int kMqThreads = 128;
constexpr int kMqMaxItems = 4;  // 4-element items per thread: covers Hq * Dv <= 8 * 128 * 4 * 4

template <typename T>
__global__ void __launch_bounds__(kMqThreads)
attn_merge_quant_kernel(const float* __restrict__ part_o, const float* __restrict__ part_lse,
                        T* __restrict__ o, int64_t o_stride, uint8_t* __restrict__ q_out,
                        int64_t q_stride, float* __restrict__ q_scales,
                        const int64_t* __restrict__ seq_lens, int Hq, int Dv, int num_splits,
                        int align, int per_cta) {
  __shared__ float red[kMqThreads / 32];
  __shared__ float cl_slots[8];
  uint32_t S, rank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(S));
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  if (S > 1)  // every CTA of the cluster runs before any remote store is issued
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  griddep_wait();
  griddep_launch_dependents();
  const int b = blockIdx.x / S;
  const int len = static_cast<int>(seq_lens[b]);
  T* orow = o + static_cast<int64_t>(b) * o_stride;
  const int n4 = Hq * Dv / 4;
  const int i0 = static_cast<int>(rank) * per_cta, i1 = min(n4, i0 + per_cta);
  const int chunk = split_chunk(max(len, 1), num_splits, align);
  const int nvalid = len > 0 ? ceil_div(len, chunk) : 0;
  uint2 vals[kMqMaxItems];
  float amax = 0.f;
#pragma unroll
  for (int k = 0; k < kMqMaxItems; ++k) {
    const int it = i0 + threadIdx.x + k * kMqThreads;
    vals[k] = make_uint2(0u, 0u);
    if (it < i1 && len > 0) {
      const int e0 = it * 4, h = e0 / Dv, d = e0 - h * Dv;
      if (num_splits > 1) {
        const int64_t base = (static_cast<int64_t>(b) * Hq + h) * num_splits;
        float M = -INFINITY;
#pragma unroll 8
        for (int s = 0; s < nvalid; ++s) M = fmaxf(M, __ldg(part_lse + base + s));
        float den = 0.f, num[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int s = 0; s < nvalid; ++s) {
          const float w = fast_exp2(__ldg(part_lse + base + s) - M);
          const float4 x = __ldg(reinterpret_cast<const float4*>(part_o + (base + s) * Dv + d));
          den += w;
          num[0] += w * x.x;
          num[1] += w * x.y;
          num[2] += w * x.z;
          num[3] += w * x.w;
        }
        const float inv = 1.f / den;
        vals[k].x = pack2<T>(num[0] * inv, num[1] * inv);
        vals[k].y = pack2<T>(num[2] * inv, num[3] * inv);
        *reinterpret_cast<uint2*>(orow + e0) = vals[k];
      } else {
        vals[k] = *reinterpret_cast<const uint2*>(orow + e0);
      }
      const float2 a = unpack2<T>(vals[k].x), c = unpack2<T>(vals[k].y);
      amax = fmaxf(fmaxf(amax, fmaxf(fabsf(a.x), fabsf(a.y))), fmaxf(fabsf(c.x), fabsf(c.y)));
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < kMqThreads / 32; ++w) amax = fmaxf(amax, red[w]);
  if (S > 1) {
    if (threadIdx.x < S) {  // thread j publishes this CTA's amax into CTA j's slot [rank]
      uint32_t local = smem_u32(cl_slots + rank), remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(local), "r"(threadIdx.x));
      asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(remote), "f"(amax) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    amax = cl_slots[0];
    for (uint32_t j = 1; j < S; ++j) amax = fmaxf(amax, cl_slots[j]);
  }
  if (len <= 0) return;
  const float scale = amax / 448.0f;
  if (threadIdx.x == 0 && rank == 0) q_scales[b] = scale;
  const float inv = scale > 0.f ? 1.0f / scale : 0.f;
  uint8_t* qrow = q_out + static_cast<int64_t>(b) * q_stride;
#pragma unroll
  for (int k = 0; k < kMqMaxItems; ++k) {
    const int it = i0 + threadIdx.x + k * kMqThreads;
    if (it < i1) {
      const float2 a = unpack2<T>(vals[k].x), c = unpack2<T>(vals[k].y);
      const float x0 = fmaxf(fminf(a.x * inv, 448.0f), -448.0f), x1 = fmaxf(fminf(a.y * inv, 448.0f), -448.0f);
      const float x2 = fmaxf(fminf(c.x * inv, 448.0f), -448.0f), x3 = fmaxf(fminf(c.y * inv, 448.0f), -448.0f);
      uint16_t lo, hi;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;\n" : "=h"(lo) : "f"(x1), "f"(x0));
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;\n" : "=h"(hi) : "f"(x3), "f"(x2));
      *reinterpret_cast<uint32_t*>(qrow + it * 4) = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
    }
  }
}

template <typename T>
static int launch_merge_quant(const DecodeParams& p, int Dv, int align, cudaStream_t st) {
  const int n4 = p.Hq * Dv / 4;
  int S = ceil_div(n4, kMqThreads);  // one item per thread where the cluster limit allows it
  if (S > 8) S = 8;
  const int per_cta = ceil_div(n4, S);
  B200_REQUIRE(per_cta <= kMqThreads * kMqMaxItems,
               "attn_merge_quant: row of %d x %d is too long for one cluster", p.Hq, Dv);
  auto kern = attn_merge_quant_kernel<T>;
  {
    ScopedKernelTimer timer("attn_merge_quant", st);
    B200_CUDA_OK(launch_kernel(kern, dim3(p.bs * S), dim3(kMqThreads), 0, st, S,
                               pdl_family(p.bs, kPdlMerge), static_cast<const float*>(p.part_o),
                               static_cast<const float*>(p.part_lse), static_cast<T*>(p.o), p.o_stride,
                               p.q_out, p.q_out_stride, p.q_scales, p.seq_lens, p.Hq, Dv, p.num_splits,
                               align, per_cta));
  }
  B200_CHECK_LAUNCH("attn_merge_quant_kernel");
  return 0;
}

// ---- host-side dispatch -----------------------------------------------------------------------
// One instance family, tuned on the B200 for the HBM-bound regime:
// 16-token tiles, 2 stages, 3 warps -> 48 KiB per CTA at D=128, 4 CTAs (12 warps) per SM.  More
// resident warps beat deeper per-warp rings; 12 warps x 8 KiB keeps ~100 KiB of gathers in flight.
constexpr int kNT = 16, kStages = 2, kNW = 3;

static int tile_heads(int group) { return group <= 8 ? 8 : 16; }
static int decode_align() { return kNW * kNT; }
static int decode_ctas_per_sm(int D) {
  const int smem = MmaCfg<128, kNT, kStages, kNW>::SMEM_BYTES * D / 128 + 1024;
  int n = (227 * 1024) / smem;
  const int by_regs = 65536 / (kNW * 32 * 168);
  n = n < by_regs ? n : by_regs;
  return n < 1 ? 1 : n;
}

template <typename C, auto KERN>
static int launch_decode_kernel(const DecodeParamsNew& p, cudaStream_t st, const char* timer_name, const char* kernel_name) {
  static std::atomic<bool> attr_done{false};
  if (!attr_done.load(std::memory_order_relaxed)) {
    B200_CUDA_OK(cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    attr_done.store(true, std::memory_order_relaxed);
  }
  const dim3 grid = p.pieces ? dim3(p.pieces, p.Hkv * p.head_tiles) : dim3(p.num_splits, p.Hkv * p.head_tiles, p.bs);
  {
    ScopedKernelTimer timer(timer_name, st);
    B200_CUDA_OK(launch_kernel(KERN, grid, dim3(C::THREADS), C::SMEM_BYTES, st, 1, pdl_family(p.bs, kPdlAttn), p));
  }
  B200_CHECK_LAUNCH(kernel_name);
  return 0;
}

template <typename T, int D, bool HI>
static int launch_decode(const DecodeParamsNew& p, cudaStream_t st) {
  using C = MmaCfg<D, kNT, kStages, kNW>;
  using P = DecodeParams;
  using N = DecodeParamsNew;
#define DECODE_LAUNCH(...) \
  launch_decode_kernel<C, attn_decode_mma_kernel<__VA_ARGS__>>(p, st, "attn_decode_split", "attn_decode_mma_kernel")
  if (p.tickets) return DECODE_LAUNCH(P, T, D, kNT, kStages, kNW, HI, true);
  if (p.row_list || p.gate) return DECODE_LAUNCH(P, T, D, kNT, kStages, kNW, HI, false, true);
  if (p.pieces)
    return p.new_k ? DECODE_LAUNCH(N, T, D, kNT, kStages, kNW, HI, false, false, true)
                   : DECODE_LAUNCH(P, T, D, kNT, kStages, kNW, HI, false, false, true);
  return p.new_k ? DECODE_LAUNCH(N, T, D, kNT, kStages, kNW, HI, false) : DECODE_LAUNCH(P, T, D, kNT, kStages, kNW, HI, false);
#undef DECODE_LAUNCH
}

template <typename T>
static int dispatch_decode(const DecodeParamsNew& p, int D, int G, cudaStream_t st) {
  if (D == 128) return G > 8 ? launch_decode<T, 128, true>(p, st) : launch_decode<T, 128, false>(p, st);
  if (D == 64) return G > 8 ? launch_decode<T, 64, true>(p, st) : launch_decode<T, 64, false>(p, st);
  set_error("b200_attn_decode: unsupported head_dim %d (supported: 64, 128)", D);
  return 1;
}

// ---- FP8 KV pool: 32-token tiles (same 8 KiB per stage as the bf16 kernel's 16-token tiles) ------
constexpr int kNT8 = 32;
static int decode_align_fp8kv() { return kNW * kNT8; }

static int fp8kv_stages() {
  static int v = [] {
    const char* e = std::getenv("B200_FP8KV_STAGES");
    const int s = (e && *e) ? std::atoi(e) : 2;
    return s == 3 ? 3 : 2;
  }();
  return v;
}

template <typename T, int D, bool HI, int ST>
static int launch_decode_fp8kv_st(const DecodeParamsNew& p, cudaStream_t st) {
  using C = Fp8KvCfg<D, kNT8, ST, kNW>;
  using P = DecodeParams;
  using N = DecodeParamsNew;
#define DECODE_LAUNCH(...) \
  launch_decode_kernel<C, attn_decode_fp8kv_kernel<__VA_ARGS__>>(p, st, "attn_decode_fp8kv", "attn_decode_fp8kv_kernel")
  if (p.tickets) return DECODE_LAUNCH(P, T, D, kNT8, ST, kNW, HI, true);
  if (p.pieces)
    return p.new_k ? DECODE_LAUNCH(N, T, D, kNT8, ST, kNW, HI, false, false, true)
                   : DECODE_LAUNCH(P, T, D, kNT8, ST, kNW, HI, false, false, true);
  return p.new_k ? DECODE_LAUNCH(N, T, D, kNT8, ST, kNW, HI, false) : DECODE_LAUNCH(P, T, D, kNT8, ST, kNW, HI, false);
#undef DECODE_LAUNCH
}

template <typename T, int D, bool HI>
static int launch_decode_fp8kv(const DecodeParamsNew& p, cudaStream_t st) {
  return fp8kv_stages() == 3 ? launch_decode_fp8kv_st<T, D, HI, 3>(p, st)
                             : launch_decode_fp8kv_st<T, D, HI, 2>(p, st);
}

// e5m2 pool (`--kv-cache-dtype fp8_e5m2`): the same kernel with the byte -> f16 conversion swapped
// (one PRMT instead of a cvt); 2-stage ring, no in-kernel tail.
template <typename T, int D, bool HI>
static int launch_decode_e5m2kv(const DecodeParamsNew& p, cudaStream_t st) {
  using C = Fp8KvCfg<D, kNT8, 2, kNW>;
  using P = DecodeParams;
  using N = DecodeParamsNew;
#define DECODE_LAUNCH(...) \
  launch_decode_kernel<C, attn_decode_fp8kv_kernel<__VA_ARGS__>>(p, st, "attn_decode_fp8kv", "attn_decode_fp8kv_kernel<e5m2>")
  if (p.pieces)
    return p.new_k ? DECODE_LAUNCH(N, T, D, kNT8, 2, kNW, HI, false, true, true)
                   : DECODE_LAUNCH(P, T, D, kNT8, 2, kNW, HI, false, true, true);
  return p.new_k ? DECODE_LAUNCH(N, T, D, kNT8, 2, kNW, HI, false, true) : DECODE_LAUNCH(P, T, D, kNT8, 2, kNW, HI, false, true);
#undef DECODE_LAUNCH
}

template <typename T>
static int dispatch_decode_fp8kv(const DecodeParamsNew& p, int D, int G, bool e5m2, cudaStream_t st) {
  if (e5m2 && D == 128)
    return G > 8 ? launch_decode_e5m2kv<T, 128, true>(p, st) : launch_decode_e5m2kv<T, 128, false>(p, st);
  if (e5m2 && D == 64)
    return G > 8 ? launch_decode_e5m2kv<T, 64, true>(p, st) : launch_decode_e5m2kv<T, 64, false>(p, st);
  if (D == 128)
    return G > 8 ? launch_decode_fp8kv<T, 128, true>(p, st) : launch_decode_fp8kv<T, 128, false>(p, st);
  if (D == 64)
    return G > 8 ? launch_decode_fp8kv<T, 64, true>(p, st) : launch_decode_fp8kv<T, 64, false>(p, st);
  set_error("b200_attn_decode_fp8kv: unsupported head_dim %d (supported: 64, 128)", D);
  return 1;
}

// Host side of the fused tail (see decode_fused_tail).
struct DecodeTail {
  void* tickets;
  size_t ticket_bytes;
  void* q_out;
  int64_t q_out_stride;
  float* q_scales;
};

// New rows of b200_attn_decode_layer / _fp8kv_layer.
struct DecodeNewRows {
  const void* k;
  const void* v;
  int64_t k_stride, v_stride;
  const int64_t* loc;
  int has_scale;
  int own_slots;
};

// The split kernel stores the rows itself where 16-byte pieces of a head fit them, it is not the instance with the
// in-kernel tail, and either no entry reads another's new slot or the entries are few (store_new_rows); else they are
// written by a launch of their own before it, which takes pools without gaps between the rows only.
static int apply_new_rows(DecodeParamsNew& p, const DecodeNewRows* rows, int D, int dtype, bool fp8, int e5m2, float k_scale,
                          float v_scale, void* stream, const char* who) {
  if (!rows) return 0;
  B200_REQUIRE(rows->k && rows->v && rows->loc, "%s: null pointer", who);
  const bool dense = p.kv_row_stride == static_cast<int64_t>(p.Hkv) * D;
  if (!p.tickets && aligned16(rows->k) && aligned16(rows->v) && rows->k_stride % 8 == 0 && rows->v_stride % 8 == 0 &&
      (rows->own_slots || p.bs <= kNewRowsAll || !dense)) {
    p.new_k = rows->k;
    p.new_v = rows->v;
    p.new_k_stride = rows->k_stride;
    p.new_v_stride = rows->v_stride;
    p.loc = rows->loc;
    p.k_scale_w = k_scale;
    p.v_scale_w = v_scale;
    p.scale_new = rows->has_scale;
    p.new_all = !rows->own_slots;
    return 0;
  }
  B200_REQUIRE(dense, "%s: pool rows of %lld elements for %d heads", who,
               static_cast<long long>(p.kv_row_stride), p.Hkv);
  void *kc = const_cast<void*>(p.k_cache), *vc = const_cast<void*>(p.v_cache);
  const int row = p.Hkv * D;
  if (fp8)
    return b200_kv_write_fp8(rows->k, rows->v, rows->k_stride, rows->v_stride, kc, vc, rows->loc, p.bs, row, k_scale, v_scale,
                             rows->has_scale, dtype | e5m2, stream);
  return b200_kv_write(rows->k, rows->v, rows->k_stride * 2, rows->v_stride * 2, kc, vc, rows->loc, p.bs, row * 2, row * 2, stream);
}

static int apply_tail(DecodeParams& p, const DecodeTail* tail, int D, const char* who) {
  p.tickets = nullptr;
  p.q_out = nullptr;
  p.q_out_stride = 0;
  p.q_scales = nullptr;
  if (!tail) return 0;
  const size_t need = static_cast<size_t>(p.bs) * (1 + p.Hkv * p.head_tiles) * sizeof(unsigned);
  B200_REQUIRE(!tail->tickets || tail->ticket_bytes >= need,
               "%s: ticket buffer too small (%zu < %zu bytes)", who, tail->ticket_bytes, need);
  B200_REQUIRE((tail->q_out == nullptr) == (tail->q_scales == nullptr),
               "%s: q_out and q_scales go together", who);
  B200_REQUIRE(tail->q_out || p.num_splits > 1, "%s: nothing to fuse (one split, no q_out)", who);
  B200_REQUIRE(!tail->q_out || (tail->q_out_stride % 8 == 0 &&
                                (reinterpret_cast<uintptr_t>(tail->q_out) & 7u) == 0),
               "%s: q_out must be 8-byte aligned with q_out_stride %% 8 == 0", who);
  B200_REQUIRE(p.o_stride % 8 == 0 && aligned16(p.o) && (p.Hq * D) % 8 == 0,
               "%s: o must be 16-byte aligned with o_stride %% 8 == 0", who);
  p.tickets = static_cast<unsigned*>(tail->tickets);  // null: the tail is one merge(+quant) launch
  p.q_out = static_cast<uint8_t*>(tail->q_out);
  p.q_out_stride = tail->q_out_stride;
  p.q_scales = tail->q_scales;
  return 0;
}

}  // namespace b200

extern "C" {

size_t b200_attn_decode_workspace_bytes(int bs, int Hq, int Dv, int num_splits) {
  if (num_splits <= 1) return 0;
  const size_t rows = static_cast<size_t>(bs) * Hq * num_splits;
  return rows * Dv * sizeof(float) + rows * sizeof(float);
}

static int decode_num_splits(int bs, int Hkv, int group, int D, int64_t avg_len, int64_t max_len, int num_sms) {
  using namespace b200;
  if (bs <= 0 || Hkv <= 0 || group <= 0) return 1;
  if (num_sms <= 0) num_sms = 148;
  const int G = tile_heads(group);
  const int head_tiles = ceil_div(group, G);
  const int64_t base = static_cast<int64_t>(bs) * Hkv * head_tiles;
  const int ctas_per_sm = decode_ctas_per_sm(D);
  const int64_t slots = static_cast<int64_t>(num_sms) * ctas_per_sm;
  const int64_t by_slots = slots / base;
  // Up to one wave of CTAs: the chain of 48-token tiles in a CTA, which is slower with more CTAs on its SM, against the
  // merge launch and what each split adds to it.  Microseconds fitted to 1592 batches (1 to 64 requests of 64 to 131072
  // tokens, equal and unequal ones, bf16 and FP8 rows, 2 to 8 kv heads), each timed at up to 20 split counts; the
  // choice is 2.0 % slower than the best of them on average.  The longest request is what the others are waited for.
  // (us, 1 request: 128 tokens 5.8 whole, 7.4 in 2; 512 tokens 10.6 whole, 7.6 in 8, 7.1 in 12; 1500 tokens 9.3 in 8,
  // 7.7 in 16, 9.1 in 64; 131072 tokens 116 in 32, 92 in 64; 16 requests: 384 tokens 9.6 whole, 10.5 in 2; 700 tokens
  // 13.9 whole, 12.9 in 4, 15.4 in 8.)  From 900 tokens on, with fewer than 4 splits in the wave, the bandwidth
  // decides.
  const int64_t longest = avg_len > max_len ? avg_len : max_len;
  const int64_t align = decode_align();
  constexpr double kTile[4] = {0.46, 0.62, 0.90, 0.82};        // 1 to 4 CTAs an SM
  int64_t fit = 1;
  double fit_us = 0.0;
  for (int64_t s = 1; s <= 64 && (s == 1 || (s <= by_slots && s * align <= longest)); ++s) {
    const int64_t tiles = ((longest + s - 1) / s + align - 1) / align;
    const int64_t on_sm = (base * s + num_sms - 1) / num_sms;
    const double us = 0.04 * s * (1.0 + 0.001 * base) + (s > 1 ? 2.0 + 0.009 * base : 0.0) +
                      tiles * (on_sm <= 4 ? kTile[on_sm - 1] : 0.25 * kTile[3] * on_sm);
    if (s == 1 || us < fit_us) {
      fit = s;
      fit_us = us;
    }
  }
  if (by_slots >= 4 || longest < 900) return static_cast<int>(fit);
  // Equal-length CTAs that all fit the resident slots at once finish together, while any overflow runs as a thin
  // second wave: the estimate's count, where one wave fills three quarters of the slots.  Per-rank shapes of
  // Llama-3.1-8B at TP 2 / 4 / 8, batch 64 x 4k: 2 / 4 / 9 splits = 512 / 512 / 576 CTAs on 592 slots (90.8 / 50.7 /
  // 29.9 us) against 93.9 / 56.4 / 35.3 us for the oversubscription rule below; 1 split (512 CTAs, no merge) 170.4 us
  // against 174.4 + merge.
  // Not for few splits of unequal requests, where the longest ones would run alone at the end (us, one wave or 1.5 ->
  // 2.1 times the slots: 40 x up to 3000 tokens 61.3 -> 57.9, 64 x up to 4096 FP8 77.0 -> 69.3, 27 x up to 6000 FP8
  // 50.4 -> 48.2); short ones lose more to the merge than the even end gives.
  const bool unequal = max_len * 8 > avg_len * 9;
  if (by_slots >= 1 && static_cast<double>(base * by_slots) >= 0.75 * static_cast<double>(slots) &&
      !(unequal && avg_len >= 1536))
    return static_cast<int>(fit);
  // HBM-bound: what matters is that enough CTAs stay resident until the end, not whole waves: late CTAs run faster
  // because they share the bandwidth with fewer neighbours.  The smallest split count that oversubscribes the resident
  // slots, where the requests are long enough for it (40 equal requests, 1 / 3 splits: 1024 tokens 37.2 / 40.0 us, 3000
  // tokens 94.4 / 88.6).
  const double over = unequal ? 2.1 : 1.5;
  const int64_t least = unequal ? 192 : 640;
  for (int64_t s = 1; s < 64 && avg_len >= least * s; ++s)
    if (static_cast<double>(base * s) >= over * static_cast<double>(slots)) return static_cast<int>(s);
  return static_cast<int>(fit);
}

int b200_attn_decode_num_splits(int bs, int Hkv, int group, int D, int64_t avg_len, int num_sms) {
  return decode_num_splits(bs, Hkv, group, D, avg_len, avg_len, num_sms);
}

int b200_attn_decode_num_splits_ragged(int bs, int Hkv, int group, int D, int64_t avg_len, int64_t max_len,
                                       int num_sms) {
  return decode_num_splits(bs, Hkv, group, D, avg_len, max_len, num_sms);
}

static size_t pieces_plan_offset(int Hq, int Dv, int pieces) {
  return (b200_attn_decode_workspace_bytes(1, Hq, Dv, pieces < 2 ? 2 : pieces) + 15) / 16 * 16;
}

size_t b200_attn_decode_pieces_workspace_bytes(int bs, int Hq, int Dv, int pieces) {
  if (pieces <= 0 || bs <= 0) return 0;
  return pieces_plan_offset(Hq, Dv, pieces) + static_cast<size_t>(bs) * sizeof(int2);
}

static int use_pieces(b200::DecodeParams& p, int pieces, int Dv, void* workspace, size_t bytes, const char* who) {
  using namespace b200;
  B200_REQUIRE(pieces >= p.bs && p.bs <= kPieceMaxBatch && pieces <= 65535, "%s: %d pieces for %d requests", who, pieces, p.bs);
  B200_REQUIRE(workspace && aligned16(workspace) && bytes >= b200_attn_decode_pieces_workspace_bytes(p.bs, p.Hq, Dv, pieces),
               "%s: workspace too small for %d pieces", who, pieces);
  p.pieces = pieces;
  p.part_o = static_cast<float*>(workspace);
  p.part_lse = p.part_o + static_cast<size_t>(pieces) * p.Hq * Dv;
  p.plan = reinterpret_cast<int2*>(static_cast<char*>(workspace) + pieces_plan_offset(p.Hq, Dv, pieces));
  return 0;
}

static int merge_pieces(const b200::DecodeParams& p, int D, int dtype, void* stream) {
  using namespace b200;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid(ceil_div(p.Hq, kMergeWarps), p.bs);
  ScopedKernelTimer timer("attn_merge", st);
#define MERGE_PIECES(T, D_)                                                                                                \
  B200_CUDA_OK(launch_kernel(attn_merge_pieces_kernel<T, D_>, grid, dim3(kMergeWarps * 32), 0, st, 1,                      \
                             pdl_family(p.bs, kPdlMerge), p.part_o, p.part_lse, static_cast<T*>(p.o), p.o_stride, p.plan, p.Hq))
  if (dtype == B200_BF16) {
    if (D == 128) MERGE_PIECES(__nv_bfloat16, 128);
    else MERGE_PIECES(__nv_bfloat16, 64);
  } else {
    if (D == 128) MERGE_PIECES(__half, 128);
    else MERGE_PIECES(__half, 64);
  }
#undef MERGE_PIECES
  B200_CHECK_LAUNCH("attn_merge_pieces_kernel");
  return 0;
}

/* How many pieces a decode batch of unequal requests is cut into, or 0 where a split count for all serves it. */
int b200_attn_decode_pieces_for(int bs, int Hkv, int group, int D, int64_t total_len, int64_t max_len, int num_sms) {
  using namespace b200;
  if (bs < 2 || bs > kPieceMaxBatch || Hkv <= 0 || group <= 0 || D <= 0) return 0;
  if (num_sms <= 0) num_sms = 148;
  // One wave at four CTAs an SM (two and three waves were slower in every batch timed).  Not where the longest request is
  // within an eighth of the average; from 1.5 pieces a request on (64 x up to 1500 tokens, 1.2 pieces a request: 50.1 us in
  // splits, 53.0 in pieces); up to 16 (4 x up to 4000, 18 a request: 10.3 / 11.4, where splits of every request fill the
  // wave as well); and from 250 tokens a piece on (8 x up to 2000, 135 a piece: 11.6 / 12.1; 16 x up to 2000, 270: 17.5 /
  // 15.2), below which the plan and the merge cost what the even end gives.
  const int64_t tiles = static_cast<int64_t>(Hkv) * ceil_div(group, tile_heads(group));
  const int64_t slots = static_cast<int64_t>(num_sms) * 4, pieces = slots / tiles;
  const bool unequal = max_len * 8 * bs > total_len * 9;
  if (!unequal || 2 * pieces < 3 * bs || pieces > 16 * bs || total_len < 250 * pieces || pieces > 65535) return 0;
  // And, where the splits are all resident at once, only if the longest of them is 220 tokens of head size 128 longer than a
  // piece: short splits end early and leave their SM to the long ones, so less unevenness than that is evened out anyway.
  // Of 450 random batches that pass the lines above (profiles/decode_pieces_batches.json) this one keeps 396, 1.150 x (0.969
  // at worst, 5 below 0.98); the 54 others were 0.98 x (D 64, 34 x up to 3663 FP8 11.9 us in splits, 13.3 in pieces).
  const int64_t splits = decode_num_splits(bs, Hkv, group, D, total_len / bs > 1 ? total_len / bs : 1, max_len, num_sms);
  if (bs * tiles * splits <= slots && (max_len / splits - total_len / pieces) * D < 220 * 128) return 0;
  return static_cast<int>(pieces);
}

int b200_attn_decode_pieces(int bs, int Hkv, int group, int64_t total_len, int64_t max_len, int num_sms) {
  return b200_attn_decode_pieces_for(bs, Hkv, group, 128, total_len, max_len, num_sms);
}

static int attn_merge_impl(const float* part_o, const float* part_lse, void* o, int64_t o_stride,
                           const int64_t* seq_lens, int bs, int Hq, int Dv, int num_splits,
                           int split_align, const int32_t* row_list, const void* gate,
                           int64_t gate_stride, int dtype, void* stream) {
  using namespace b200;
  if (bs == 0) return 0;
  const int align = split_align;
  B200_REQUIRE(num_splits >= 1 && split_align >= 1, "b200_attn_merge: bad split config %d/%d",
               num_splits, split_align);
  B200_REQUIRE(part_o && part_lse && o && seq_lens, "b200_attn_merge: null pointer");
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16, "b200_attn_merge: dtype %d", dtype);
  // By columns while their CTAs, one per head, are at most two an SM: more CTAs cost what the round trips save (us, with
  // the split kernel, a warp per head / by columns: 32 heads in 9 splits 8.1 / 7.4, 128 in 14 11.0 / 10.7, 256 in 10
  // 13.4 / 12.9, 320 in 16 16.4 / 17.1, 512 in 10 18.8 / 19.4, 1024 in 12 44.2 / 44.8).
  const bool bycols = num_splits > 8 && static_cast<int64_t>(bs) * Hq <= 2 * device_sm_count();
  dim3 grid(bycols ? Hq : ceil_div(Hq, kMergeWarps), bs);
  const int threads = kMergeWarps * 32;
  const bool wide = Dv % 4 == 0 && aligned16(part_o);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ScopedKernelTimer timer("attn_merge", st);
#define LAUNCH_MERGE(T, V, C)                                                                                         \
  B200_CUDA_OK(launch_kernel(attn_merge_kernel<T, V, C>, grid, dim3(threads), 0, st, 1, pdl_family(bs, kPdlMerge),    \
                             part_o, part_lse, static_cast<T*>(o), o_stride, seq_lens, Hq, Dv, num_splits, align,     \
                             row_list, static_cast<const T*>(gate), gate_stride))
  if (dtype == B200_BF16) {
    if (bycols) LAUNCH_MERGE(__nv_bfloat16, 1, true);
    else if (wide) LAUNCH_MERGE(__nv_bfloat16, 4, false);
    else LAUNCH_MERGE(__nv_bfloat16, 1, false);
  } else {
    if (bycols) LAUNCH_MERGE(__half, 1, true);
    else if (wide) LAUNCH_MERGE(__half, 4, false);
    else LAUNCH_MERGE(__half, 1, false);
  }
#undef LAUNCH_MERGE
  B200_CHECK_LAUNCH("attn_merge_kernel");
  return 0;
}

static int attn_decode_impl(const void* q, int64_t q_stride, const void* k_cache,
                            const void* v_cache, int64_t kv_row_stride, void* o, int64_t o_stride,
                            const int32_t* req_to_token, int64_t req_to_token_stride,
                            const int64_t* req_pool_indices, const int64_t* seq_lens, int bs,
                            int Hq, int Hkv, int D, int Dv, float scale, float logit_cap, int dtype,
                            void* workspace, size_t workspace_bytes, int num_splits, void* stream,
                            const b200::DecodeTail* tail, const int32_t* row_list = nullptr,
                            const void* gate = nullptr, int64_t gate_stride = 0,
                            const b200::DecodeNewRows* rows = nullptr, int pieces = 0) {
  using namespace b200;
  if (bs == 0) return 0;
  B200_REQUIRE(q && k_cache && v_cache && o && req_to_token && req_pool_indices && seq_lens,
               "b200_attn_decode: null pointer");
  B200_REQUIRE(!tail || (!row_list && !gate), "b200_attn_decode: the fused tail takes no row list or gate");
  B200_REQUIRE(bs > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0,
               "b200_attn_decode: bad head config bs=%d Hq=%d Hkv=%d", bs, Hq, Hkv);
  B200_REQUIRE(D == Dv, "b200_attn_decode: qk_head_dim (%d) != v_head_dim (%d) is not supported",
               D, Dv);
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16,
               "b200_attn_decode: dtype %d not supported (bf16/f16 KV only)", dtype);
  B200_REQUIRE(num_splits >= 1 && num_splits <= 1024, "b200_attn_decode: bad num_splits %d",
               num_splits);
  B200_REQUIRE(aligned16(q) && aligned16(k_cache) && aligned16(v_cache) && q_stride % 8 == 0 &&
                   kv_row_stride % 8 == 0,
               "b200_attn_decode: q/k_cache/v_cache must be 16-byte aligned with strides %% 8 == 0");
  B200_REQUIRE(bs <= 65535 && Hkv * 8 <= 65535, "b200_attn_decode: grid too large");
  const size_t need = b200_attn_decode_workspace_bytes(bs, Hq, Dv, num_splits);
  B200_REQUIRE(num_splits == 1 || pieces > 0 || (workspace && workspace_bytes >= need),
               "b200_attn_decode: workspace too small (%zu < %zu)", workspace_bytes, need);

  DecodeParamsNew p = {};
  p.q = q;
  p.q_stride = q_stride;
  p.k_cache = k_cache;
  p.v_cache = v_cache;
  p.kv_row_stride = kv_row_stride;
  p.o = o;
  p.o_stride = o_stride;
  p.req_to_token = req_to_token;
  p.rtt_stride = req_to_token_stride;
  p.req_pool_indices = req_pool_indices;
  p.seq_lens = seq_lens;
  p.bs = bs;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.group = Hq / Hkv;
  const int G = tile_heads(p.group);
  p.head_tiles = ceil_div(p.group, G);
  p.num_splits = num_splits;
  p.logit_cap = logit_cap;
  p.v_scale = 1.f;
  p.row_list = row_list;
  p.gate = gate;
  p.gate_stride = gate_stride;
  p.qk_scale = logit_cap > 0.f ? scale : scale * kLog2e;
  { static const char* e = std::getenv("B200_PDL_LATE"); p.pdl_late = e ? std::atoi(e) : 1; }
  p.part_o = static_cast<float*>(workspace);
  p.part_lse = p.part_o ? p.part_o + static_cast<size_t>(bs) * Hq * num_splits * Dv : nullptr;

  if (int rc = apply_tail(p, tail, D, "b200_attn_decode_fused")) return rc;
  if (int rc = apply_new_rows(p, rows, D, dtype, false, 0, 1.f, 1.f, stream, "b200_attn_decode_layer")) return rc;
  if (pieces > 0) {
    B200_REQUIRE(!tail && !row_list && !gate, "b200_attn_decode_layer: pieces take no fused tail");
    if (int rc = use_pieces(p, pieces, Dv, workspace, workspace_bytes, "b200_attn_decode_layer")) return rc;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = dtype == B200_BF16 ? dispatch_decode<__nv_bfloat16>(p, D, G, st)
                              : dispatch_decode<__half>(p, D, G, st);
  if (rc) return rc;
  if (pieces > 0) return merge_pieces(p, D, dtype, stream);
  if (tail && !tail->tickets && tail->q_out)
    return dtype == B200_BF16 ? launch_merge_quant<__nv_bfloat16>(p, Dv, decode_align(), st)
                              : launch_merge_quant<__half>(p, Dv, decode_align(), st);
  if (num_splits > 1 && !(tail && tail->tickets))
    return attn_merge_impl(p.part_o, p.part_lse, o, o_stride, seq_lens, bs, Hq, Dv, num_splits,
                           decode_align(), row_list, gate, gate_stride, dtype, stream);
  return 0;
}

int b200_attn_decode(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache,
                     int64_t kv_row_stride, void* o, int64_t o_stride,
                     const int32_t* req_to_token, int64_t req_to_token_stride,
                     const int64_t* req_pool_indices, const int64_t* seq_lens, int bs, int Hq,
                     int Hkv, int D, int Dv, float scale, float logit_cap, int dtype,
                     void* workspace, size_t workspace_bytes, int num_splits, void* stream) {
  return attn_decode_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride, req_to_token,
                          req_to_token_stride, req_pool_indices, seq_lens, bs, Hq, Hkv, D, Dv, scale,
                          logit_cap, dtype, workspace, workspace_bytes, num_splits, stream, nullptr);
}

int b200_attn_decode_rows(const void* q, int64_t q_stride, const void* k_cache, const void* v_cache,
                          int64_t kv_row_stride, void* o, int64_t o_stride,
                          const int32_t* req_to_token, int64_t req_to_token_stride,
                          const int64_t* req_pool_indices, const int64_t* seq_lens,
                          const int32_t* row_list, const void* gate, int64_t gate_stride, int bs, int Hq,
                          int Hkv, int D, int Dv, float scale, float logit_cap, int dtype,
                          void* workspace, size_t workspace_bytes, int num_splits, void* stream) {
  return attn_decode_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride, req_to_token,
                          req_to_token_stride, req_pool_indices, seq_lens, bs, Hq, Hkv, D, Dv, scale,
                          logit_cap, dtype, workspace, workspace_bytes, num_splits, stream, nullptr, row_list,
                          gate, gate_stride);
}

int b200_attn_decode_fused(const void* q, int64_t q_stride, const void* k_cache,
                           const void* v_cache, int64_t kv_row_stride, void* o, int64_t o_stride,
                           const int32_t* req_to_token, int64_t req_to_token_stride,
                           const int64_t* req_pool_indices, const int64_t* seq_lens, int bs, int Hq,
                           int Hkv, int D, int Dv, float scale, float logit_cap, int dtype,
                           void* workspace, size_t workspace_bytes, int num_splits, void* tickets,
                           size_t ticket_bytes, void* q_out, int64_t q_out_stride, float* q_scales,
                           void* stream) {
  b200::DecodeTail tail = {tickets, ticket_bytes, q_out, q_out_stride, q_scales};
  return attn_decode_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride, req_to_token,
                          req_to_token_stride, req_pool_indices, seq_lens, bs, Hq, Hkv, D, Dv, scale,
                          logit_cap, dtype, workspace, workspace_bytes, num_splits, stream, &tail);
}

size_t b200_attn_decode_fused_ticket_bytes(int bs, int Hq, int Hkv) {
  using namespace b200;
  if (bs <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv) return 0;
  const int group = Hq / Hkv;
  return static_cast<size_t>(bs) * (1 + Hkv * ceil_div(group, tile_heads(group))) * sizeof(unsigned);
}

int b200_attn_decode_fp8kv_split_align(void) { return b200::decode_align_fp8kv(); }

static int attn_decode_fp8kv_impl(const void* q, int64_t q_stride, const void* k_cache,
                                  const void* v_cache, int64_t kv_row_stride, void* o,
                                  int64_t o_stride, const int32_t* req_to_token,
                                  int64_t req_to_token_stride, const int64_t* req_pool_indices,
                                  const int64_t* seq_lens, int bs, int Hq, int Hkv, int D, int Dv,
                                  float scale, float logit_cap, float k_scale, float v_scale,
                                  int dtype, void* workspace, size_t workspace_bytes, int num_splits,
                                  void* stream, const b200::DecodeTail* tail,
                                  const b200::DecodeNewRows* rows = nullptr, int pieces = 0) {
  using namespace b200;
  if (bs == 0) return 0;
  const bool e5m2 = (dtype & B200_KV_FP8_E5M2) != 0;
  dtype &= ~B200_KV_FP8_E5M2;
  DecodeTail tail_e5m2;
  if (e5m2 && tail && tail->tickets) {  // no in-kernel tail instance for e5m2: one merge launch
    tail_e5m2 = *tail;
    tail_e5m2.tickets = nullptr;
    tail_e5m2.ticket_bytes = 0;
    tail = &tail_e5m2;
  }
  B200_REQUIRE(q && k_cache && v_cache && o && req_to_token && req_pool_indices && seq_lens,
               "b200_attn_decode_fp8kv: null pointer");
  B200_REQUIRE(bs > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0,
               "b200_attn_decode_fp8kv: bad head config bs=%d Hq=%d Hkv=%d", bs, Hq, Hkv);
  B200_REQUIRE(D == Dv, "b200_attn_decode_fp8kv: qk_head_dim (%d) != v_head_dim (%d)", D, Dv);
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16,
               "b200_attn_decode_fp8kv: q/o dtype %d not supported (bf16/f16)", dtype);
  B200_REQUIRE(num_splits >= 1 && num_splits <= 1024, "b200_attn_decode_fp8kv: bad num_splits %d",
               num_splits);
  B200_REQUIRE(aligned16(q) && aligned16(k_cache) && aligned16(v_cache) && q_stride % 8 == 0 &&
                   kv_row_stride % 16 == 0,
               "b200_attn_decode_fp8kv: q/k_cache/v_cache must be 16-byte aligned, q_stride %% 8 == 0 "
               "and kv_row_stride %% 16 == 0");
  B200_REQUIRE(bs <= 65535 && Hkv * 8 <= 65535, "b200_attn_decode_fp8kv: grid too large");
  B200_REQUIRE(k_scale > 0.f && v_scale > 0.f, "b200_attn_decode_fp8kv: scales must be positive");
  const size_t need = b200_attn_decode_workspace_bytes(bs, Hq, Dv, num_splits);
  B200_REQUIRE(num_splits == 1 || pieces > 0 || (workspace && workspace_bytes >= need),
               "b200_attn_decode_fp8kv: workspace too small (%zu < %zu)", workspace_bytes, need);
  DecodeParamsNew p = {};
  p.q = q;
  p.q_stride = q_stride;
  p.k_cache = k_cache;
  p.v_cache = v_cache;
  p.kv_row_stride = kv_row_stride;
  p.o = o;
  p.o_stride = o_stride;
  p.req_to_token = req_to_token;
  p.rtt_stride = req_to_token_stride;
  p.req_pool_indices = req_pool_indices;
  p.seq_lens = seq_lens;
  p.bs = bs;
  p.Hq = Hq;
  p.Hkv = Hkv;
  p.group = Hq / Hkv;
  const int G = tile_heads(p.group);
  p.head_tiles = ceil_div(p.group, G);
  p.num_splits = num_splits;
  p.logit_cap = logit_cap;
  p.v_scale = v_scale;
  p.qk_scale = (logit_cap > 0.f ? scale : scale * kLog2e) * k_scale;
  { static const char* e = std::getenv("B200_PDL_LATE"); p.pdl_late = e ? std::atoi(e) : 1; }
  p.part_o = static_cast<float*>(workspace);
  p.part_lse = p.part_o ? p.part_o + static_cast<size_t>(bs) * Hq * num_splits * Dv : nullptr;
  if (int rc = apply_tail(p, tail, D, "b200_attn_decode_fp8kv_fused")) return rc;
  if (int rc = apply_new_rows(p, rows, D, dtype, true, e5m2 ? B200_KV_FP8_E5M2 : 0, k_scale, v_scale, stream,
                              "b200_attn_decode_fp8kv_layer"))
    return rc;
  if (pieces > 0) {
    B200_REQUIRE(!tail, "b200_attn_decode_fp8kv_layer: pieces take no fused tail");
    if (int rc = use_pieces(p, pieces, Dv, workspace, workspace_bytes, "b200_attn_decode_fp8kv_layer")) return rc;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rc = dtype == B200_BF16 ? dispatch_decode_fp8kv<__nv_bfloat16>(p, D, G, e5m2, st)
                                    : dispatch_decode_fp8kv<__half>(p, D, G, e5m2, st);
  if (rc) return rc;
  if (pieces > 0) return merge_pieces(p, D, dtype, stream);
  if (tail && !tail->tickets && tail->q_out)
    return dtype == B200_BF16 ? launch_merge_quant<__nv_bfloat16>(p, Dv, decode_align_fp8kv(), st)
                              : launch_merge_quant<__half>(p, Dv, decode_align_fp8kv(), st);
  if (num_splits > 1 && !(tail && tail->tickets))
    return b200_attn_merge(p.part_o, p.part_lse, o, o_stride, seq_lens, bs, Hq, Dv, num_splits,
                           decode_align_fp8kv(), dtype, stream);
  return 0;
}

int b200_attn_decode_fp8kv(const void* q, int64_t q_stride, const void* k_cache,
                           const void* v_cache, int64_t kv_row_stride, void* o, int64_t o_stride,
                           const int32_t* req_to_token, int64_t req_to_token_stride,
                           const int64_t* req_pool_indices, const int64_t* seq_lens, int bs,
                           int Hq, int Hkv, int D, int Dv, float scale, float logit_cap,
                           float k_scale, float v_scale, int dtype, void* workspace,
                           size_t workspace_bytes, int num_splits, void* stream) {
  return attn_decode_fp8kv_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride,
                                req_to_token, req_to_token_stride, req_pool_indices, seq_lens, bs, Hq,
                                Hkv, D, Dv, scale, logit_cap, k_scale, v_scale, dtype, workspace,
                                workspace_bytes, num_splits, stream, nullptr);
}

int b200_attn_decode_fp8kv_fused(const void* q, int64_t q_stride, const void* k_cache,
                                 const void* v_cache, int64_t kv_row_stride, void* o,
                                 int64_t o_stride, const int32_t* req_to_token,
                                 int64_t req_to_token_stride, const int64_t* req_pool_indices,
                                 const int64_t* seq_lens, int bs, int Hq, int Hkv, int D, int Dv,
                                 float scale, float logit_cap, float k_scale, float v_scale,
                                 int dtype, void* workspace, size_t workspace_bytes, int num_splits,
                                 void* tickets, size_t ticket_bytes, void* q_out,
                                 int64_t q_out_stride, float* q_scales, void* stream) {
  b200::DecodeTail tail = {tickets, ticket_bytes, q_out, q_out_stride, q_scales};
  return attn_decode_fp8kv_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride,
                                req_to_token, req_to_token_stride, req_pool_indices, seq_lens, bs, Hq,
                                Hkv, D, Dv, scale, logit_cap, k_scale, v_scale, dtype, workspace,
                                workspace_bytes, num_splits, stream, &tail);
}

int b200_attn_decode_layer(const void* k, int64_t k_stride, const void* v, int64_t v_stride, const int64_t* loc,
                           const void* q, int64_t q_stride, void* k_cache, void* v_cache, int64_t kv_row_stride, void* o,
                           int64_t o_stride, const int32_t* req_to_token, int64_t req_to_token_stride,
                           const int64_t* req_pool_indices, const int64_t* seq_lens, int bs, int Hq, int Hkv, int D, int Dv,
                           float scale, float logit_cap, int dtype, void* workspace, size_t workspace_bytes, int num_splits,
                           int pieces, void* tickets, size_t ticket_bytes, void* q_out, int64_t q_out_stride, float* q_scales,
                           void* stream) {
  const b200::DecodeTail tail = {tickets, ticket_bytes, q_out, q_out_stride, q_scales};
  const b200::DecodeNewRows rows = {k, v, k_stride, v_stride, loc, 0, dtype & B200_OWN_SLOTS};
  dtype &= ~B200_OWN_SLOTS;
  return attn_decode_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride, req_to_token, req_to_token_stride,
                          req_pool_indices, seq_lens, bs, Hq, Hkv, D, Dv, scale, logit_cap, dtype, workspace, workspace_bytes,
                          num_splits, stream, tickets || q_out ? &tail : nullptr, nullptr, nullptr, 0, k ? &rows : nullptr, pieces);
}

int b200_attn_decode_fp8kv_layer(const void* k, int64_t k_stride, const void* v, int64_t v_stride, const int64_t* loc,
                                 int has_scale, const void* q, int64_t q_stride, void* k_cache, void* v_cache,
                                 int64_t kv_row_stride, void* o, int64_t o_stride, const int32_t* req_to_token,
                                 int64_t req_to_token_stride, const int64_t* req_pool_indices, const int64_t* seq_lens, int bs,
                                 int Hq, int Hkv, int D, int Dv, float scale, float logit_cap, float k_scale, float v_scale,
                                 int dtype, void* workspace, size_t workspace_bytes, int num_splits, int pieces,
                                 void* tickets, size_t ticket_bytes, void* q_out, int64_t q_out_stride, float* q_scales,
                                 void* stream) {
  const b200::DecodeTail tail = {tickets, ticket_bytes, q_out, q_out_stride, q_scales};
  const b200::DecodeNewRows rows = {k, v, k_stride, v_stride, loc, has_scale, dtype & B200_OWN_SLOTS};
  dtype &= ~B200_OWN_SLOTS;
  return attn_decode_fp8kv_impl(q, q_stride, k_cache, v_cache, kv_row_stride, o, o_stride, req_to_token, req_to_token_stride,
                                req_pool_indices, seq_lens, bs, Hq, Hkv, D, Dv, scale, logit_cap, k_scale, v_scale, dtype,
                                workspace, workspace_bytes, num_splits, stream, tickets || q_out ? &tail : nullptr, k ? &rows : nullptr, pieces);
}

int b200_attn_decode_split_align(int D, int group) {
  (void)D;
  (void)group;
  return b200::decode_align();
}

int b200_attn_merge(const float* part_o, const float* part_lse, void* o, int64_t o_stride,
                    const int64_t* seq_lens, int bs, int Hq, int Dv, int num_splits,
                    int split_align, int dtype, void* stream) {
  return attn_merge_impl(part_o, part_lse, o, o_stride, seq_lens, bs, Hq, Dv, num_splits, split_align, nullptr,
                         nullptr, 0, dtype, stream);
}

}  // extern "C"
