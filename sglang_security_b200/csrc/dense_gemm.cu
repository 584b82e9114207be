// Dense 16-bit GEMM on tcgen05 for the layers the quantisation configs leave unquantised
// (UnquantizedLinearMethod.apply = F.linear, python/sglang/srt/layers/linear.py:170-176; the
// lm_head of the decode step, vocab_parallel_embedding.py / logits_processor.py:_get_logits):
//   out[M, N] = x[M, K] . w[N, K]^T (+ bias[N]),  bf16 / f16 operands, fp32 accumulation in TMEM.
// Same CTA-pair TMA + tcgen05 kernel as the FP8 path (gemm_pair.cuh) with kind::f16; K-major
// operands, so the reference's [N, K] weight is used as stored.
#include "fp8_gemm_smallm.cuh"
#include "gemm_pair.cuh"

namespace b200 {

static WaitCounter wait_counter_registered(tc::wait_counter());

// Decode sizes: the swap-AB kernel with K split over a cluster (fp8_gemm_smallm.cuh), two CTAs an SM, whose weight ring is
// filled before the CTA is set up; a CTA pair of gemm_pair_kernel has to meet first, and ends with an exchange of 4-byte
// loads.  Its sums meet token by token, so it pays with a long K: of 24 shapes timed on both, one call after the other
// (profiles/dense_small_m_forms.json), from K 2048 up to 24 tokens (us, pair / this: 4096 x 4096 1 token 10.2 / 7.1, 24 10.2 /
// 9.4; 5120 x 2560 8.8 / 6.9 and equal); with a short K up to 4 tokens and 8192 channels (4096 x 1024 1 token equal, 24 4.8 /
// 5.6; 9728 x 896 1 token 5.5 / 5.7, 24 5.8 / 7.7; 151936 x 896 24 tokens 43.1 / 54.9).  Where K is not split the two are even
// call after call, or pairs up to 4 % ahead from 16 tokens on, but not between other linears, whose kernel it shares (four
// linears of Llama-3.1-8B, 16 tokens, all here 79.1, gate_up in pairs 85.9; a whole step with the head here / in pairs, 20
// tokens, 399 / 402).  Four linears, bf16: Llama-3.1-8B 1 token 83.9 / 73.7, 16 86.1 / 79.2, 24 86.6 / 81.9; at TP 4 34.5 /
// 28.9, 36.1 / 30.4, 36.6 / 33.2; Qwen2.5-32B at TP 2 90.0 / 81.8, 91.5 / 85.2, 92.0 / 88.5.
static bool dense_small(int M, int N, int K) {
  return ceil_div(K, 64) >= 32 ? M <= 24 : M <= 4 && ceil_div(N, 128) <= 64;
}
template <int KIND, typename OutT>
static int launch_dense_small(const void* x, int64_t ldx, const void* w, int64_t ldw, const GemmEpilogueParams& ep,
                              cudaStream_t st) {
  SmallMParams p = {};
  p.out = ep.out;
  p.ldc = ep.ldc;
  p.bias = ep.bias;
  p.M = ep.M;
  p.N = ep.N;
  p.K = ep.K;
  const bool big = static_cast<int64_t>(ep.N) * ep.K * 2 >= (48ll << 20);
  if (ep.M > 16) return launch_smallm_ks<32, false, OutT, false, 1, true, KIND>(x, ldx, w, ldw, p, st, "dense_gemm");
  if (ep.M > 4)
    return big ? launch_smallm_ks<16, false, OutT, false, 2, true, KIND>(x, ldx, w, ldw, p, st, "dense_gemm")
               : launch_smallm_ks<16, false, OutT, false, 1, true, KIND>(x, ldx, w, ldw, p, st, "dense_gemm");
  return big ? launch_smallm_ks<16, false, OutT, false, 2, false, KIND>(x, ldx, w, ldw, p, st, "dense_gemm")
             : launch_smallm_ks<16, false, OutT, false, 1, false, KIND>(x, ldx, w, ldw, p, st, "dense_gemm");
}

static int gemm_16bit(const void* x, int64_t ldx, const void* w, int64_t ldw, const void* bias, void* out,
                      int64_t ldc, int M, int N, int K, bool act, float act_pos, float act_neg, int dtype,
                      void* stream) {
  if (M == 0 || N == 0) return 0;
  B200_REQUIRE(x && w && out, "b200_gemm_16bit: null pointer");
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "b200_gemm_16bit: bad shape %dx%dx%d", M, N, K);
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16, "b200_gemm_16bit: dtype %d", dtype);
  B200_REQUIRE(aligned16(x) && aligned16(w) && ldx % 8 == 0 && ldw % 8 == 0,
               "b200_gemm_16bit: x / w must be 16-byte aligned with row strides %% 8 == 0 (TMA)");
  B200_REQUIRE(ldc % 8 != 0 || aligned16(out), "b200_gemm_16bit: out must be 16-byte aligned when its rows are");
  GemmEpilogueParams ep;
  ep.out = out;
  ep.ldc = ldc;
  ep.sa = nullptr;
  ep.sb = nullptr;
  ep.sa_stride = 0;
  ep.sb_stride = 0;
  ep.bias = bias;
  ep.M = M;
  ep.N = N;
  ep.K = K;
  ep.act_pos = act_pos;
  ep.act_neg = act_neg;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (act)
    return dtype == B200_BF16 ? launch_gemm_pair<kKindBf16, __nv_bfloat16, true>(x, ldx, w, ldw, ep, st, "dense_gemm")
                              : launch_gemm_pair<kKindF16, __half, true>(x, ldx, w, ldw, ep, st, "dense_gemm");
  if (dense_small(M, N, K))
    return dtype == B200_BF16 ? launch_dense_small<kKindBf16, __nv_bfloat16>(x, ldx, w, ldw, ep, st)
                              : launch_dense_small<kKindF16, __half>(x, ldx, w, ldw, ep, st);
  return dtype == B200_BF16 ? launch_gemm_pair<kKindBf16, __nv_bfloat16>(x, ldx, w, ldw, ep, st, "dense_gemm")
                            : launch_gemm_pair<kKindF16, __half>(x, ldx, w, ldw, ep, st, "dense_gemm");
}

}  // namespace b200

extern "C" int b200_gemm_16bit(const void* x, int64_t ldx, const void* w, int64_t ldw,
                               const void* bias, void* out, int64_t ldc, int M, int N, int K,
                               int dtype, void* stream) {
  return b200::gemm_16bit(x, ldx, w, ldw, bias, out, ldc, M, N, K, false, 0.f, 0.f, dtype, stream);
}

extern "C" int b200_gemm_16bit_xielu(const void* x, int64_t ldx, const void* w, int64_t ldw,
                                     const void* bias, void* out, int64_t ldc, int M, int N, int K,
                                     float act_pos, float act_neg, int dtype, void* stream) {
  return b200::gemm_16bit(x, ldx, w, ldw, bias, out, ldc, M, N, K, true, act_pos, act_neg, dtype, stream);
}
