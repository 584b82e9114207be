// Int4 weights at prefill sizes in two passes: the stream copy of the weight (w4a16_gemv2.cu) is expanded once to a
// 16-bit [N, K] weight in a caller's workspace, then the CTA-pair GEMM (gemm_pair.cuh) multiplies with it.
//
// Why: the fused kernel (w4a16.cu) expands a weight tile again for every 256 tokens and moves ~120 KiB through shared
// memory per 512 clocks of tensor work, which caps it at about 60 % of the tensor rate.  The expansion costs
// (0.5 + 2) bytes per weight of HBM time once; the products are the same 16-bit (w - z) * s.  Measured (f16, Qwen2.5-32B
// at TP 2, 2048 tokens, qkv / o / gate_up / down, us): fused 73.2 / 60.9 / 466 / 275, here 65.0 / 51.7 / 425 / 255.
#include "gemm_pair.cuh"

namespace b200 {

static WaitCounter wait_counter_registered(tc::wait_counter());

template <typename T>
struct ExpandMagic;
template <>
struct ExpandMagic<__half> {
  using T2 = __half2;
  static constexpr uint32_t kBits = 0x64006400u;   // (1024, 1024): the nibble lands in the low mantissa bits
};
template <>
struct ExpandMagic<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  static constexpr uint32_t kBits = 0x43004300u;   // (128, 128)
};

// A warp per 16-column x 64-k tile of the stream; lane 4 g + t holds columns g and g + 8 at k = 32 s + 8 t ..+7, so its
// four words become four 16-byte pieces of two rows.  Same rounding as awq_dequant_kernel: (magic + w) - (magic + z),
// exact, then one multiplication in 16 bits.  HBM-bound.
template <typename T>
__global__ void __launch_bounds__(256)
w4a16_stream_expand_kernel(const uint4* __restrict__ qw, const T* __restrict__ zeros, const T* __restrict__ scales,
                           T* __restrict__ out, int N, int K, int group) {
  using T2 = typename ExpandMagic<T>::T2;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int KB = K >> 6;
  const int64_t tile = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const int nt = static_cast<int>(tile / KB), kb = static_cast<int>(tile - static_cast<int64_t>(nt) * KB);
  if (nt * 16 >= N) return;
  const uint4 v = __ldg(qw + tile * 32 + lane);
  const uint32_t w[2][2] = {{v.x, v.y}, {v.z, v.w}};            // [32-k step][column g, g + 8]
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const int k = kb * 64 + s * 32 + t * 8;
    const int64_t grow = static_cast<int64_t>(k / group) * N;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int n = nt * 16 + g + c * 8;
      T2 z2, s2;
      z2.x = z2.y = zeros[grow + n];
      s2.x = s2.y = scales[grow + n];
      uint32_t r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t b = ((w[s][c] >> (4 * i)) & 0x000f000fu) | ExpandMagic<T>::kBits;
        const T2 d = __hmul2(__hsub2(*reinterpret_cast<const T2*>(&b), z2), s2);
        r[i] = *reinterpret_cast<const uint32_t*>(&d);
      }
      *reinterpret_cast<uint4*>(out + static_cast<int64_t>(n) * K + k) = make_uint4(r[0], r[1], r[2], r[3]);
    }
  }
}

}  // namespace b200

extern "C" {

size_t b200_w4a16_gemm_stream_workspace_bytes(int N, int K) { return static_cast<size_t>(N) * K * 2; }

int b200_w4a16_gemm_stream(const void* x, int64_t ldx, const void* qweight_stream, const void* zeros, const void* scales,
                           const void* bias, void* out, int64_t ldc, int M, int N, int K, int group_size,
                           void* workspace, size_t workspace_bytes, int dtype, void* stream) {
  using namespace b200;
  if (M == 0 || N == 0) return 0;
  B200_REQUIRE(x && qweight_stream && zeros && scales && out && workspace, "b200_w4a16_gemm_stream: null pointer");
  B200_REQUIRE(M > 0 && N > 0 && N % 16 == 0 && K > 0 && K % 64 == 0 && group_size > 0 && group_size % 8 == 0 &&
                   K % group_size == 0,
               "b200_w4a16_gemm_stream: bad shape M=%d N=%d K=%d group=%d", M, N, K, group_size);
  B200_REQUIRE(aligned16(x) && ldx % 8 == 0 && aligned16(qweight_stream) && aligned16(workspace) &&
                   workspace_bytes >= b200_w4a16_gemm_stream_workspace_bytes(N, K),
               "b200_w4a16_gemm_stream: x, weight and workspace must be 16-byte aligned, ldx %% 8 == 0, workspace of "
               "%zu bytes (got %zu)",
               b200_w4a16_gemm_stream_workspace_bytes(N, K), workspace_bytes);
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16, "b200_w4a16_gemm_stream: dtype %d", dtype);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t tiles = static_cast<int64_t>(N / 16) * (K / 64);
  const unsigned blocks = static_cast<unsigned>((tiles + 7) / 8);
  {
    ScopedKernelTimer timer("w4a16_expand", st);
    if (dtype == B200_F16)
      w4a16_stream_expand_kernel<__half><<<blocks, 256, 0, st>>>(
          static_cast<const uint4*>(qweight_stream), static_cast<const __half*>(zeros), static_cast<const __half*>(scales),
          static_cast<__half*>(workspace), N, K, group_size);
    else
      w4a16_stream_expand_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(
          static_cast<const uint4*>(qweight_stream), static_cast<const __nv_bfloat16*>(zeros),
          static_cast<const __nv_bfloat16*>(scales), static_cast<__nv_bfloat16*>(workspace), N, K, group_size);
    B200_CHECK_LAUNCH("w4a16_stream_expand_kernel");
  }
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
  // the GEMM requests its first weight tiles before its dependency wait: not here, where the weight is new
  const int rc = dtype == B200_F16
                     ? launch_gemm_pair<kKindF16, __half>(x, ldx, workspace, K, ep, st, "w4a16_gemm", false)
                     : launch_gemm_pair<kKindBf16, __nv_bfloat16>(x, ldx, workspace, K, ep, st, "w4a16_gemm", false);
  if (rc == 0) {
    char pair[128];
    std::snprintf(pair, sizeof(pair), "%s", b200_last_variant());
    note_variant("w4a16_expand + %s expanded", pair);
  }
  return rc;
}

}  // extern "C"
