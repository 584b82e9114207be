// What the tcgen05 GEMMs of the library share: operand kinds, epilogue parameters, cluster helpers.
// All of them compute out[M, N] = epilogue( x[M, K] . w[N, K]^T ) with both operands K-major ("TN"): token rows
// and output-channel rows, exactly how the reference stores activations and (transposed-view) weights
// (fp8.py:349,391; fp8_utils.py:636-648).
#pragma once
#include <type_traits>

#include "activation.cuh"
#include "tc_common.cuh"

namespace b200 {

enum GemmKind { kKindFp8 = 0, kKindBf16 = 1, kKindF16 = 2 };

struct GemmEpilogueParams {
  void* out;            // [M, N] OutT, row stride ldc
  int64_t ldc;
  const float* sa;      // per-token scale (stride sa_stride: 1 = per token, 0 = per tensor) or null
  const float* sb;      // per-channel scale (stride sb_stride) or null
  int sa_stride, sb_stride;
  const void* bias;     // [N] OutT or null
  int M, N, K;
  // ACT instances: out = xielu(result; act_pos, act_neg) before the store (activation.cuh)
  float act_pos = 0.f, act_neg = 0.f;
};

template <int KIND>
struct GemmKindTraits;
template <>
struct GemmKindTraits<kKindFp8> {
  static constexpr int ELT = 1;
  static constexpr uint32_t FMT = 0;  // E4M3
};
template <>
struct GemmKindTraits<kKindBf16> {
  static constexpr int ELT = 2;
  static constexpr uint32_t FMT = 1;  // BF16
};
template <>
struct GemmKindTraits<kKindF16> {
  static constexpr int ELT = 2;
  static constexpr uint32_t FMT = 0;  // F16
};

__device__ __forceinline__ void named_bar_sync_gemm(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

template <typename OutT>
__device__ __forceinline__ uint32_t pack_out2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack_out2<__nv_bfloat16>(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
template <>
__device__ __forceinline__ uint32_t pack_out2<__half>(float a, float b) {
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

}  // namespace b200
