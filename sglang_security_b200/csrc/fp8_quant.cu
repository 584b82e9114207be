// FP8 (e4m3) activation quantisers of the W8A8 linear path.
//   per-token      : scale[m] = absmax(x[m,:]) / 448 ; q = sat(x * (1/scale))       (reference
//                    sgl-kernel/csrc/gemm/per_token_quant_fp8.cu:9-76)
//   per-token-group: scale[m,g] = max(absmax, eps) / 448 ; q = sat(x / scale), group = 128
//                    (sgl-kernel/csrc/gemm/per_token_group_quant_8bit.cu:19-98,
//                     native_per_token_group_quant_fp8, python/sglang/test/test_block_fp8.py:23-48)
//   static         : q = sat(x * (1/scale)) with one given scale             (fp8_kernel.py:336-376)
// The arithmetic (reciprocal-multiply vs. true division, clamp order, RN conversion) follows the
// reference kernels so that the quantised bytes agree.
#include <cuda_fp8.h>

#include "common.cuh"

namespace b200 {

constexpr float kFp8Max = 448.0f;

__device__ __forceinline__ uint8_t to_e4m3(float v) {
  return static_cast<uint8_t>(__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3));
}

// four finite values within +-448 -> four e4m3 bytes
__device__ __forceinline__ uint32_t e4m3x4(float2 a, float2 b) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(a, __NV_SATFINITE, __NV_E4M3);
  return lo | static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(b, __NV_SATFINITE, __NV_E4M3)) << 16;
}

template <typename T>
__device__ __forceinline__ void load8(const T* p, float (&f)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 v = unpack2<T>(w[e]);
    f[2 * e] = v.x;
    f[2 * e + 1] = v.y;
  }
}

__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  v = lane < nw ? red[lane] : 0.f;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

// One CTA per token row.  K % 8 == 0.
// MODE 0: dynamic, q = sat(x * (1/scale))           (per_token_quant_fp8.cu)
// MODE 1: static scale, q = sat(x * (1/scale))      (_static_quant_fp8)
// MODE 2: dynamic, scale = max(absmax, eps)/448, q = sat(x / scale): the group_size == K case of
//         per_token_group_quant_fp8 used for load-time per-channel weight quantisation.
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
fp8_quant_per_token_kernel(const T* __restrict__ x, int64_t ldx, uint8_t* __restrict__ q,
                           int64_t ldq, float* __restrict__ scales,
                           const float* __restrict__ static_scale, int K, float eps) {
  constexpr bool STATIC = MODE == 1;
  __shared__ float red[32];
  griddep_wait();
  // MODE 2 quantises WEIGHTS at load time: its consumers (the GEMMs) prefetch their weight operand
  // before their own dependency wait, so this kernel must not release them early
  if (MODE != 2) griddep_launch_dependents();
  const int m = blockIdx.x;
  const T* row = x + m * ldx;
  uint8_t* out = q + m * ldq;
  const int nvec = K / 8;
  float scale;
  if (STATIC) {
    scale = __ldg(static_scale);
  } else {
    float amax = 0.f;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      float f[8];
      load8(row + i * 8, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(f[e]));
    }
    amax = block_max(amax, red);
    if (MODE == 2) amax = fmaxf(amax, eps);
    scale = amax / kFp8Max;
    if (threadIdx.x == 0) scales[m] = scale;
  }
  // an all-zero row keeps scale 0 and quantises to zeros (the reference would emit NaN bytes)
  const float inv = scale > 0.f ? 1.0f / scale : 0.f;
  for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
    float f[8];
    load8(row + i * 8, f);
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float a = MODE == 2 ? f[e] / scale : f[e] * inv;
      const float b = MODE == 2 ? f[4 + e] / scale : f[4 + e] * inv;
      lo |= static_cast<uint32_t>(to_e4m3(fmaxf(fminf(a, kFp8Max), -kFp8Max))) << (8 * e);
      hi |= static_cast<uint32_t>(to_e4m3(fmaxf(fminf(b, kFp8Max), -kFp8Max))) << (8 * e);
    }
    *reinterpret_cast<uint2*>(out + i * 8) = make_uint2(lo, hi);
  }
}

// Dynamic per-token form of up to VPT * blockDim.x * 8 columns: the row stays in registers between its maximum and
// its quantisation, so it is read once and all loads are in flight together.  Same values as MODE 0 above.
// Bound by HBM at many tokens (2048 x 14336 bf16, us: reading the row twice 22.3, now 16.2; 13.6 of HBM time), by one
// round trip and one barrier at few (1 x 4096: 2.0, now 1.3).
template <typename T, int VPT>
__global__ void __launch_bounds__(512)
fp8_quant_row_kernel(const T* __restrict__ x, int64_t ldx, uint8_t* __restrict__ q, int64_t ldq,
                     float* __restrict__ scales, int nvec) {
  __shared__ float red[32];
  griddep_wait();
  griddep_launch_dependents();
  const int m = blockIdx.x;
  const T* row = x + m * ldx;
  uint4 raw[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = v * blockDim.x + threadIdx.x;
    raw[v] = i < nvec ? *reinterpret_cast<const uint4*>(row + i * 8) : make_uint4(0, 0, 0, 0);
  }
  float amax = 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const uint32_t w[4] = {raw[v].x, raw[v].y, raw[v].z, raw[v].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = unpack2<T>(w[e]);
      amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
  }
  amax = block_max(amax, red);
  const float scale = amax / kFp8Max;
  if (threadIdx.x == 0) scales[m] = scale;
  const float inv = scale > 0.f ? 1.0f / scale : 0.f;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int i = v * blockDim.x + threadIdx.x;
    if (i >= nvec) continue;
    const uint32_t w[4] = {raw[v].x, raw[v].y, raw[v].z, raw[v].w};
    float2 f[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f[e] = unpack2<T>(w[e]);
      f[e].x = fmaxf(fminf(f[e].x * inv, kFp8Max), -kFp8Max);
      f[e].y = fmaxf(fminf(f[e].y * inv, kFp8Max), -kFp8Max);
    }
    *reinterpret_cast<uint2*>(q + m * ldq + i * 8) = make_uint2(e4m3x4(f[0], f[1]), e4m3x4(f[2], f[3]));
  }
}

// 16 lanes per 128-element group (8 elements per lane), 2 groups per warp.
// scales[m * s_row + g * s_col]: row-major (s_row = K/128, s_col = 1) or column-major / TMA
// aligned (s_row = 1, s_col = padded M).
// x / scale is a true division.  With r = 1 / scale rounded to nearest, q = x r and one remainder step
// q + (x - q scale) r give the rounded quotient (Markstein 1990) up to halfway cases; that the e4m3 byte is the
// division's for every significand of x and of the maximum is checked exhaustively by the tests.  That holds while
// the remainder is exact: a quotient that is not rounded to zero is at least 2^-11, so its product with the scale is
// a multiple of 2^-57 scale, which fp32 holds from a scale of 2^-92 on.  Smaller scales (a caller's eps; below 3e-39
// their reciprocal is infinite) and infinite ones are divided by.  The compiler's division and one load in flight per lane bound the kernel.
constexpr float kReciprocalMin = 0x1p-90f;
// The general rules (NaN, infinities and tiny scales among them): a group's maximum from `amax` up, over LANES lanes that
// hold N pairs each, and its elements divided by the scale and clamped.
template <int LANES, int N>
__device__ __forceinline__ float group_max(const float2 (&f)[N], float amax) {
#pragma unroll
  for (int e = 0; e < N; ++e) amax = fmaxf(amax, fmaxf(fabsf(f[e].x), fabsf(f[e].y)));
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  return amax;
}
template <int N>
__device__ __forceinline__ void group_scale(float2 (&f)[N], float s) {
  if (s >= kReciprocalMin && s < INFINITY) {
    const float r = 1.0f / s;
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const float qx = f[e].x * r, qy = f[e].y * r;
      f[e].x = copysignf(fmaf(fmaf(-qx, s, f[e].x), r, qx), qx);   // -0 stays -0
      f[e].y = copysignf(fmaf(fmaf(-qy, s, f[e].y), r, qy), qy);
    }
  } else {
#pragma unroll
    for (int e = 0; e < N; ++e) f[e] = make_float2(f[e].x / s, f[e].y / s);
  }
#pragma unroll
  for (int e = 0; e < N; ++e) {
    f[e].x = fminf(fmaxf(f[e].x, -kFp8Max), kFp8Max);
    f[e].y = fminf(fmaxf(f[e].y, -kFp8Max), kFp8Max);
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
fp8_quant_group128_kernel(const T* __restrict__ x, int64_t ldx, uint8_t* __restrict__ q,
                          int64_t ldq, float* __restrict__ scales, int64_t s_row, int64_t s_col,
                          int M, int groups_per_row, float eps) {
  griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 15;
  const unsigned total = static_cast<unsigned>(M) * groups_per_row;   // below 2^31: the launcher cuts the rows
  const unsigned gid = blockIdx.x * 16u + (threadIdx.x >> 4);
  const unsigned row = gid / static_cast<unsigned>(groups_per_row);
  const int64_t m = row;
  const int g = static_cast<int>(gid - row * groups_per_row);
  const uint4 raw = gid < total ? *reinterpret_cast<const uint4*>(x + m * ldx + g * 128 + lane * 8) : make_uint4(0, 0, 0, 0);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  float2 f[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) f[e] = unpack2<T>(w[e]);
  const float s = group_max<16>(f, eps) / kFp8Max;
  if (gid >= total) return;
  if (lane == 0) scales[m * s_row + g * s_col] = s;
  group_scale(f, s);
  *reinterpret_cast<uint2*>(q + m * ldq + g * 128 + lane * 8) = make_uint2(e4m3x4(f[0], f[1]), e4m3x4(f[2], f[3]));
}

// The same for 8192 groups or more: 8 lanes x 16 elements a group, 32 rows a block, GPT groups a lane along K.  Half as many
// lanes share the group's maximum, division and reciprocal; products and remainder steps are packed; groups without a NaN
// (nearly all) need no clamp, since the conversion saturates; the general rules are a function of their own, so that six
// or eight blocks fit an SM.  Issue slots and, with fewer blocks, bytes in flight bounded the kernel above: 3001 x 14336
// bf16 32.7 -> 22.0 us (19.7 of HBM time), 2048 x 4096 9.5 -> 7.0, 512 x 4096 3.2 -> 2.4.  Two groups a lane from 65536 on
// (3001 x 14336 one / two / four 23.9 / 22.0 / 29.6; 1024 x 4096 4.4 / 5.0).  Of 154 sizes of 100 to 3001 rows 1.2 x on
// average; slower at 19000 to 22400 groups alone, where its 600 to 700 blocks are an uneven few an SM (300 x 8192 2.85 / 3.13).
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;\n" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// One group by the general rules, 8 lanes of a full warp.
template <typename T>
__device__ __noinline__ void quant_group_general(const T* src, uint8_t* out, float* scale, bool store, bool lane0, float eps) {
  float2 f[8];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint4 raw = *reinterpret_cast<const uint4*>(src + h * 64);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) f[h * 4 + e] = unpack2<T>(w[e]);
  }
  const float s = group_max<8>(f, eps) / kFp8Max;
  if (!store) return;
  if (lane0) *scale = s;
  group_scale(f, s);
  *reinterpret_cast<uint2*>(out) = make_uint2(e4m3x4(f[0], f[1]), e4m3x4(f[2], f[3]));
  *reinterpret_cast<uint2*>(out + 64) = make_uint2(e4m3x4(f[4], f[5]), e4m3x4(f[6], f[7]));
}

template <typename T, int GPT>
__global__ void __launch_bounds__(256, GPT == 1 ? 8 : 6)
fp8_quant_group128_rows_kernel(const T* __restrict__ x, int64_t ldx, uint8_t* __restrict__ q, int64_t ldq,
                               float* __restrict__ scales, int64_t s_row, int64_t s_col, int M, int groups_per_row, float eps) {
  griddep_wait();
  griddep_launch_dependents();
  const int lane = threadIdx.x & 7;
  const unsigned along = static_cast<unsigned>(ceil_div(groups_per_row, GPT));
  const int m = static_cast<int>(blockIdx.x / along) * 32 + (threadIdx.x >> 3);
  const int g0 = static_cast<int>(blockIdx.x % along) * GPT;
  const bool row_ok = m < M;
  const T* src = x + static_cast<int64_t>(row_ok ? m : M - 1) * ldx + g0 * 128 + lane * 8;
  uint8_t* out = q + m * ldq + g0 * 128 + lane * 8;
  float* sc = scales + m * s_row + g0 * s_col;
  uint4 raw[GPT][2];
#pragma unroll
  for (int i = 0; i < GPT; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      raw[i][h] = g0 + i < groups_per_row ? *reinterpret_cast<const uint4*>(src + i * 128 + h * 64) : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int i = 0; i < GPT; ++i) {
    if (g0 + i >= groups_per_row) break;
    float2 f[8];
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t w[4] = {raw[i][h].x, raw[i][h].y, raw[i][h].z, raw[i][h].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f[h * 4 + e] = unpack2<T>(w[e]);
        a0 = max_nan(a0, fabsf(f[h * 4 + e].x));
        a1 = max_nan(a1, fabsf(f[h * 4 + e].y));
      }
    }
    a0 = max_nan(a0, a1);
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) a0 = max_nan(a0, __shfl_xor_sync(0xffffffffu, a0, off));
    const float s = fmaxf(a0, eps) / kFp8Max;
    if (__any_sync(0xffffffffu, !(a0 == a0 && s >= kReciprocalMin && s < INFINITY))) {
      quant_group_general(src + i * 128, out + i * 128, sc + i * s_col, row_ok, lane == 0, eps);
      continue;
    }
    const float r = 1.0f / s;
    const float2 r2 = make_float2(r, r), ns = make_float2(-s, -s);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float2 qe = fmul2(f[e], r2);
      const float2 y = ffma2(ffma2(qe, ns, f[e]), r2, qe);
      f[e] = make_float2(copysignf(y.x, qe.x), copysignf(y.y, qe.y));
    }
    if (!row_ok) continue;
    if (lane == 0) sc[i * s_col] = s;
    *reinterpret_cast<uint2*>(out + i * 128) = make_uint2(e4m3x4(f[0], f[1]), e4m3x4(f[2], f[3]));
    *reinterpret_cast<uint2*>(out + i * 128 + 64) = make_uint2(e4m3x4(f[4], f[5]), e4m3x4(f[6], f[7]));
  }
}

}  // namespace b200

extern "C" {

int b200_fp8_quant_per_token(const void* x, int64_t ldx, void* q, int64_t ldq, float* scales,
                             const float* static_scale, int M, int K, int use_division, float eps,
                             int dtype, void* stream) {
  using namespace b200;
  if (M == 0) return 0;
  B200_REQUIRE(x && q && (scales || static_scale), "b200_fp8_quant_per_token: null pointer");
  B200_REQUIRE(K > 0 && K % 8 == 0 && ldx % 8 == 0 && ldq % 8 == 0 && aligned16(x) &&
                   (reinterpret_cast<uintptr_t>(q) & 7u) == 0,
               "b200_fp8_quant_per_token: K/ld must be multiples of 8 and pointers aligned (K=%d)",
               K);
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16, "b200_fp8_quant_per_token: dtype %d",
               dtype);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ScopedKernelTimer timer("fp8_quant", st);
  // a row that fits 512 threads x 8 pieces stays in registers: as few threads as keep 4 pieces each busy at many
  // rows (2048 x 4096: 128 threads), more and shorter ones where there are fewer rows than SMs
  const int nvec = K / 8;
  if (!static_scale && !use_division && nvec <= 512 * 8) {
    const int want = M >= 4 * device_sm_count() ? 4 : 1;
    int threads = (ceil_div(nvec, want) + 31) / 32 * 32;
    threads = threads < 64 ? 64 : threads > 512 ? 512 : threads;
    if (want == 4 && threads > 256 && ceil_div(nvec, 256) <= 8) threads = 256;
    const int vpt = ceil_div(nvec, threads);
#define LAUNCH_ROW(T, V)                                                                                             \
  B200_CUDA_OK(launch_kernel(fp8_quant_row_kernel<T, V>, dim3(M), dim3(threads), 0, st, 1, pdl_family(M, kPdlQuant), \
                             static_cast<const T*>(x), ldx, static_cast<uint8_t*>(q), ldq, scales, nvec))
#define LAUNCH_ROW_T(T)                  \
  if (vpt == 1) LAUNCH_ROW(T, 1);        \
  else if (vpt == 2) LAUNCH_ROW(T, 2);   \
  else if (vpt <= 4) LAUNCH_ROW(T, 4);   \
  else LAUNCH_ROW(T, 8)
    if (dtype == B200_BF16) {
      LAUNCH_ROW_T(__nv_bfloat16);
    } else {
      LAUNCH_ROW_T(__half);
    }
#undef LAUNCH_ROW_T
#undef LAUNCH_ROW
    B200_CHECK_LAUNCH("fp8_quant_row_kernel");
    return 0;
  }
  const int threads = K >= 2048 ? 256 : 128;
#define LAUNCH(T, MODE)                                                                          \
  B200_CUDA_OK(launch_kernel(fp8_quant_per_token_kernel<T, MODE>, dim3(M), dim3(threads), 0, st, 1, pdl_family(M, kPdlQuant), \
                             static_cast<const T*>(x), ldx, static_cast<uint8_t*>(q), ldq, scales,  \
                             static_scale, K, eps))
  if (dtype == B200_BF16) {
    if (static_scale) LAUNCH(__nv_bfloat16, 1);
    else if (use_division) LAUNCH(__nv_bfloat16, 2);
    else LAUNCH(__nv_bfloat16, 0);
  } else {
    if (static_scale) LAUNCH(__half, 1);
    else if (use_division) LAUNCH(__half, 2);
    else LAUNCH(__half, 0);
  }
#undef LAUNCH
  B200_CHECK_LAUNCH("fp8_quant_per_token_kernel");
  return 0;
}

int b200_fp8_quant_group128(const void* x, int64_t ldx, void* q, int64_t ldq, float* scales,
                            int64_t scale_row_stride, int64_t scale_col_stride, int M, int K,
                            float eps, int dtype, void* stream) {
  using namespace b200;
  if (M == 0) return 0;
  B200_REQUIRE(x && q && scales, "b200_fp8_quant_group128: null pointer");
  B200_REQUIRE(K > 0 && K % 128 == 0 && ldx % 8 == 0 && ldq % 8 == 0 && aligned16(x) &&
                   (reinterpret_cast<uintptr_t>(q) & 7u) == 0,
               "b200_fp8_quant_group128: K must be a multiple of 128 (K=%d)", K);
  B200_REQUIRE(dtype == B200_BF16 || dtype == B200_F16, "b200_fp8_quant_group128: dtype %d", dtype);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ScopedKernelTimer timer("fp8_quant", st);
  const int gpr = K / 128;
  const int step = 0x7fffff00 / gpr;               // rows per launch: group numbers stay below 2^31
  for (int m0 = 0; m0 < M; m0 += step) {
    const int rows = M - m0 < step ? M - m0 : step;
    const unsigned total = static_cast<unsigned>(rows) * gpr;
    const int64_t xo = static_cast<int64_t>(m0) * ldx, qo = static_cast<int64_t>(m0) * ldq;
    float* sc = scales + static_cast<int64_t>(m0) * scale_row_stride;
#define LAUNCH_GROUP(KERNEL, BLOCKS)                                                                                  \
  B200_CUDA_OK(launch_kernel(KERNEL, dim3(BLOCKS), dim3(256), 0, st, 1, pdl_family(M, kPdlQuant),                     \
                             static_cast<const T*>(x) + xo, ldx, static_cast<uint8_t*>(q) + qo, ldq, sc, scale_row_stride, scale_col_stride, rows, gpr, eps))
    auto launch = [&](auto type) -> int {
      using T = decltype(type);
      if (total >= 65536) LAUNCH_GROUP((fp8_quant_group128_rows_kernel<T, 2>), ceil_div(gpr, 2) * ceil_div(rows, 32));
      else if (total >= 8192) LAUNCH_GROUP((fp8_quant_group128_rows_kernel<T, 1>), gpr * ceil_div(rows, 32));
      else LAUNCH_GROUP(fp8_quant_group128_kernel<T>, (total + 15) / 16);
      return 0;
    };
    if (int rc = dtype == B200_BF16 ? launch(__nv_bfloat16()) : launch(__half())) return rc;
#undef LAUNCH_GROUP
  }
  B200_CHECK_LAUNCH("fp8_quant_group128_kernel");
  return 0;
}

}  // extern "C"
