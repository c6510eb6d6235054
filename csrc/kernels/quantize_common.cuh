// The 1 x 128 power-of-two quantiser of one (row, K block), shared by the kernels that quantise activations
// (quantize.cu) and those that quantise on the way somewhere (moe.cu). Half a warp takes a block, eight elements per lane.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>
#include <type_traits>

namespace {

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

// Eight elements as they lie in memory. vec: 2 the rows are 16-byte aligned, 1 they are aligned to four elements
// (8 bytes of a 16-bit type), 0 element-wise, as a row's ragged tail always is.
template <typename T>
struct Raw8 {
  static constexpr int kWords = (int)sizeof(T) * 8 / 16;
  uint4 w[kWords];
  __device__ __forceinline__ void load(const T* p, int n_valid, int vec) {
    if (vec == 2 && n_valid >= 8) {
#pragma unroll
      for (int i = 0; i < kWords; ++i) w[i] = ((const uint4*)p)[i];
    } else if (vec == 1 && n_valid >= 8) {
#pragma unroll
      for (int i = 0; i < 2 * kWords; ++i) ((uint2*)w)[i] = ((const uint2*)p)[i];
    } else {
      T* e = (T*)w;
#pragma unroll
      for (int i = 0; i < 8; ++i) e[i] = i < n_valid ? p[i] : T(0.f);
    }
  }
  __device__ __forceinline__ float get(int i) const { return to_f32<T>(((const T*)w)[i]); }
};

// Largest magnitude among the lane's eight values. 16-bit types: on pairs as they lie (a maximum of magnitudes is exact in
// any format, and NaN loses against a number as in fmaxf).
template <typename T>
__device__ __forceinline__ float block_amax_lane(const Raw8<T>& raw) {
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(raw.get(j)));
  return amax;
}
template <>
__device__ __forceinline__ float block_amax_lane<__nv_bfloat16>(const Raw8<__nv_bfloat16>& raw) {
  const __nv_bfloat162* h = (const __nv_bfloat162*)raw.w;
  const __nv_bfloat162 m = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
  const float2 f = __bfloat1622float2(m);
  return fmaxf(fmaxf(f.x, f.y), 0.f);
}
template <>
__device__ __forceinline__ float block_amax_lane<__half>(const Raw8<__half>& raw) {
  const __half2* h = (const __half2*)raw.w;
  const __half2 m = __hmax2(__hmax2(__habs2(h[0]), __habs2(h[1])), __hmax2(__habs2(h[2]), __habs2(h[3])));
  const float2 f = __half22float2(m);
  return fmaxf(fmaxf(f.x, f.y), 0.f);
}
// Exponent of the scale of a block with this largest magnitude: the smallest power of two >= amax / 448.
__device__ __forceinline__ int scale_exponent(float amax) {
  const int e = (int)ceilf(log2f(fmaxf(amax, 1e-12f) * (1.0f / 448.0f)));
  return max(-127, min(127, e));
}
// The same for the 16 lanes that hold one block.
template <typename T>
__device__ __forceinline__ int block_exponent(const Raw8<T>& raw) {
  float amax = block_amax_lane(raw);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  return scale_exponent(amax);
}
// NaN counts as the format's lowest value. 16-bit types: -inf in its place, two elements at a time; fp32 is left alone.
template <typename T>
__device__ __forceinline__ Raw8<T> nan_lowest(const Raw8<T>& raw) {
  if constexpr (sizeof(T) == 4) return raw;
  else {
    using T2 = std::conditional_t<std::is_same<T, __half>::value, __half2, __nv_bfloat162>;
    const uint32_t inf = std::is_same<T, __half>::value ? 0xfc00fc00u : 0xff80ff80u;
    Raw8<T> out;
#pragma unroll
    for (int i = 0; i < 4; ++i) ((T2*)out.w)[i] = __hmax2(((const T2*)raw.w)[i], *(const T2*)&inf);
    return out;
  }
}
// Four values as e4m3, the first in the lowest byte (saturating at 448).
__device__ __forceinline__ uint32_t e4m3x4(float a, float b, float c, float d) {
  uint32_t r;
  asm("{\n\t.reg .b16 lo, hi;\n\tcvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\tcvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\tmov.b32 %0, {lo, hi};\n\t}"
      : "=r"(r) : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}
// The lane's eight values divided by 2^e, as e4m3.
template <typename T>
__device__ __forceinline__ uint2 quantised8(const Raw8<T>& raw, int e) {
  const float inv = e == 127 ? 0x1p-127f : __int_as_float((127 - e) << 23);      // 2^-e
  const Raw8<T> clean = nan_lowest(raw);
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = clean.get(j) * inv;
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], -448.f);      // (NaN becomes -448)
  }
  return make_uint2(e4m3x4(v[0], v[1], v[2], v[3]), e4m3x4(v[4], v[5], v[6], v[7]));
}

}  // namespace
