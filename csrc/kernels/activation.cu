// Activation passes of the tensor-parallel MLP's training step (silu, gelu with the tanh approximation), 16-bit
// values, fp32 arithmetic:
//   forward   h = act(pre)
//   backward  dpre = dh * act'(pre)  and, in the same pass, h = act(pre) again for the weight gradient
// (the reference's autograd wrapper, examples/07_gemm_all_scatter/matmul_wrapper.py, has no activation).
//
// Bound by memory: 4 bytes per element forward, 8 backward. Written as tensor expressions the backward took
// eleven passes, most of them over fp32 copies (2048 x 3584 bf16: 108 us of kernels); one pass that reads dh and
// pre and writes dpre and h moves 59 MB (11.6 us). Each thread takes eight elements (16-byte loads and stores); the
// last n % 8 elements go one by one.
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <type_traits>

#include "iris/host_api.h"

namespace {

enum Act { kSilu = 1, kGelu = 2 };

// act(x) and act'(x)
template <int kAct>
__device__ __forceinline__ void act_and_grad(float x, float& y, float& g) {
  if constexpr (kAct == kSilu) {
    const float s = 1.f / (1.f + expf(-x));
    y = x * s;
    g = s * (1.f + x * (1.f - s));
  } else {
    // 0.5 x (1 + tanh(u)), u = sqrt(2 / pi) (x + 0.044715 x^3)
    const float k0 = 0.7978845608028654f, k1 = 0.044715f;
    const float t = tanhf(k0 * (x + k1 * x * x * x));
    y = 0.5f * x * (1.f + t);
    g = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
  }
}

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// h may be null; dh and dpre are null together (forward).
template <typename T, int kAct>
__global__ void __launch_bounds__(256) activation_kernel(const T* __restrict__ pre, const T* __restrict__ dh, T* __restrict__ h,
                                                         T* __restrict__ dpre, int64_t n) {
  const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (i0 >= n) return;
  if (i0 + 8 <= n) {
    uint4 vp = *(const uint4*)(pre + i0), vd = make_uint4(0, 0, 0, 0), vh, vo;
    if (dh) vd = *(const uint4*)(dh + i0);
    const T* ep = (const T*)&vp;
    const T* ed = (const T*)&vd;
    T* eh = (T*)&vh;
    T* eo = (T*)&vo;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float y, g;
      act_and_grad<kAct>(to_f32<T>(ep[j]), y, g);
      eh[j] = from_f32<T>(y);
      eo[j] = from_f32<T>(to_f32<T>(ed[j]) * g);
    }
    if (h) *(uint4*)(h + i0) = vh;
    if (dpre) *(uint4*)(dpre + i0) = vo;
  } else {
    for (int64_t i = i0; i < n; ++i) {
      float y, g;
      act_and_grad<kAct>(to_f32<T>(pre[i]), y, g);
      if (h) h[i] = from_f32<T>(y);
      if (dpre) dpre[i] = from_f32<T>(to_f32<T>(dh[i]) * g);
    }
  }
}

}  // namespace

// act: 1 silu, 2 gelu (tanh). dtype IRIS_BF16 / IRIS_F16. n contiguous elements, every pointer 16-byte aligned.
// Forward: dh = dpre = null. Backward: h may be null.
extern "C" int iris_activation(const void* pre, const void* dh, void* h, void* dpre, int64_t n, int32_t act, int32_t dtype, void* stream) {
  if (n < 0 || (dh == nullptr) != (dpre == nullptr)) return -3;
  if (n == 0) return 0;
  if (((uintptr_t)pre | (uintptr_t)dh | (uintptr_t)h | (uintptr_t)dpre) & 15) return -11;
  const int64_t blocks = (n + 2047) / 2048;
  if (blocks > 0x7fffffffll) return -3;
  cudaStream_t s = (cudaStream_t)stream;
  auto run = [&](auto* t) {
    using T = std::remove_pointer_t<decltype(t)>;
    auto* k = act == kSilu ? activation_kernel<T, kSilu> : activation_kernel<T, kGelu>;
    k<<<(unsigned)blocks, 256, 0, s>>>((const T*)pre, (const T*)dh, (T*)h, (T*)dpre, n);
  };
  if (act != kSilu && act != kGelu) return -3;
  if (dtype == IRIS_BF16) run((__nv_bfloat16*)nullptr);
  else if (dtype == IRIS_F16) run((__half*)nullptr);
  else return -2;
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
