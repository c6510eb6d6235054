// Activation quantiser for the block-scaled fp8 paths: x [M, K] (fp32 / bf16 / fp16) -> e4m3 values with
// one power-of-two scale per row and 128-wide K block, written in the three forms the kernels use:
//   q      [M, K] e4m3
//   scale  [M, KB] fp32 (optional; what the PyTorch oracle multiplies by)
//   atoms  [ceil(M / 128), KB, 512] UE8M0 bytes in the layout tcgen05.cp copies into TMEM: row r of a
//          128-row tile at byte (r % 32) * 16 + (r / 32) * 4, four equal bytes (the four 32-element K
//          groups of the block share the scale).
//   rows   [M, ld_rows] one UE8M0 byte per row and K block (optional): the form that travels with a row when
//          rows are routed one by one (MoE dispatch); the consumer builds the atoms of its tiles from it.
// The reference has no quantised path; this plays the role of the activation cast in front of its
// 16-bit GEMMs (iris/ops/matmul_all_reduce.py:95-105 consumes 16-bit tiles directly).
//
// Half a warp takes one (row, K block): eight elements per lane, so a lane's load is 16 bytes (two for fp32) and its store
// 8, and a warp keeps kUnroll pairs of blocks in flight before it reduces the first. With one block per warp and 8-byte loads
// the kernel waited on latency (4096 x 8192 bf16: 61 us); since then the arithmetic per element bounds it, not its bytes
// (15 us): maxima on pairs of 16-bit values, one exponent and one scale write per block instead of one per lane and
// block, 32-bit index arithmetic (33 us, then 23). Collecting the scale atoms in shared memory was slower (38 us).
// amax by shuffles, scale = 2^ceil(log2(amax / 448)).
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>
#include <type_traits>

#include "iris/host_api.h"
#include "iris/ptx.cuh"
#include "launch_pdl.cuh"
#include "quantize_common.cuh"

namespace {

// Up to this many blocks, about a wave, the kernel starts behind the one in front of it and lets the next one start (launch_pdl.cuh;
// 16 x 4096 and its GEMM 17.6 -> 14.2 us). Of many waves the first would be placed around the last CTAs of the kernel in front, and the
// next kernel's CTAs between the last: 4096 x 8192 and its GEMM 117 us instead of 114.
constexpr unsigned kBehindMax = 1024;
constexpr int kUnroll = 4;      // pairs of blocks a warp has in flight (the reduction below is written for four)

// The four blocks' maxima by halving: each exchange leaves a lane with half of its blocks, until four lanes share one
// block; they work its exponent out once, and everybody fetches the four exponents. Returns that of block sub / 4.
template <typename T>
__device__ __forceinline__ int shared_exponent(const Raw8<T> (&raw)[kUnroll], int sub) {
  float amax[kUnroll];
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) amax[i] = block_amax_lane(raw[i]);
  const bool hi8 = sub & 8, hi4 = sub & 4;
  float m0 = hi8 ? amax[2] : amax[0], m1 = hi8 ? amax[3] : amax[1];
  m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, hi8 ? amax[0] : amax[2], 8));
  m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, hi8 ? amax[1] : amax[3], 8));
  float mine = fmaxf(hi4 ? m1 : m0, __shfl_xor_sync(0xffffffffu, hi4 ? m0 : m1, 4));
  mine = fmaxf(mine, __shfl_xor_sync(0xffffffffu, mine, 2));
  mine = fmaxf(mine, __shfl_xor_sync(0xffffffffu, mine, 1));
  return scale_exponent(mine);
}

// Rows of whole blocks on 16-byte boundaries: a warp takes eight blocks of ONE row, so its addresses are one base and constants.
// The general kernel below spends half of its instructions on rows and columns that change from block to block, and it is
// bound by issue slots (4096 x 8192 bf16: 24.0 us, 152 instructions per warp and 256 values; this one 18.1 us and 98, with NaN
// replaced two values at a time and four conversions to a word).
template <typename T>
__global__ void __launch_bounds__(128) quantize_rows_kernel(const T* x, int64_t ldx, uint8_t* q, int64_t ldq, float* scale, uint8_t* atoms, uint8_t* rows,
                                                             int64_t ld_rows, int M, int M_pad, int KB, int groups) {
  if (gridDim.x <= kBehindMax) iris::ptx::pdl_trigger();
  iris::ptx::pdl_wait();
  const unsigned unit = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31, sub = lane & 15;
  const int row = (int)(unit / (unsigned)groups), kb0 = (int)(unit % (unsigned)groups) * (2 * kUnroll) + (lane >> 4);
  if (row >= M_pad) return;
  Raw8<T> raw[kUnroll];
  const T* src = x + (int64_t)row * ldx + kb0 * 128 + sub * 8;
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) raw[i].load(src + i * 256, row < M && kb0 + 2 * i < KB ? 8 : 0, 2);
  const int e_mine = shared_exponent(raw, sub);       // of block sub / 4
  const int kb_mine = kb0 + 2 * (sub >> 2);
  if ((sub & 3) == 0 && kb_mine < KB) {               // whose scale one of the four lanes writes
    if (row < M) {
      if (scale) scale[(int64_t)row * KB + kb_mine] = exp2f((float)e_mine);
      if (rows) rows[(int64_t)row * ld_rows + kb_mine] = (uint8_t)(e_mine + 127);
    }
    if (atoms) {
      const uint32_t byte = row < M ? (uint32_t)(e_mine + 127) : 127u;      // rows past M: scale 1
      *(uint32_t*)(atoms + ((int64_t)(row >> 7) * KB + kb_mine) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4) = byte * 0x01010101u;
    }
  }
  uint8_t* dst = q + (int64_t)row * ldq + kb0 * 128 + sub * 8;
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) {
    const int e = __shfl_sync(0xffffffffu, e_mine, (lane & 16) + i * 4);
    if (row < M && kb0 + 2 * i < KB) *(uint2*)(dst + i * 256) = quantised8(raw[i], e);
  }
}

template <typename T>
__global__ void __launch_bounds__(128) quantize_1x128_pow2_kernel(const T* x, int64_t ldx, uint8_t* q, int64_t ldq, float* scale, uint8_t* atoms,
                                                                   uint8_t* rows, int64_t ld_rows, int M, int M_pad, int K, int KB,
                                                                   int x_aligned, int q_aligned) {
  if (gridDim.x <= kBehindMax) iris::ptx::pdl_trigger();
  iris::ptx::pdl_wait();
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, half = lane >> 4, sub = lane & 15;
  const int64_t units = (int64_t)M_pad * KB, u0 = warp * (2 * kUnroll);
  if (u0 >= units) return;
  const int64_t first = u0 + half;
  // (a 64-bit division costs as much as the rest of the thread's addressing: only when the count needs it)
  int row = units <= 0x7fffffffll ? (int)((unsigned)first / (unsigned)KB) : (int)(first / KB);
  int kb = (int)(first - (int64_t)row * KB);
  int rows_u[kUnroll], kbs_u[kUnroll];
  Raw8<T> raw[kUnroll];
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) {
    rows_u[i] = row; kbs_u[i] = kb;
    const int k0 = kb * 128 + sub * 8;
    const int n_valid = row < M ? max(0, min(8, K - k0)) : 0;
    raw[i].load(x + (int64_t)row * ldx + k0, n_valid, x_aligned);
    for (kb += 2; kb >= KB; kb -= KB) ++row;
  }
  const bool hi8 = sub & 8, hi4 = sub & 4;
  const int e_mine = shared_exponent(raw, sub);       // of block sub / 4
  if ((sub & 3) == 0) {                               // whose scale one of the four lanes writes
    const int r = hi8 ? (hi4 ? rows_u[3] : rows_u[2]) : (hi4 ? rows_u[1] : rows_u[0]);
    const int b = hi8 ? (hi4 ? kbs_u[3] : kbs_u[2]) : (hi4 ? kbs_u[1] : kbs_u[0]);
    if (r < M) {
      if (scale) scale[(int64_t)r * KB + b] = exp2f((float)e_mine);
      if (rows) rows[(int64_t)r * ld_rows + b] = (uint8_t)(e_mine + 127);
    }
    if (atoms && r < M_pad) {
      const uint32_t byte = r < M ? (uint32_t)(e_mine + 127) : 127u;      // rows past M: scale 1
      const int tile = r >> 7, rr = r & 127;
      *(uint32_t*)(atoms + ((int64_t)tile * KB + b) * 512 + (rr & 31) * 16 + (rr >> 5) * 4) = byte * 0x01010101u;
    }
  }
#pragma unroll
  for (int i = 0; i < kUnroll; ++i) {
    const int r = rows_u[i], b = kbs_u[i];
    const int e = __shfl_sync(0xffffffffu, e_mine, (lane & 16) + i * 4);
    if (r < M) {
      const uint2 v = quantised8(raw[i], e);
      const int k0 = b * 128 + sub * 8, n_valid = max(0, min(8, K - k0));
      uint8_t* dst = q + (int64_t)r * ldq + k0;
      if (n_valid == 8 && q_aligned == 2) {
        *(uint2*)dst = v;
      } else if (n_valid == 8 && q_aligned == 1) {
        ((uint32_t*)dst)[0] = v.x; ((uint32_t*)dst)[1] = v.y;
      } else
        for (int j = 0; j < n_valid; ++j) dst[j] = (uint8_t)((j < 4 ? v.x : v.y) >> (8 * (j & 3)));
    }
  }
}

}  // namespace

// x: [M, K] of `dtype` (IRIS_F32 / IRIS_BF16 / IRIS_F16), row pitch ldx elements. q: [M, K] bytes, pitch ldq.
// scale (may be null): [M, ceil(K / 128)] fp32. atoms (may be null): [ceil(M / 128), ceil(K / 128), 512] bytes;
// rows past M inside the last 128-row tile are written as 127 (scale 1).
static int quantize_launch(const void* x, int64_t ldx, int32_t dtype, void* q, int64_t ldq, float* scale, void* atoms, void* rows,
                           int64_t ld_rows, int32_t M, int32_t K, void* stream) {
  if (M <= 0 || K <= 0) return 0;
  const int KB = (K + 127) / 128;
  const int M_pad = atoms ? (int)(((int64_t)M + 127) / 128 * 128) : M;
  const int64_t warps = ((int64_t)M_pad * KB + 2 * kUnroll - 1) / (2 * kUnroll);
  const int64_t blocks = (warps * 32 + 127) / 128;
  if (blocks > 0x7fffffffll) return -3;
  cudaStream_t s = (cudaStream_t)stream;
  const int esz = dtype == IRIS_F32 ? 4 : 2;
  auto level = [](const void* p, int64_t pitch, int big, int small) {     // alignment of every row start
    const uint64_t bits = (uint64_t)(uintptr_t)p | (uint64_t)pitch;
    return bits % big == 0 ? 2 : (bits % small == 0 ? 1 : 0);
  };
  const int xa = level(x, ldx * esz, 16, 8), qa = level(q, ldq, 8, 4);
  // by rows while at most a fifth of a warp's eight blocks fall behind the row's end
  const int groups = (KB + 2 * kUnroll - 1) / (2 * kUnroll);
  const bool by_rows = xa == 2 && qa == 2 && K % 128 == 0 && 5 * KB >= 4 * groups * 2 * kUnroll && (int64_t)M_pad * groups < (1ll << 31);
  int r = 0;
  auto run = [&](auto* typed) {
    using T = std::remove_cv_t<std::remove_pointer_t<decltype(typed)>>;
    if (by_rows) {
      const unsigned n = (unsigned)(((int64_t)M_pad * groups + 3) / 4);
      if (n <= kBehindMax)
        r = launch_pdl(quantize_rows_kernel<T>, dim3(n), 128, 0, s, (const T*)typed, ldx, (uint8_t*)q, ldq, scale, (uint8_t*)atoms, (uint8_t*)rows, ld_rows,
                       M, M_pad, KB, groups);
      else
        quantize_rows_kernel<T><<<n, 128, 0, s>>>(typed, ldx, (uint8_t*)q, ldq, scale, (uint8_t*)atoms, (uint8_t*)rows, ld_rows, M, M_pad, KB, groups);
    } else if (blocks <= kBehindMax)
      r = launch_pdl(quantize_1x128_pow2_kernel<T>, dim3((unsigned)blocks), 128, 0, s, (const T*)typed, ldx, (uint8_t*)q, ldq, scale, (uint8_t*)atoms,
                     (uint8_t*)rows, ld_rows, M, M_pad, K, KB, xa, qa);
    else
      quantize_1x128_pow2_kernel<T><<<(unsigned)blocks, 128, 0, s>>>(typed, ldx, (uint8_t*)q, ldq, scale, (uint8_t*)atoms, (uint8_t*)rows, ld_rows, M,
                                                                     M_pad, K, KB, xa, qa);
  };
  if (dtype == IRIS_F32) run((const float*)x);
  else if (dtype == IRIS_BF16) run((const __nv_bfloat16*)x);
  else if (dtype == IRIS_F16) run((const __half*)x);
  else
    return -2;
  return r ? r : cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int iris_quantize_1x128_pow2(const void* x, int64_t ldx, int32_t dtype, void* q, int64_t ldq, float* scale, void* atoms,
                                        int32_t M, int32_t K, void* stream) {
  return quantize_launch(x, ldx, dtype, q, ldq, scale, atoms, nullptr, 0, M, K, stream);
}
// Same, writing one scale byte per row and K block into rows [M, ld_rows] (bytes past ceil(K / 128) of a row are left alone).
extern "C" int iris_quantize_1x128_pow2_rows(const void* x, int64_t ldx, int32_t dtype, void* q, int64_t ldq, void* rows, int64_t ld_rows,
                                             int32_t M, int32_t K, void* stream) {
  return quantize_launch(x, ldx, dtype, q, ldq, nullptr, nullptr, rows, ld_rows, M, K, stream);
}
