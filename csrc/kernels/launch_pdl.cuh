// Programmatic dependent launch (see ptx::pdl_wait in iris/ptx.cuh).
//
// A kernel launched this way may start while the stream's last kernel still runs: when all of its CTAs have issued
// ptx::pdl_trigger(), or have left. So the launch latency, the set-up (barriers, tensor memory) and the last wave of the
// kernel in front overlap; back to back that was 2 to 4 us of every pass. Rules for the kernels:
//   * ptx::pdl_wait() by every thread before it touches memory that an earlier kernel may have written or may still read;
//   * and by no read-only promise about such memory: a `const T* __restrict__` parameter, __ldg or ld.global.nc lets a load move in front
//     of the wait, or return what lay there before;
//   * a kernel that allocates tensor memory triggers only when it has its columns: a later kernel must not take columns that
//     an earlier one still waits for.
// A kernel behind one of these that is launched the ordinary way waits for it to finish, as always.
#pragma once
#include <cuda_runtime.h>

namespace {

template <class... P, class... A>
int launch_pdl(void (*kern)(P...), dim3 grid, int block, int smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<A&&>(args)...) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // namespace
