// Programmatic dependent launch (see ptx::pdl_wait in iris/ptx.cuh).
//
// A kernel launched this way may start while the stream's last kernel still runs: when all of its CTAs have issued
// ptx::pdl_trigger(), or have left. So the launch latency, the set-up (barriers, descriptors) and the last wave of the
// kernel in front overlap; back to back that was 2 to 4 us of every pass. Rules for the kernels:
//   * ptx::pdl_wait() by every thread before it touches memory that an earlier kernel may have written or may still read. Before it a kernel may
//     read only what was complete when the kernel in front of it triggered, and so only behind one that triggers behind its own wait: everything
//     in front of that one has completed by then. The MoE layer on one rank does so: the gather of 16-bit tokens reads them behind the preparation or the
//     sort, stage 1 of the grouped GEMMs reads weights and the preparation's tables behind the gather, stage 2 the same behind stage 1 (which
//     starts when the gather has triggered). Their triggers must not move in front of their waits. An L2 prefetch is no read;
//   * and by no read-only promise about such memory: a `const T* __restrict__` parameter, __ldg or ld.global.nc lets a load move in front
//     of the wait, or return what lay there before;
//   * tensor memory is allocated behind pdl_wait(). A CTA that held columns while it waits could share an SM with a CTA of the kernel in
//     front that still asks for its own (a library's kernel may trigger before it has them), and each would wait for the other;
//   * pdl_trigger() stands behind the allocation, for the same reason the other way round: a kernel behind this one may allocate first.
// So nothing is expected of kernels from elsewhere, in front or behind. (Allocating behind the wait instead of in front of it costs nothing where the
// loading warp goes ahead meanwhile: 16 x 3584 x 8192 13.2 us both ways, two products of 2048 x 2048 x 2048 33.5 and 33.1, but 34.7 when
// the loads waited for the allocation too; e4m3 4096 x 3584 x 8192 128.7 and 128.2.) expert_gemm_kernel allocates in front of its
// wait: it is launched behind the MoE layer's own kernels only, and everything that was in front of those has completed by then.
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
