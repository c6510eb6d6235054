// Local GEMM for few rows (tokens of a decode step, a short prompt): C[M, N] = A[M, K] @ B (+ bias), M <= 256,
// 16-bit operands, fp32 accumulation. Same operand layouts as the main loop of sm100_mainloop.cuh.
//
// Bound by reading B once (N * K * 2 bytes). The main loop gives every 128- to 256-wide column tile to one CTA, which for few
// rows means N / 128 CTAs that walk all of K: 16 x 3584 x 8192 ran on 28 of 148 SMs, 32.8 us against 8.9 us of
// HBM time, now 13.3 (16.4 before it started behind the kernel in front of it, launch_pdl.cuh). Here
//   * the tile is turned round: 128 columns of B are the M side of tcgen05.mma and the tokens, padded to 16,
//     the N side, so a stage holds 16 KB of weights and 128 bytes per token instead of 128 rows of padding;
//   * K is split over the CTAs of a cluster (up to 8). Each CTA keeps its partial tile in its own shared memory as fp32
//     and after one cluster barrier every CTA adds up a share of the tokens over distributed shared memory, in rank order:
//     no workspace, no atomics, the same bits on every run, one launch;
//   * the stage ring takes about 100 KB, so two CTAs fit an SM and clusters pack into any GPC (wider token tiles: see skinny_one_per_sm).
// The reference has no counterpart (its GEMMs go through tritonblas, iris/ops/matmul_all_reduce.py:95-105).
#include "gemm_host.cuh"
#include "gemm_skinny.h"

namespace {

constexpr int kSkinnyThreads = 192;      // warp 0 TMA, warp 1 MMA, warps 2..5 read TMEM; all of them reduce
constexpr int kWTile = 128 * kBK * 2;    // 16 KB of weights per stage
constexpr int kMaxStages = 12;
constexpr uint64_t kSkinnyWaitNs = 4000000000ull;

struct SkinnyArgs {
  CUtensorMap tmW, tmX;
  uint8_t* C;
  int64_t ldc;
  const void* bias_row;     // [M] or null
  const void* bias_col;     // [N] or null
  int32_t* status;
  int M, N, kblocks;
  int tn;                   // tokens padded to a multiple of 16
  int stages;
  int bf16, bias16, vec8;   // bias16: the bias has the output's type, else fp32; vec8: C rows take 8-byte stores
};

__device__ __forceinline__ float load_bias(const void* p, int i, int b16, int bf16) {
  if (!b16) return ((const float*)p)[i];
  return bf16 ? __bfloat162float(((const __nv_bfloat16*)p)[i]) : __half2float(((const __half*)p)[i]);
}

// kKMajor: B given as [N, K] (the weight's K is contiguous), else [K, N].
template <bool kKMajor>
__global__ void __launch_bounds__(kSkinnyThreads) skinny_gemm_kernel(const __grid_constant__ SkinnyArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = gridDim.x, rank = blockIdx.x;          // the cluster is one row of the grid
  const int n0 = blockIdx.y * 128;
  const int stage_bytes = kWTile + g.tn * (kBK * 2);
  const int ring_bytes = max(g.stages * stage_bytes, S > 1 ? g.tn * 512 : 0);
  uint64_t* full = (uint64_t*)(smem + ring_bytes);
  uint64_t* empty = full + kMaxStages;
  uint64_t* acc_full = empty + kMaxStages;
  uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
  uint32_t cols = 32;
  while ((int)cols < g.tn) cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) { ptx::mbar_init(&full[s], 1); ptx::mbar_init(&empty[s], 1); }
    ptx::mbar_init(acc_full, 1);
    ptx::fence_mbar_init();
    ptx::fence_proxy_async();
  }
  __syncthreads();
  const int kb0 = (int)((int64_t)g.kblocks * rank / S), kb1 = (int)((int64_t)g.kblocks * (rank + 1) / S);
  // The first ring's weights on their way into L2 while the kernel in front drains (its writes, if it wrote them, are in L2 as well):
  // 16 x 3584 x 8192 13.7 -> 13.3 us back to back, 48-token MLP 29.6 -> 28.9. More than the ring holds was slower (14.0, 30.1), and so
  // were smaller rings that leave room for a third CTA, whose prefetches met the running kernel's own loads (15.2, 33.2).
  if (warp == 0) {
    for (int kb = kb0 + lane; kb < min(kb1, kb0 + g.stages); kb += 32) {
      if constexpr (kKMajor) {
        ptx::tma_prefetch_2d(&g.tmW, kb * kBK, n0);
      } else {
        ptx::tma_prefetch_2d(&g.tmW, n0, kb * kBK);
        ptx::tma_prefetch_2d(&g.tmW, n0 + 64, kb * kBK);
      }
    }
    __syncwarp();
  }
  ptx::pdl_wait();
  // only now the columns (launch_pdl.cuh), while warp 0 already loads
  uint32_t tmem_base = 0;
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, cols);
    ptx::tmem_relinquish();
    ptx::tc_fence_before();
    ptx::pdl_trigger();
  }
  if (warp != 0) {
    ptx::named_barrier(1, kSkinnyThreads - 32);
    ptx::tc_fence_after();
    tmem_base = *(volatile uint32_t*)tmem_slot;
  }
  auto fail = [&]() { if (g.status) atomicCAS(g.status, 0, (int)kTimeoutPipeline); };

  bool live = true;
  if (warp == 0) {
    const uint32_t base = ptx::smem_u32(smem);
    int s = 0;
    uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&empty[s], ph ^ 1, kSkinnyWaitNs))) { fail(); break; }
      const uint32_t sw = base + s * stage_bytes, sx = sw + kWTile;
      ptx::mbar_expect_tx_elect(&full[s], stage_bytes);
      if constexpr (kKMajor) {
        ptx::tma_load_2d_elect(sw, &g.tmW, &full[s], kb * kBK, n0);
      } else {
        ptx::tma_load_2d_elect(sw, &g.tmW, &full[s], n0, kb * kBK);
        ptx::tma_load_2d_elect(sw + 8192, &g.tmW, &full[s], n0 + 64, kb * kBK);
      }
      ptx::tma_load_2d_elect(sx, &g.tmX, &full[s], kb * kBK, 0);
      if (++s == g.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const uint32_t tmem_u = __reduce_or_sync(0xffffffffu, tmem_base);
    const uint32_t idesc = make_idesc(g.tn, g.bf16 != 0, false) | (kKMajor ? 0u : 1u << 15);      // bit 15: A is M-major
    const uint32_t base = ptx::smem_u32(smem);
    int s = 0;
    uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&full[s], ph, kSkinnyWaitNs))) { fail(); break; }
      ptx::tc_fence_after();
      const uint32_t sw = base + s * stage_bytes, sx = sw + kWTile;
#pragma unroll
      for (int k = 0; k < kBK / kUmmaK; ++k) {
        const uint64_t ad = kKMajor ? desc_kmajor(sw + k * (kUmmaK * 2)) : desc_mnmajor(sw + k * (kUmmaK * 128));
        ptx::mma_f16_elect(tmem_u, ad, desc_kmajor(sx + k * (kUmmaK * 2)), idesc, (kb - kb0) | k);
      }
      ptx::mma_commit_elect(&empty[s]);
      if (kb == kb1 - 1) ptx::mma_commit_elect(acc_full);
      if (++s == g.stages) { s = 0; ph ^= 1; }
    }
  } else {
    // TMEM lane = column of the tile, TMEM column = token
    live = ptx::mbar_wait(acc_full, 0, kSkinnyWaitNs);
    if (!live) fail();
    live = __all_sync(0xffffffffu, live);
    ptx::tc_fence_after();
    if (live) {
      const int quarter = warp & 3, col = quarter * 32 + lane, n = n0 + col;
      const uint32_t t_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
      float* part = (float*)smem;            // [tokens][128]: the stages have been read by then
      const float bc = (S == 1 && g.bias_col && n < g.N) ? load_bias(g.bias_col, n, g.bias16, g.bf16) : 0.f;
      for (int c = 0; c < g.tn; c += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32(t_addr + c, r);   // (tn is a multiple of 16: the last load may read allocated columns past it)
        ptx::tmem_ld_wait();
        if (S > 1) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (c + j < g.tn) part[(c + j) * 128 + col] = __uint_as_float(r[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int t = c + j;
            if (t < g.M && n < g.N) {
              float v = __uint_as_float(r[j]) + bc;
              if (g.bias_row) v += load_bias(g.bias_row, t, g.bias16, g.bf16);
              uint16_t* dst = (uint16_t*)g.C + (int64_t)t * g.ldc + n;
              if (g.bf16) { const __nv_bfloat16 h = __float2bfloat16_rn(v); *dst = *(const uint16_t*)&h; }
              else { const __half h = __float2half_rn(v); *dst = *(const uint16_t*)&h; }
            }
          }
        }
      }
    }
  }
  ptx::tc_fence_before();
  if (S > 1) {
    __syncwarp();
    ptx::cluster_sync();
    // token t of the tile is finished by CTA t % S: a warp per token, four columns per lane
    const uint32_t part0 = ptx::smem_u32(smem);
#pragma unroll 2
    for (int t = rank + (warp * S); t < g.M; t += S * (kSkinnyThreads / 32)) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      const uint32_t local = part0 + (uint32_t)(t * 512 + lane * 16);
      float4 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c >= S) break;
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(c));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[c].x), "=f"(v[c].y), "=f"(v[c].z), "=f"(v[c].w) : "r"(remote) : "memory");
      }
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (c >= S) break;
        acc.x += v[c].x; acc.y += v[c].y; acc.z += v[c].z; acc.w += v[c].w;
      }
      const int n = n0 + lane * 4;
      if (n < g.N) {                         // N is a multiple of 8: four columns are inside together
        float o[4] = {acc.x, acc.y, acc.z, acc.w};
        const float br = g.bias_row ? load_bias(g.bias_row, t, g.bias16, g.bf16) : 0.f;
        uint16_t h[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float x = o[e] + br;
          if (g.bias_col) x += load_bias(g.bias_col, n + e, g.bias16, g.bf16);
          if (g.bf16) { const __nv_bfloat16 b = __float2bfloat16_rn(x); h[e] = *(const uint16_t*)&b; }
          else { const __half b = __float2half_rn(x); h[e] = *(const uint16_t*)&b; }
        }
        uint16_t* dst = (uint16_t*)g.C + (int64_t)t * g.ldc + n;
        if (g.vec8) *(uint2*)dst = make_uint2(h[0] | ((uint32_t)h[1] << 16), h[2] | ((uint32_t)h[3] << 16));
        else
          for (int e = 0; e < 4; ++e) dst[e] = h[e];
      }
    }
    // a CTA's shared memory stays until every CTA has read it (with a release here, the CTA stayed until its output was written: 1.5 us)
    __syncwarp();
    ptx::cluster_sync_relaxed();
  } else {
    __syncthreads();
  }
  ptx::tc_fence_after();
  if (warp == 1) ptx::tmem_dealloc(tmem_base, cols);
}

}  // namespace

// Up to 64 tokens, and mostly up to 128, the ring is kept to about 100 KB and two CTAs share an SM; wider token tiles take an SM each, and then
// clusters of 8 leave SMs of a GPC unused (256 x 2000 x 3000: 16 clusters of 8 did not fit at once, 26 us), so 4 is
// the limit unless there are few of them.
static int split_for(int tiles, int kb, int slots, int most) {
  int s = 1;
  while (s < most && tiles * (s * 2) <= slots && kb >= 4 * (s * 2)) s *= 2;
  return s;
}
// 65 to 128 tokens fill 100 KB with three stages. Where CTAs that take an SM each, with six, still cover most of the chip, or a handful of
// tiles is split by 8 either way, those are the faster ones (us, two CTAs per SM / one): 100 x 4096 x 2048 10.7 / 8.2, 128 x 3584 x 8192
// 18.9 / 16.7, 100 x 4096 x 4096 13.7 / 12.6, 128 x 1024 x 8192 11.8 / 9.6, but 100 x 8192 x 8192 (64 tiles, split by 2 then) 27.4 / 28.8
// and 100 x 2048 x 4096 (16 clusters of 8 do not fit at once) 10.2 / 14.4.
static bool skinny_one_per_sm(int tn, int tiles, int kb) {
  if (tn <= 64) return false;
  if (tn > 128) return true;
  const int s = split_for(tiles, kb, sm_count(), tiles <= 12 ? 8 : 4);
  return tiles <= 12 || (s == 4 && 8 * tiles * s >= 5 * sm_count());      // (24 tiles and more of 148 SMs)
}
int iris_gemm_skinny_split(int M, int N, int K) {
  const int tiles = ceil_div(N, 128), kb = ceil_div(K, kBK), tn = ceil_div(M, 16) * 16;
  if (!skinny_one_per_sm(tn, tiles, kb)) return split_for(tiles, kb, 2 * sm_count(), 8);
  return split_for(tiles, kb, sm_count(), tiles <= 12 ? 8 : 4);
}

// Where the split-K kernel is the faster one, both measured in us with weights that are not in L2 (main loop / this):
//   M = 8     1024 x 1024  6.9 / 4.5    3584 x 8192  31.7 / 14.1    8192 x 3584  27.3 / 13.7    8192 x 8192  35.0 / 25.2
//   M = 48    8192 x 1024  9.4 / 9.2 (weights [N, K]), 8.6 / 9.2 ([K, N])    5120 x 2048  11.6 / 9.8
//   M = 128   1024 x 1024  7.2 / 7.8    5120 x 2048  11.8 / 13.1    8192 x 3584  18.0 / 18.2    2048 x 2048  11.5 / 11.4
//             3584 x 4096  18.3 / 14.4    8192 x 8192  36.2 / 30.4
//   M = 256   2048 x 2048  11.5 / 13.4    8192 x 8192  37.2 / 42.7    5120 x 8192  33.9 / 37.5
//             2000 x 3000  22.0 / 17.1    3584 x 4096  18.5 / 17.4    3584 x 8192  32.1 / 23.5
// It pays while K is long against N (the main loop's few CTAs walk all of it) and its partial tiles, which grow with M,
// stay small.
// A tile that the caller asked for is honoured; a fused op on one rank otherwise carries the tile of its workspace's
// plan, which binds nobody there.
extern "C" int iris_gemm_skinny_takes(const IrisGemmDesc* d) {
  if (d->op == IRIS_GEMM_LOCAL ? d->bn != 0 || d->two_sm != 0 : d->tile_asked != 0) return 0;
  if (d->timeline || (d->in_dtype != 0 && d->in_dtype != d->dtype)) return 0;
  if (d->M <= 32) return 1;
  if (d->M <= 64) return d->K >= 2048 || d->N <= 4096;
  return d->M <= 256 && d->K >= (d->M <= 128 ? 2048 : 2816) && 2ll * d->K >= d->N && (int64_t)d->M * d->N <= (1 << 20);
}

int iris_gemm_skinny(const IrisGemmDesc* d, cudaStream_t stream) {
  if (d->M < 1 || d->M > 256 || d->N % 8 || d->K % 8) return -3;
  if (d->dtype != IRIS_BF16 && d->dtype != IRIS_F16) return -2;
  SkinnyArgs g;
  g.M = d->M; g.N = d->N; g.kblocks = ceil_div(d->K, kBK);
  g.tn = ceil_div(d->M, 16) * 16;
  int r = make_map(&g.tmX, d->A, d->dtype, d->M, d->K, d->lda, kBK, g.tn);
  if (r) return r;
  if (d->b_kmajor) r = make_map(&g.tmW, d->B, d->dtype, d->N, d->K, d->ldb, kBK, 128);
  else r = make_map(&g.tmW, d->B, d->dtype, d->K, d->N, d->ldb, 64, 64);
  if (r) return r;
  g.C = (uint8_t*)d->C; g.ldc = d->ldc;
  g.bias_row = d->bias_row; g.bias_col = d->bias_col; g.bias16 = d->bias16;
  g.status = d->ctx.status;
  g.bf16 = d->dtype == IRIS_BF16;
  g.vec8 = ((uintptr_t)d->C & 7) == 0 && d->ldc % 4 == 0;
  const int S = iris_gemm_skinny_split(d->M, d->N, d->K);
  const int stage = kWTile + g.tn * (kBK * 2);
  const int budget = skinny_one_per_sm(g.tn, ceil_div(g.N, 128), g.kblocks) ? 208 * 1024 : 104 * 1024;
  g.stages = budget / stage;
  if (g.stages > kMaxStages) g.stages = kMaxStages;
  const int ring = S > 1 && g.tn * 512 > g.stages * stage ? g.tn * 512 : g.stages * stage;
  const int smem = 1024 + ring + (2 * kMaxStages + 1) * 8 + 64;
  auto* kern = d->b_kmajor ? skinny_gemm_kernel<true> : skinny_gemm_kernel<false>;
  static bool attr = false;
  if (!attr) {
    const int most = 1024 + 208 * 1024 + (2 * kMaxStages + 1) * 8 + 64;
    if (cudaFuncSetAttribute(skinny_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return -20;
    if (cudaFuncSetAttribute(skinny_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess) return -20;
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S, ceil_div(d->N, 128), 1);
  cfg.blockDim = dim3(kSkinnyThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = S; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // see launch_pdl.cuh
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, g) == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -21;
}
