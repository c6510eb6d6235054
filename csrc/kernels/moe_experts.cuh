// The two grouped GEMMs of the MoE layer on one rank (weights stored K-major), included by moe.cu.
//
// Decode batches are bound by reading every used expert's weights once, prefill batches by the tensor cores. Both want the
// same tile: 256 rows of WEIGHTS on the M side of a CTA pair's tcgen05.mma (128 per CTA) and the expert's TOKENS, padded
// to a multiple of 16, on the N side. An expert's rows are cut into equal tiles of at most kMaxN tokens, so no MMA works
// on padding beyond 15 rows per tile, whereas 128-row token tiles multiplied the padding of every expert's last tile (and, for
// 16 tokens per expert, seven eighths of all rows); 256-row weight tiles cut 32 experts' gate|up weights into 512 units for
// 74 pairs (6.9 rounds in the time of 7), where 148 single CTAs took the time of 4 for 3.5.
//   warp 0      TMA producer: weights, tokens and (e4m3) scale atoms into a ring of stages
//   warp 1      MMA issuer (even CTA of the pair), fp32 accumulators in TMEM, two buffers
//   warps 2..9  epilogue: TMEM lane = weight row, TMEM column = token; read as mma fragments and transposed by stmatrix
// Stage 1 (gate|up): the weight rows are stored as blocks of [gate 128 | up 128]. Each CTA loads 64 gate and 64 up rows
// interleaved by 16, so a warp reads the gate and up values of 16 features into the same threads. In e4m3 a 128-feature
// quantisation block of H spans the pair: the CTAs exchange each token's largest magnitude by asynchronous stores into each
// other's shared memory (a release at cluster scope waited for the warp's global stores of the tile before).
// Stage 2 (down): every output row goes to the (token, k) slot it came from.
// Gate and up stay fp32 up to SwiGLU (the kernel of several ranks rounds e4m3's to bf16 first, and is the further one from 64 bits: 1.81e-2 and 1.64e-2 with
// hidden values rounded once). The division is exact; a fast one, which returns 0 for denominators above 2^126, saves 1 to 3 % of a pass.
// Whole layer, before (128-row token tiles on single CTAs) and now: 32 experts top-8 of 7168 x 2048, 64 tokens e4m3 316 and 241 us
// (its weights' HBM time is 226), bf16 498 and 430; 4096 tokens bf16, the kernels alone, stage 1 1583 and 1320 us, stage 2 780 and 628.
// 4096 tokens, 32 experts top-8 of 2048 x 1024: stage 1 bf16 218 and 184 us, e4m3 280 and 142 (336 with one shuffle and one 2-byte
// store per value, four epilogue warps and full-precision divisions), stage 2 117 and 102, 119 and 79.
#pragma once
#include "gemm_host.cuh"

namespace {

constexpr int kExpertMax = 1024;         // experts of a layer (the router's limit)
constexpr int kXEpiWarps = 8;            // epilogue warps: two per quarter of the TMEM lanes, every other 32 tokens each
constexpr int kXThreads = 64 + 32 * kXEpiWarps;

struct ExpertArgs {
  CUtensorMap tmW;         // weights: stage 1 [2 * blocks][128][D], stage 2 [El * D, F]
  CUtensorMap tmX[4];      // token rows, boxes of kMaxN / 2, 64, 32 and 16 rows (a tile takes the smallest that holds its half)
  CUtensorMap tmWS;        // e4m3: scale atoms of the weights, rows of 128 x u32
  CUtensorMap tmXS;        // e4m3: scale atoms of the tokens, [tile][K block][atoms per tile]
  const int32_t* row0;     // [El + 1] first row of every expert
  const int32_t* tiles;    // [El + 1] first token tile of every expert
  const int32_t* pairs;    // stage 2: (token, k) pair of every row
  uint8_t* out;            // stage 1: H [capacity, F]; stage 2: [pairs, D] 16-bit
  uint8_t* out_sf;         // e4m3 stage 1: scale atoms of H
  int32_t* status;
  int El, tiles_w, kblocks, capacity;
  int ldo;                 // elements per row of out
};

template <int kStage_, bool kFp8_, int kMaxN_>
struct ExpertCfg {
  static constexpr int kStage = kStage_, kMaxN = kMaxN_;
  static constexpr bool kFp8 = kFp8_, kQuant = kFp8_ && kStage_ == 1;
  static constexpr int kBKE = kFp8_ ? 128 : 64;                        // K elements per stage: 128 bytes of a row
  static constexpr int kWBytes = 128 * 128, kXBytes = kMaxN_ / 2 * 128;
  static constexpr int kAtoms = kFp8_ ? (kMaxN_ + 127) / 128 : 0;
  static constexpr int kSfBytes = kFp8_ ? 512 * (1 + kAtoms) : 0;
  static constexpr int kStageBytes = kWBytes + kXBytes;
  static constexpr int kSetCols = 4 + 4 * kAtoms;                      // scale cells of one K block; two sets alternate
  static constexpr int kSfCol = 2 * kMaxN_;
  static constexpr int kUsedCols = 2 * kMaxN_ + (kFp8_ ? 2 * kSetCols : 0);
  static constexpr int kTmemCols = kUsedCols <= 128 ? 128 : kUsedCols <= 256 ? 256 : 512;
  // staging: e4m3 stage 1 keeps the tile's H values [token][64 features] and three arrays of magnitudes, else 2 KB per warp
  static constexpr int kEpiBytes = kQuant ? kMaxN_ * 128 + 3 * kMaxN_ * 4 : kXEpiWarps * 2048;
  static constexpr int kTabBytes = 2 * (kExpertMax + 4) * 4;
  static constexpr int kFree = 227 * 1024 - 1024 - kEpiBytes - kTabBytes - 512;
  static constexpr int kFit = kFree / (kStageBytes + kSfBytes);
  static constexpr int kStages = kFit > 10 ? 10 : kFit;
  static constexpr int kSmemBytes = 1024 + kStages * (kStageBytes + kSfBytes) + kEpiBytes + kTabBytes + 512;
  static_assert(kMaxN_ % 16 == 0 && kMaxN_ <= 256 && kUsedCols <= 512 && kXBytes % 1024 == 0 && kStages >= 4, "expert tile");
};

// Token tiles an expert of `rows` rows is cut into, and the rows of each: equal shares rounded up to 16.
__host__ __device__ __forceinline__ int expert_tiles(int rows, int max_n) { return (rows + max_n - 1) / max_n; }
__host__ __device__ __forceinline__ int expert_tile_rows(int rows, int tiles) { return ((rows + tiles - 1) / tiles + 15) & ~15; }

// Byte offset of row `r`'s cell inside a tile's scale atoms of one K block (row r of an atom at (r % 32) * 16 + (r / 32) * 4).
__device__ __forceinline__ int sf_cell(int r) { return (r >> 7) * 512 + (r & 31) * 16 + ((r >> 5) & 3) * 4; }

struct ExpertTile {
  int e, w, tile;      // expert, weight tile, token tile (counted over all experts)
  int row, cnt, n;     // first row, rows, rows padded to 16
};

// Unit t of the walk: experts in order, in an expert the token tiles of one weight tile next to each other (they read the
// same weights at about the same time). Asked by a whole converged warp.
__device__ __forceinline__ ExpertTile expert_unit(const int32_t* s_tiles, const int32_t* s_row0, int El, int tiles_w, int t) {
  const int lane = threadIdx.x & 31, tt = t / tiles_w;
  int e = 0;
  for (int base = 0; base + 1 < El; base += 32) {
    const int i = base + lane;
    const int n = __popc(__ballot_sync(0xffffffffu, i + 1 < El && s_tiles[i + 1] <= tt));
    e += n;
    if (n < 32) break;
  }
  ExpertTile u;
  u.e = e;
  const int first = s_tiles[e], nt = s_tiles[e + 1] - first, local = t - first * tiles_w, rows = s_row0[e + 1] - s_row0[e];
  u.w = local / nt;
  const int i = local - u.w * nt, per = expert_tile_rows(rows, nt);
  u.tile = first + i;
  u.row = s_row0[e] + i * per;
  u.cnt = min(per, rows - i * per);
  u.n = (u.cnt + 15) & ~15;
  return u;
}

template <class Cfg>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kXThreads, 1) expert_gemm_kernel(const __grid_constant__ ExpertArgs g) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kStages = Cfg::kStages, kStage = Cfg::kStage, kMaxN = Cfg::kMaxN;
  constexpr bool kFp8 = Cfg::kFp8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = ptx::cluster_ctarank();
  const bool leader = cta == 0;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sf_base = smem + kStages * Cfg::kStageBytes;
  uint8_t* epi = sf_base + kStages * Cfg::kSfBytes;
  int32_t* s_tiles = (int32_t*)(epi + Cfg::kEpiBytes);
  int32_t* s_row0 = s_tiles + kExpertMax + 4;
  uint64_t* full = (uint64_t*)(s_row0 + kExpertMax + 4);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;      // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2] in the even CTA: the epilogue warps of both
  uint64_t* peer_max = acc_empty + 2;        // [2] e4m3 stage 1: the peer's magnitudes have arrived
  uint32_t* tmem_slot = (uint32_t*)(peer_max + 2);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { ptx::mbar_init(&full[s], 1); ptx::mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(&acc_full[b], 1);
      ptx::mbar_init(&acc_empty[b], 2 * kXEpiWarps);
      ptx::mbar_init(&peer_max[b], 1);
    }
    ptx::fence_mbar_init();
    ptx::fence_proxy_async();
  }
  // (in front of pdl_wait: the kernel in front is the gather, which has no tensor memory and triggered when all kernels before it had completed,
  // or stage 1, which triggered when it had its columns. Behind it: 64 tokens, 32 experts, e4m3 236 -> 240 us)
  if (warp == 1) {
    ptx::tmem_alloc_pair(tmem_slot, Cfg::kTmemCols);
    ptx::tmem_relinquish_pair();
  }
  for (int i = threadIdx.x; i <= g.El; i += kXThreads) { s_tiles[i] = __ldcg(g.tiles + i); s_row0[i] = __ldcg(g.row0 + i); }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  // Launched behind the gather (stage 1) or stage 1 (stage 2). What is read before pdl_wait - the weights and the tables of
  // the preparation - was complete when the gather triggered, without which neither stage starts (launch_pdl.cuh).
  ptx::pdl_trigger();
  const int units = s_tiles[g.El] * g.tiles_w, first = blockIdx.x >> 1, step = gridDim.x >> 1;
  auto fail = [&]() { if (g.status) atomicCAS(g.status, 0, (int)kTimeoutPipeline); };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    const uint32_t stage0 = ptx::smem_u32(smem), sf0 = ptx::smem_u32(sf_base);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = first; t < units && ok; t += step) {
      const ExpertTile u = expert_unit(s_tiles, s_row0, g.El, g.tiles_w, t);
      const int half = u.n >> 1;
      const int box = half <= 16 ? 3 : half <= 32 ? 2 : half <= 64 ? 1 : 0;
      const CUtensorMap* mx = &g.tmX[box];
      const uint32_t x_bytes = (box == 0 ? kMaxN / 2 : 128 >> box) * 128;
      const uint32_t bytes = 2 * (Cfg::kWBytes + Cfg::kSfBytes + x_bytes);
      const int xrow = u.row + (int)cta * half;
      const int wblk = u.e * g.tiles_w + u.w;
      auto load_w = [&](int s, int kb) {
        const uint32_t sw = stage0 + s * Cfg::kStageBytes;
        if (leader) ptx::mbar_expect_tx_elect(&full[s], bytes);
        if constexpr (kStage == 1) {
#pragma unroll
          for (int i = 0; i < 4; ++i)          // 16 gate rows and their 16 up rows, one warp's lanes of the accumulator
            ptx::tma_load_3d_pair_elect(sw + i * 4096, &g.tmW, &full[s], kb * Cfg::kBKE, (int)cta * 64 + i * 16, 2 * wblk);
        } else {
          ptx::tma_load_2d_pair_elect(sw, &g.tmW, &full[s], kb * Cfg::kBKE, wblk * 256 + (int)cta * 128);
        }
        // stage 1: both CTAs hold the same interleaved rows' scales, one atom per block; stage 2: one atom per 128 rows
        if constexpr (kFp8)
          ptx::tma_load_2d_pair_elect(sf0 + s * Cfg::kSfBytes, &g.tmWS, &full[s], 0,
                                      kStage == 1 ? wblk * g.kblocks + kb : (wblk * g.kblocks + kb) * 2 + (int)cta);
      };
      auto load_x = [&](int s, int kb) {
        ptx::tma_load_2d_pair_elect(stage0 + s * Cfg::kStageBytes + Cfg::kWBytes, mx, &full[s], kb * Cfg::kBKE, xrow);
        if constexpr (kFp8)
          ptx::tma_load_2d_pair_elect(sf0 + s * Cfg::kSfBytes + 512, &g.tmXS, &full[s], 0, (u.tile * g.kblocks + kb) * Cfg::kAtoms);
      };
      int kb = 0;
      if (t == first) {                        // the ring fills with weights while the kernel in front finishes
        const int pre = min(kStages, g.kblocks);
        for (int i = 0; i < pre; ++i) load_w(i, i);
        ptx::pdl_wait();
        for (int i = 0; i < pre; ++i) load_x(i, i);
        kb = pre;
        if (pre == kStages) ph ^= 1;
        else s = pre;
      }
      for (; kb < g.kblocks; ++kb) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait<true>(&empty[s], ph ^ 1, kPipeTimeoutNs))) { fail(); ok = false; break; }
        load_w(s, kb);
        load_x(s, kb);
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (even CTA)
    const uint32_t tmem_u = __reduce_or_sync(0xffffffffu, tmem_base);
    const uint32_t stage0 = ptx::smem_u32(smem), sf0 = ptx::smem_u32(sf_base);
    int s = 0, it = 0;
    uint32_t ph = 0;
    bool ok = leader;
    for (int t = first; t < units && ok; t += step, ++it) {
      const ExpertTile u = expert_unit(s_tiles, s_row0, g.El, g.tiles_w, t);
      const int n = __shfl_sync(0xffffffffu, u.n, 0);
      const int buf = it & 1;
      if (!__all_sync(0xffffffffu, ptx::mbar_wait<true>(&acc_empty[buf], ((it >> 1) & 1) ^ 1, kPipeTimeoutNs))) { fail(); break; }
      ptx::tc_fence_after();
      const uint32_t d = tmem_u + buf * kMaxN;
      const uint32_t idesc = make_idesc(n, true, false, 2 * kBM);
      for (int kb = 0; kb < g.kblocks; ++kb) {
        if (!__all_sync(0xffffffffu, ptx::mbar_wait<true>(&full[s], ph, kPipeTimeoutNs))) { fail(); ok = false; break; }
        ptx::tc_fence_after();
        const uint32_t sw = stage0 + s * Cfg::kStageBytes, sx = sw + Cfg::kWBytes;
        if constexpr (kFp8) {
          const uint32_t ss = sf0 + s * Cfg::kSfBytes;
          const uint32_t t_sfw = tmem_u + Cfg::kSfCol + (kb & 1) * Cfg::kSetCols, t_sfx = t_sfw + 4;
          ptx::tmem_cp_sf_pair_elect(t_sfw, desc_sf(ss));
          ptx::tmem_cp_sf_pair_elect(t_sfx, desc_sf(ss + 512));
          if (Cfg::kAtoms == 2 && n > 128) ptx::tmem_cp_sf_pair_elect(t_sfx + 4, desc_sf(ss + 1024));
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ptx::mma_mxf8_pair_elect(d, desc_kmajor(sw + k * 32), desc_kmajor(sx + k * 32), make_idesc_mxf8(n, 2 * kBM, (uint32_t)k), (kb | k) != 0,
                                     t_sfw, t_sfx);
        } else {
#pragma unroll
          for (int k = 0; k < kBK / kUmmaK; ++k)
            ptx::mma_f16_pair_elect(d, desc_kmajor(sw + k * (kUmmaK * 2)), desc_kmajor(sx + k * (kUmmaK * 2)), idesc, (kb | k) != 0);
        }
        ptx::mma_commit_pair_elect(&empty[s], 3);
        if (kb == g.kblocks - 1) ptx::mma_commit_pair_elect(&acc_full[buf], 3);
        if (++s == kStages) { s = 0; ph ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9)
    const int q = warp & 3, w8 = warp - 2;     // TMEM lanes [32 q, 32 q + 32)
    const int c_first = (w8 >> 2) * 32;        // and of those the 32-token chunks from here, every other one
    auto release_acc = [&](int buf) {
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (leader) ptx::mbar_arrive(&acc_empty[buf]);
        else ptx::mbar_arrive_cluster_tmem(&acc_empty[buf], 0);
      }
    };
    uint8_t* stage = epi + w8 * 2048;
    ptx::pdl_wait();
    bool live = true;                          // after a wait that ran out the tiles pass without work: barriers stay in step
    int it = 0;
    for (int t = first; t < units; t += step, ++it) {
      const int buf = it & 1;
      const ExpertTile u = expert_unit(s_tiles, s_row0, g.El, g.tiles_w, t);
      const int keep = min(u.cnt, g.capacity - u.row);      // rows to be stored
      int pr[4];                               // stage 2: the destinations of the chunks' tokens, fetched while the MMAs run
      if constexpr (kStage == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int tk = c_first + 64 * i + lane;
          pr[i] = tk < keep ? __ldcg(g.pairs + u.row + tk) : -1;
        }
      }
      if (live) {
        live = __all_sync(0xffffffffu, ptx::mbar_wait<true>(&acc_full[buf], (it >> 1) & 1, kPipeTimeoutNs));
        if (!live) fail();
      }
      ptx::tc_fence_after();
      const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * kMaxN;
      if (live && c_first >= u.n) release_acc(buf);
      for (int c = c_first; c < u.n && live; c += 64) {
        // lanes [0, 16) and [16, 32) of the quarter, as fragments: thread l has lanes l / 4 and l / 4 + 8 of each half, and of every
        // eight tokens the two at 2 (l % 4). (The last load may read allocated columns past the tile.)
        uint32_t lo[16], hi[16];
        ptx::tmem_ld_16x256_x4(t_addr + c, lo);
        ptx::tmem_ld_16x256_x4(t_addr + (16u << 16) + c, hi);
        ptx::tmem_ld_wait();
        if (c + 64 >= u.n) release_acc(buf);
        const int mrow = lane & 7, mat = lane >> 3;              // this thread's row of the stored matrices
        if constexpr (kStage == 1) {
          // gate (lo) and up (hi) of the same features and tokens. A row of padding holds anything; a zero or worse would send the warp through
          // the division's long way (4 tokens, 16 experts of 7168 x 512, e4m3: 8 % slower than with a fast division, 2.5 % with a one in its place).
          const int t0 = c + 2 * (lane & 3);
          uint32_t h[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float gv = t0 + 8 * (i >> 1) + e < u.cnt ? __uint_as_float(lo[2 * i + e]) : 1.f, uv = __uint_as_float(hi[2 * i + e]);
              v[e] = gv / (1.f + __expf(-gv)) * uv;
            }
            const __nv_bfloat162 p = __floats2bfloat162_rn(v[0], v[1]);
            h[i] = *(const uint32_t*)&p;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {                          // 16 tokens: matrices (token octet mat / 2, feature octet mat % 2)
            const int tk = 16 * i + 8 * (mat >> 1) + mrow, f = mat & 1;
            if constexpr (Cfg::kQuant) {
              // rows of 128 bytes, their 16-byte groups permuted by the token
              const int t = c + tk;
              const uint32_t dst = ptx::smem_u32(epi + t * 128 + (((q * 2 + f) ^ (t & 7)) * 16));
              if (c + 16 * i < kMaxN) ptx::stmatrix_x4_trans(dst, h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
            } else {
              ptx::stmatrix_x4_trans(ptx::smem_u32(stage + tk * 32 + ((f ^ ((tk >> 2) & 1)) * 16)), h[4 * i], h[4 * i + 1], h[4 * i + 2], h[4 * i + 3]);
            }
          }
          if constexpr (!Cfg::kQuant) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int tk = i * 16 + (lane >> 1), f = lane & 1;
              const uint4 v = *(const uint4*)(stage + tk * 32 + ((f ^ ((tk >> 2) & 1)) * 16));
              if (c + tk < keep) *(uint4*)(g.out + ((size_t)(u.row + c + tk) * g.ldo + u.w * 128 + cta * 64 + q * 16 + f * 8) * 2) = v;
            }
            __syncwarp();
          }
        } else {
          const int pc = c < 64 ? pr[0] : c < 128 ? pr[1] : c < 192 ? pr[2] : pr[3];
          auto pack = [](uint32_t a, uint32_t b) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
            return *(const uint32_t*)&p;
          };
#pragma unroll
          for (int i = 0; i < 4; ++i) {                          // 8 tokens: matrix = feature octet
            const int tk = 8 * i + mrow;
            ptx::stmatrix_x4_trans(ptx::smem_u32(stage + tk * 64 + ((mat ^ ((tk >> 1) & 3)) * 16)), pack(lo[4 * i], lo[4 * i + 1]),
                                   pack(lo[4 * i + 2], lo[4 * i + 3]), pack(hi[4 * i], hi[4 * i + 1]), pack(hi[4 * i + 2], hi[4 * i + 3]));
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int tk = i * 8 + (lane >> 2), f = lane & 3;
            const int p = __shfl_sync(0xffffffffu, pc, tk);
            const uint4 v = *(const uint4*)(stage + tk * 64 + ((f ^ ((tk >> 1) & 3)) * 16));
            if (p >= 0) *(uint4*)(g.out + ((size_t)p * g.ldo + u.w * 256 + cta * 128 + q * 32 + f * 8) * 2) = v;
          }
          __syncwarp();
        }
      }
      if constexpr (Cfg::kQuant) {
        // the tile's H values of this CTA's 64 features lie in shared memory: largest magnitude per token, the peer's
        // for the other 64, then values and scale. Eight lanes per token.
        float* own = (float*)(epi + kMaxN * 128);
        float* box = own + kMaxN + buf * kMaxN;            // written by the peer
        ptx::named_barrier(1, kXEpiWarps * 32);
        const int sub = lane & 7;
        auto group_of = [&](int tk) { return (const uint4*)(epi + tk * 128 + ((sub ^ (tk & 7)) * 16)); };
        if (live) {
          if (w8 == 0 && lane == 0) ptx::mbar_expect_tx(&peer_max[buf], u.n * 4);
          for (int tk = w8 * 4 + (lane >> 3); tk < u.n; tk += 4 * kXEpiWarps) {
            const uint4 v = *group_of(tk);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            float m = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f = __bfloat1622float2(*(const __nv_bfloat162*)&w[i]);
              m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (sub == 0) {
              own[tk] = m;
              ptx::st_async_f32(&box[tk], &peer_max[buf], cta ^ 1, m);
            }
          }
          live = __all_sync(0xffffffffu, ptx::mbar_wait<true>(&peer_max[buf], (it >> 1) & 1, kPipeTimeoutNs));
          if (!live) fail();
        }
        if (live) {
          __syncwarp();
          for (int tk = w8 * 4 + (lane >> 3); tk < keep; tk += 4 * kXEpiWarps) {
            const float m = fmaxf(own[tk], box[tk]);
            // the smallest power of two >= m / 448, from the bits
            const uint32_t mb = __float_as_uint(fmaxf(m, 1e-12f) * (1.0f / 448.0f));
            const int e8 = min(127, (int)(mb >> 23) - 127 + ((mb & 0x7fffffu) ? 1 : 0));
            const float inv = e8 == 127 ? 0x1p-127f : __uint_as_float((uint32_t)(127 - e8) << 23);
            const uint4 v = *group_of(tk);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            uint32_t o[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&w[2 * i]), b = __bfloat1622float2(*(const __nv_bfloat162*)&w[2 * i + 1]);
              o[i] = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(a.x * inv, a.y * inv), __NV_SATFINITE, __NV_E4M3) |
                     (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(b.x * inv, b.y * inv), __NV_SATFINITE, __NV_E4M3) << 16;
            }
            *(uint2*)(g.out + (size_t)(u.row + tk) * g.ldo + u.w * 128 + cta * 64 + sub * 8) = make_uint2(o[0], o[1]);
            if (sub == 0 && cta == 0)
              *(uint32_t*)(g.out_sf + (size_t)(u.tile * g.tiles_w + u.w) * (Cfg::kAtoms * 512) + sf_cell(tk)) = (uint32_t)(e8 + 127) * 0x01010101u;
          }
        }
        ptx::named_barrier(1, kXEpiWarps * 32);             // the values are read before the next tile's overwrite them
      }
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();
  ptx::tc_fence_after();
  if (warp == 1) ptx::tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
}

// Map over [2 * blocks][128][K] weight rows (a gate block of 128 rows, its up block, the next gate block ...): a box is one
// K slice of 16 gate rows and the 16 up rows that belong to them.
int make_gate_up_map(CUtensorMap* m, const void* base, bool fp8, uint64_t blocks, uint64_t K) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return -10;
  const uint64_t row = K * (fp8 ? 1 : 2);
  if (((uint64_t)base & 15) || (row & 15)) return -11;
  cuuint64_t dims[3] = {K, 128, 2 * blocks};
  cuuint64_t strides[2] = {row, 128 * row};
  cuuint32_t box[3] = {fp8 ? 128u : 64u, 16, 2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -12;
}

struct ExpertProblem {
  const void *w, *w_sf, *x, *x_sf;
  int N, K;                // weight rows per expert (2 F or D), K of the product
  int max_tiles;           // bound of the token tiles of all experts (e4m3)
};

template <class Cfg>
int launch_experts(ExpertArgs& a, const ExpertProblem& p, cudaStream_t stream) {
  const int dt = Cfg::kFp8 ? IRIS_F8E4M3 : IRIS_BF16;
  a.tiles_w = p.N / 256;
  a.kblocks = ceil_div(p.K, Cfg::kBKE);
  int r = Cfg::kStage == 1 ? make_gate_up_map(&a.tmW, p.w, Cfg::kFp8, (uint64_t)a.El * a.tiles_w, p.K)
                           : make_map(&a.tmW, p.w, dt, (uint64_t)a.El * p.N, p.K, p.K, Cfg::kBKE, 128);
  if (r) return r;
  for (int i = 0; i < 4; ++i)
    if ((r = make_map(&a.tmX[i], p.x, dt, a.capacity, p.K, p.K, Cfg::kBKE, i == 0 || (128 >> i) > Cfg::kMaxN / 2 ? Cfg::kMaxN / 2 : 128 >> i))) return r;
  if (Cfg::kFp8) {
    if ((r = make_sf_map(&a.tmWS, p.w_sf, (uint64_t)a.El * a.tiles_w * a.kblocks * (Cfg::kStage == 1 ? 1 : 2), 1))) return r;
    if ((r = make_sf_map(&a.tmXS, p.x_sf, (uint64_t)p.max_tiles * a.kblocks * Cfg::kAtoms, Cfg::kAtoms))) return r;
  }
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(expert_gemm_kernel<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) return -20;
    attr = true;
  }
  return launch_pdl(expert_gemm_kernel<Cfg>, dim3(sm_count() & ~1), kXThreads, Cfg::kSmemBytes, stream, a);
}

}  // namespace
