// Distributed flash-decode: one query token per sequence, the KV cache sharded along the sequence
// over the ranks (reference: examples/13_flash_decode/decode_kernels.py:141-415 and
// flash_decode_fused_layer.py:38-148).
//
//   1. splitk kernel  two CTAs per SM; the query heads of one KV head attend over a run of tiles of 64 positions of
//      the LOCAL KV shard, paged KV gathered through the block table, online softmax; writes a normalised
//      partial output and its log-sum-exp per run. The tiles of all (sequence, KV head) pairs form one list that
//      is cut into equal pieces, one per CTA, on the device, from the lengths: a CTA may end one pair and begin the next, a pair
//      may be spread over many CTAs. (With the same number of splits for every sequence, the CTAs of the longest
//      one finished last: 32 sequences of 8192 to 32768 positions, 640 us where the bytes take 404; now 427. One
//      sequence of 32768: 512 CTAs on 296 places; 53 us, now 32.)
//      K/V stream through a ring of swizzled shared-memory tiles; QK^T and PV run on tensor
//      cores with the query heads of the group as the M dimension (each K/V byte is read from HBM
//      exactly once; the kernel is bound by HBM bandwidth). Two ways of filling the ring: a
//      warp issuing TMA box loads per page through a tensor map over the cache (page sizes 8,
//      16, 32 or a multiple of 64; completion on an mbarrier per stage), or all threads issuing
//      16-byte cp.async copies (any page size).
//   2. exchange kernel (persistent): phase A combines the local splits of every (batch, head) and
//      stores (o, lse) into slot [my_rank] of every rank's gathered buffer, then raises that
//      rank's flag for (my_rank, batch, head) with release semantics; phase B waits (acquire,
//      bounded) for the flags of all source ranks and merges the W partials into the final output.
//      All pushes are issued before any wait, so ranks never wait on each other in a cycle; the
//      buffers are double-buffered by call parity and flags carry the call number, so nothing is
//      cleared between calls (the reference zeroes its flags and runs a host barrier per call). One rank has nothing
//      to exchange: a kernel of one block per (batch, head) folds the partials into the output.
// lse is kept in fp32 (the reference stores it in the fp16 payload).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <math.h>
#include <string.h>

#include <cuda.h>

#include "iris/host_api.h"
#include "iris/iris.cuh"
#include "iris/ptx.cuh"
#include "flash_decode_static.h"
#include "launch_pdl.cuh"
#include <stdio.h>
#include <mutex>
#include <type_traits>

using namespace iris;

namespace {

constexpr int kD = 128;            // head dimension
constexpr int kBlockN = 64;        // KV positions per pipeline stage
constexpr int kStages = 3;
constexpr int kWarps = 4;
constexpr int kRowBytes = kD * 2;  // one position of one head
constexpr int kTileBytes = kBlockN * kRowBytes;   // 16 KB per K or V tile
constexpr float kLog2e = 1.4426950408889634f;

struct DecodeArgs {
  alignas(64) CUtensorMap tmK;     // TMA path: 2-D maps over the caches seen as [num_blocks * page, Hkv * D],
  alignas(64) CUtensorMap tmV;     // box = 64 columns (128 bytes, swizzled) x box_rows positions
  int box_rows;                    // min(page, 64)
  int32_t* status;                 // context status word (a TMA wait that runs out is recorded there)
  const __nv_bfloat16* q;          // [B, Hq, D]
  const __nv_bfloat16* k_cache;    // [num_blocks, page, Hkv, D]
  const __nv_bfloat16* v_cache;
  const int32_t* block_table;      // [B, max_blocks]
  const int32_t* kv_lens;          // [B] local lengths
  float* partial;                  // [B, Hq, splits, D + 1]  (o normalised, lse in log2 units; -inf in places that no run fills)
  int B, Hq, Hkv, page, max_blocks, group, head_groups;
  int splits;                      // places for partial results per (sequence, head)
  float sm_scale, soft_cap;
  int is_fp16;
};

__device__ __forceinline__ void cp_async16(uint32_t smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
template <bool kFp16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kFp16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool kFp16> __device__ __forceinline__ uint32_t pack2(float a, float b) {
  if constexpr (kFp16) { __half2 h = __floats2half2_rn(a, b); return *(uint32_t*)&h; }
  else { __nv_bfloat162 h = __floats2bfloat162_rn(a, b); return *(uint32_t*)&h; }
}

template <bool kFp16> __device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (kFp16) return __half22float2(*(const __half2*)&w);
  else return __bfloat1622float2(*(const __nv_bfloat162*)&w);
}

// Shared-memory tile of kBlockN positions x 16 chunks of 16 B.
// cp.async path: [position][16 chunks], chunk index XOR-swizzled by row & 7.
// TMA path: two halves of the head dimension, each [position][128 bytes] in the 128-byte swizzle
// TMA writes (chunk index within the half XOR row & 7; tiles are 1024-byte aligned).
template <bool kTma>
__device__ __forceinline__ uint32_t tile_off(int row, int chunk) {
  if constexpr (kTma) return (chunk >> 3) * (kBlockN * 128) + row * 128 + (((chunk & 7) ^ (row & 7)) << 4);
  else return row * kRowBytes + ((chunk ^ (row & 7)) << 4);
}

constexpr uint64_t kTmaWaitNs = 2000000000ull;
constexpr int kMaxSeqs = 1024;     // sequences of one launch (the tile list's prefix sums lie in shared memory)
constexpr int kMinRun = 4;         // tiles a CTA takes at least
constexpr int kRingBytes = kStages * 2 * kTileBytes;
static_assert(kWarps * 16 * kD * (int)sizeof(float) == 2 * kTileBytes, "a run's end uses one stage as scratch");
// ring, stage barriers, the warps' row maxima and sums, prefix sums
constexpr int kDecodeSmem = kRingBytes + 64 + kWarps * 16 * 2 * 4 + (kMaxSeqs + 2) * 4;
constexpr int kDecodeSmemTma = kDecodeSmem + 1024;      // alignment slack

// One run: tiles [t_first, t_first + n_tiles) of one (sequence, KV head, group of up to 16 query heads).
struct Run {
  int b, kvh, h0, heads_here, t_first, n_tiles, slot, n_slots, lo, hi;
};
// The CTA's runs (see the head of this file); every role walks the same list.
struct RunList {
  const DecodeArgs& a;
  const int* pre;               // [B + 1] tiles in front of sequence b, then the longest sequence's
  int heads_kv, per, flat, flat_end, whole;
  __device__ RunList(const DecodeArgs& a_, const int* pre_) : a(a_), pre(pre_) {
    heads_kv = a.Hkv * a.head_groups;
    const int total = pre[a.B] * heads_kv, longest = pre[a.B + 1];
    // tiles per CTA: an equal share, but not a handful, and no pair cut into more runs than there are places
    per = max(kMinRun, (total + (int)gridDim.x - 1) / (int)gridDim.x);
    if (a.splits > 1) per = max(per, (longest - 1 + a.splits - 2) / (a.splits - 1));
    flat = min(total, (int)blockIdx.x * per);
    flat_end = min(total, flat + per);
    whole = blockIdx.x;         // with one place per pair whole pairs are handed out instead
  }
  __device__ bool next(Run& r) {
    int x;
    if (a.splits > 1) {
      if (flat >= flat_end) return false;
      const int u = flat / heads_kv;                     // lies in the sequence's [pre[b], pre[b + 1])
      int lo_b = 0, hi_b = a.B - 1;
      while (lo_b < hi_b) {
        const int mid = (lo_b + hi_b + 1) >> 1;
        if (pre[mid] <= u) lo_b = mid; else hi_b = mid - 1;
      }
      r.b = lo_b;
      const int n_b = pre[r.b + 1] - pre[r.b], rem = flat - pre[r.b] * heads_kv;
      x = rem / n_b;
      r.t_first = rem - x * n_b;
      r.n_tiles = min(n_b - r.t_first, flat_end - flat);
      const int pair0 = flat - r.t_first;                // first tile of the pair in the list
      r.slot = blockIdx.x - pair0 / per;
      r.n_slots = (pair0 + n_b - 1) / per - pair0 / per + 1;
      flat += r.n_tiles;
    } else {
      if (whole >= a.B * heads_kv) return false;
      r.b = whole / heads_kv;
      x = whole - r.b * heads_kv;
      r.t_first = 0;
      r.n_tiles = pre[r.b + 1] - pre[r.b];
      r.slot = 0; r.n_slots = 1;
      whole += gridDim.x;
    }
    r.kvh = x / a.head_groups;
    const int hg = x - r.kvh * a.head_groups;
    r.heads_here = min(16, a.group - hg * 16);
    r.h0 = r.kvh * a.group + hg * 16;
    r.lo = r.t_first * kBlockN;
    r.hi = min(a.kv_lens[r.b], r.lo + r.n_tiles * kBlockN);
    return true;
  }
};
// One warp: the prefix sums. A sequence without positions still takes one (empty) tile: somebody has to write its result.
__device__ __forceinline__ void prefix_tiles(const DecodeArgs& a, int* pre, int lane) {
  int carry = 0, longest = 0;
  for (int base = 0; base < a.B; base += 32) {
    const int n = base + lane < a.B ? max(1, (a.kv_lens[base + lane] + kBlockN - 1) / kBlockN) : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (base + lane < a.B) pre[base + lane + 1] = carry + incl;
    carry += __shfl_sync(0xffffffffu, incl, 31);
    longest = max(longest, __reduce_max_sync(0xffffffffu, n));
  }
  if (lane == 0) { pre[0] = 0; pre[a.B + 1] = longest; }
}

// Attention state of one of the four computing warps: up to 16 query heads (rows) against the warp's 16 positions of
// each tile.
// P V is taken with P as two 16-bit numbers, its rounded value and the remainder: rounded once, P's error is as large as the output's
// own rounding, and more so the longer the runs are (only a run's largest weight is exact; 32 sequences of 8192 to 32768 positions, bf16,
// 2-norm against 64 bits: 2.21e-3 with the shorter runs of a fixed number of splits, 2.24e-3 with these, 1.65e-3 with the remainder).
// kRows8 (groups of up to 8 query heads): the remainders are rows 8 to 15 of the same MMA, which are padding otherwise, and the softmax
// skips those rows (32768 positions, 64 / 8 heads 39.1 -> 38.0 us). Wider groups take a second MMA (64 / 4 heads: 32 sequences by TMA
// 215 -> 216 us, one 42.6 -> 43.6; 16 sequences by cp.async, 32 / 2 heads, 95 -> 99).
template <bool kFp16, bool kTma, bool kRows8>
struct Attend {
  static constexpr int kE = kRows8 ? 2 : 4, kR = kRows8 ? 1 : 2;       // values per fragment and rows that a lane has
  uint32_t qf[8][4];             // Q fragments (A operand, rows = heads, padded to 16 with zeros)
  float o[16][4], m_run[2], l_run[2];

  __device__ __forceinline__ void begin(const DecodeArgs& a, const Run& r, int lane) {
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
    const uint32_t* qrow0 = (const uint32_t*)(a.q + ((size_t)r.b * a.Hq + r.h0 + r0) * kD);
    const uint32_t* qrow1 = (const uint32_t*)(a.q + ((size_t)r.b * a.Hq + r.h0 + r0 + 8) * kD);
    const bool v0 = r0 < r.heads_here, v1 = !kRows8 && r0 + 8 < r.heads_here;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const int c = (ks * 16 + c0) >> 1;
      qf[ks][0] = v0 ? qrow0[c] : 0u;
      qf[ks][1] = v1 ? qrow1[c] : 0u;
      qf[ks][2] = v0 ? qrow0[c + 4] : 0u;
      qf[ks][3] = v1 ? qrow1[c + 4] : 0u;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    m_run[0] = m_run[1] = -INFINITY;
    l_run[0] = l_run[1] = 0.f;
  }
  // ks, vs: shared-memory addresses of the K and V tile; pos0: position of the tile's first row
  __device__ __forceinline__ void tile(const DecodeArgs& a, uint32_t ks, uint32_t vs, int pos0, int hi, int warp, int lane) {
    const float scale2 = a.sm_scale * kLog2e;
    const int p0 = warp * 16;   // this warp's 16 positions of the tile
    // ---- S = Q K^T for 16 heads x 16 positions
    float s[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      uint32_t kf[4];
      const int j = lane >> 3, r = lane & 7;
      ldmatrix_x4(kf, ks + tile_off<kTma>(p0 + (j >> 1) * 8 + r, kk * 2 + (j & 1)));
      mma16816<kFp16>(s[0], qf[kk], kf[0], kf[1]);
      mma16816<kFp16>(s[1], qf[kk], kf[2], kf[3]);
    }
    // ---- online softmax (rows lane/4 and lane/4 + 8; columns: nb * 8 + (lane % 4) * 2 + {0, 1})
    const int pos_base = pos0 + p0 + (lane & 3) * 2;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nb = 0; nb < 2; ++nb)
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        float v = s[nb][e] * scale2;
        if (a.soft_cap > 0.f) v = a.soft_cap * kLog2e * tanhf(s[nb][e] * a.sm_scale / a.soft_cap);
        const int pos = pos_base + nb * 8 + (e & 1);
        v = pos < hi ? v : -INFINITY;
        s[nb][e] = v;
        mx[e >> 1] = fmaxf(mx[e >> 1], v);
      }
    float alpha[2];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
      mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
      const float m_new = fmaxf(m_run[r], mx[r]);
      alpha[r] = m_new == -INFINITY ? 1.f : exp2f(m_run[r] - m_new);
      m_run[r] = m_new;
    }
    float rs[2] = {0.f, 0.f};
    uint32_t pf[4], pl[4];
#pragma unroll
    for (int nb = 0; nb < 2; ++nb) {
      float p[4];
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        const float mr = m_run[e >> 1];
        p[e] = mr == -INFINITY ? 0.f : exp2f(s[nb][e] - mr);
        rs[e >> 1] += p[e];
      }
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        pf[nb * 2 + r] = pack2<kFp16>(p[2 * r], p[2 * r + 1]);
        const float2 f = unpack2<kFp16>(pf[nb * 2 + r]);
        (kRows8 ? pf[nb * 2 + 1] : pl[nb * 2 + r]) = pack2<kFp16>(p[2 * r] - f.x, p[2 * r + 1] - f.y);
      }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      rs[r] += __shfl_xor_sync(0xffffffffu, rs[r], 1);
      rs[r] += __shfl_xor_sync(0xffffffffu, rs[r], 2);
      l_run[r] = l_run[r] * alpha[r] + rs[r];
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      o[i][0] *= alpha[0]; o[i][1] *= alpha[0];
      o[i][2] *= alpha[kR - 1]; o[i][3] *= alpha[kR - 1];
    }
    // ---- O += P V   (A = P: 16 heads x 16 positions, B = V: 16 positions x 128 dims)
#pragma unroll
    for (int nb2 = 0; nb2 < 8; ++nb2) {
      uint32_t vf[4];
      const int j = lane >> 3, r = lane & 7;
      ldmatrix_x4_trans(vf, vs + tile_off<kTma>(p0 + (j & 1) * 8 + r, nb2 * 2 + (j >> 1)));
      mma16816<kFp16>(o[nb2 * 2], pf, vf[0], vf[1]);
      mma16816<kFp16>(o[nb2 * 2 + 1], pf, vf[2], vf[3]);
      if constexpr (!kRows8) {
        mma16816<kFp16>(o[nb2 * 2], pl, vf[0], vf[1]);
        mma16816<kFp16>(o[nb2 * 2 + 1], pl, vf[2], vf[3]);
      }
    }
  }
  // Merges the four warps (each saw a quarter of the positions) and writes the partial of the run (3 us at the end of every run while rows
  // stored met in one bank and every thread worked the weights out per value; with this and the fold below a sequence of 32768
  // positions 39.0 -> 32.1 us). `sm_o` is 32 KB that
  // nobody else uses, `sm_ml` 512 bytes; the computing warps' threads call it together (named barrier 1).
  __device__ __forceinline__ void finish(const DecodeArgs& a, const Run& run, float* sm_o, float* sm_ml, int warp, int lane) {
    // rows of 128 floats, the column XORed by the row times 8: eight rows stored and one row read meet different banks
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float* base = sm_o + (warp * 16) * kD + ((i * 8 + c0) ^ (r0 << 3));
      if constexpr (kRows8) {
        *(float2*)(base + r0 * kD) = make_float2(o[i][0] + o[i][2], o[i][1] + o[i][3]);
      } else {
        *(float2*)(base + r0 * kD) = make_float2(o[i][0], o[i][1]);
        *(float2*)(base + (r0 + 8) * kD) = make_float2(o[i][2], o[i][3]);
      }
    }
    if ((lane & 3) == 0) {
      sm_ml[(warp * 16 + r0) * 2] = m_run[0]; sm_ml[(warp * 16 + r0) * 2 + 1] = l_run[0];
      if constexpr (!kRows8) { sm_ml[(warp * 16 + r0 + 8) * 2] = m_run[1]; sm_ml[(warp * 16 + r0 + 8) * 2 + 1] = l_run[1]; }
    }
    ptx::named_barrier(1, kWarps * 32);
    const int tid = warp * 32 + lane;
    // a warp per head, four columns 32 apart per lane
#pragma unroll 2
    for (int h = warp; h < run.heads_here; h += kWarps) {
      float2 ml[kWarps];
      float m = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) { ml[w] = *(const float2*)(sm_ml + (w * 16 + h) * 2); m = fmaxf(m, ml[w].x); }
      float l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float sc = ml[w].x == -INFINITY ? 0.f : exp2f(ml[w].x - m);
        l += ml[w].y * sc;
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j] += sm_o[(w * 16 + h) * kD + ((j * 32 + lane) ^ ((h & 7) << 3))] * sc;
      }
      float* dst = a.partial + (((size_t)run.b * a.Hq + run.h0 + h) * a.splits + run.slot) * (kD + 1);
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[j * 32 + lane] = l > 0.f ? acc[j] / l : 0.f;
      if (lane == 0) dst[kD] = l > 0.f ? m + log2f(l) : -INFINITY;
    }
    // the run that begins a pair marks the places no run fills
    const int spare = a.splits - run.n_slots;
    if (run.t_first == 0)
      for (int idx = tid; idx < run.heads_here * spare; idx += kWarps * 32) {
        const int h = idx / spare, s = run.n_slots + idx % spare;
        a.partial[(((size_t)run.b * a.Hq + run.h0 + h) * a.splits + s) * (kD + 1) + kD] = -INFINITY;
      }
    ptx::named_barrier(1, kWarps * 32);       // the scratch has been read
  }
};

// TMA fill. Warp 4 fetches: a lane per box (page piece, half of the head dimension, K or V) looks up its page and
// issues its load, so the four computing warps never wait for block-table lookups (with them in thread 0 of a computing warp, 16
// boxes per tile at a page size of 16 took longer than the tile's bytes). The computing warps wait for a tile and hand
// it back one by one, no barrier of the CTA per tile.
template <bool kFp16, bool kRows8>
__global__ void __launch_bounds__(kWarps * 32 + 32, 2) decode_splitk_tma_kernel(const __grid_constant__ DecodeArgs a) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t* full = (uint64_t*)(smem + kRingBytes);
  uint64_t* empty = full + kStages;
  float* sm_ml = (float*)(smem + kRingBytes + 64);
  int* pre = (int*)(smem + kRingBytes + 64 + kWarps * 16 * 2 * 4);
  if (threadIdx.x == 32) {
    for (int i = 0; i < kStages; ++i) { ptx::mbar_init(&full[i], 1); ptx::mbar_init(&empty[i], kWarps); }
    ptx::fence_mbar_init();
    ptx::fence_proxy_async();
  }
  // Launched behind the stream's last kernel, but it does not let the next one start early: with the fold's blocks on the SMs from
  // the start one sequence of 32768 positions took 41 us, with the launch latency alone hidden 36 (38 before).
  if (threadIdx.x >= kWarps * 32 && lane < 2) ptx::prefetch_tmap(lane ? &a.tmV : &a.tmK);
  ptx::pdl_wait();
  if (warp == 0) prefix_tiles(a, pre, lane);
  __syncthreads();
  RunList list(a, pre);
  Run run;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
  uint32_t it = 0;                           // tiles so far (ring position)
  auto fail = [&]() { if (a.status) atomicCAS(a.status, 0, (int)kTimeoutPipeline); };
  if (warp == kWarps) {
    while (list.next(run)) {
      const int32_t* bt = a.block_table + (size_t)run.b * a.max_blocks;
      const int j = lane >> 2, hf = (lane >> 1) & 1, is_v = lane & 1;
      for (int t = 0; t < run.n_tiles; ++t, ++it) {
        const int stage = it % kStages;
        const int pos0 = run.lo + t * kBlockN;
        const int rows = max(0, min(kBlockN, run.hi - pos0));
        const int nbox = (rows + a.box_rows - 1) / a.box_rows;
        const int pos = pos0 + j * a.box_rows;
        int y = 0;
        if (j < nbox) y = bt[pos / a.page] * a.page + pos % a.page;      // looked up before the stage is waited for
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&empty[stage], ((it / kStages) & 1) ^ 1, kTmaWaitNs))) { fail(); return; }
        if (lane == 0) ptx::mbar_expect_tx(&full[stage], (uint32_t)(nbox * a.box_rows * 128 * 4));
        __syncwarp();
        if (j < nbox)
          ptx::tma_load_2d(smem + stage * 2 * kTileBytes + is_v * kTileBytes + hf * (kBlockN * 128) + j * a.box_rows * 128,
                           is_v ? &a.tmV : &a.tmK, &full[stage], run.kvh * kD + hf * 64, y);
        __syncwarp();
      }
    }
    return;
  }
  Attend<kFp16, true, kRows8> at;
  bool dead = false;                         // a wait ran out (recorded): walk on without data, so that no warp waits at a barrier for this one
  while (list.next(run)) {
    at.begin(a, run, lane);
    for (int t = 0; t < run.n_tiles; ++t, ++it) {
      const int stage = it % kStages;
      if (!dead && !__all_sync(0xffffffffu, ptx::mbar_wait(&full[stage], (it / kStages) & 1, kTmaWaitNs))) { fail(); dead = true; }
      uint8_t* vt = smem + stage * 2 * kTileBytes + kTileBytes;
      const int rows = max(0, run.hi - (run.lo + t * kBlockN));
      if (rows < warp * 16 + 16) {
        // rows past the end hold whatever the page (or an older tile) held; their scores are masked, and this warp's V
        // rows among them are cleared so that 0 * NaN cannot arise
        for (int idx = lane; idx < 16 * 16; idx += 32) {
          const int row = warp * 16 + (idx >> 4), chunk = idx & 15;
          if (row >= rows) *(uint4*)(vt + tile_off<true>(row, chunk)) = make_uint4(0, 0, 0, 0);
        }
        ptx::fence_proxy_async_smem();       // before TMA writes the stage again
        __syncwarp();
      }
      const uint32_t ks = base + stage * 2 * kTileBytes;
      if (!dead) at.tile(a, ks, ks + kTileBytes, run.lo + t * kBlockN, run.hi, warp, lane);
      __syncwarp();
      // the last tile's stage serves as scratch first
      if (t + 1 < run.n_tiles && lane == 0) ptx::mbar_arrive(&empty[stage]);
    }
    const int last = (it - 1) % kStages;
    ptx::named_barrier(1, kWarps * 32);      // every warp has read the last tile
    at.finish(a, run, (float*)(smem + last * 2 * kTileBytes), sm_ml, warp, lane);
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&empty[last]);
  }
}

// cp.async fill by the computing threads themselves: any page size.
template <bool kFp16, bool kRows8>
__global__ void __launch_bounds__(kWarps * 32, 2) decode_splitk_kernel(const __grid_constant__ DecodeArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* sm_ml = (float*)(smem + kRingBytes + 64);
  int* pre = (int*)(smem + kRingBytes + 64 + kWarps * 16 * 2 * 4);
  ptx::pdl_wait();
  if (warp == 0) prefix_tiles(a, pre, lane);
  __syncthreads();
  RunList list(a, pre);
  Run run;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
  const size_t pos_stride = (size_t)a.Hkv * kD;   // elements between consecutive positions of a page
  Attend<kFp16, false, kRows8> at;
  while (list.next(run)) {
    const int32_t* bt = a.block_table + (size_t)run.b * a.max_blocks;
    auto issue_tile = [&](int t) {
      const int stage = t % kStages;
      const uint32_t ks = base + stage * 2 * kTileBytes, vs = ks + kTileBytes;
      // 64 rows x 16 chunks for K and for V = 2048 chunks, 128 threads -> 16 each
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int idx = threadIdx.x + i * 128;     // 0..1023
        const int row = idx >> 4, chunk = idx & 15;
        const int pos = run.lo + t * kBlockN + row;
        if (pos < run.hi) {
          const int blk = bt[pos / a.page];
          const size_t e = ((size_t)blk * a.page + pos % a.page) * pos_stride + (size_t)run.kvh * kD + chunk * 8;
          cp_async16(ks + tile_off<false>(row, chunk), a.k_cache + e);
          cp_async16(vs + tile_off<false>(row, chunk), a.v_cache + e);
        } else {
          *(uint4*)(smem + stage * 2 * kTileBytes + tile_off<false>(row, chunk)) = make_uint4(0, 0, 0, 0);
          *(uint4*)(smem + stage * 2 * kTileBytes + kTileBytes + tile_off<false>(row, chunk)) = make_uint4(0, 0, 0, 0);
        }
      }
    };
    at.begin(a, run, lane);
    for (int t = 0; t < kStages - 1; ++t) {
      if (t < run.n_tiles) issue_tile(t);
      cp_async_commit();
    }
    for (int t = 0; t < run.n_tiles; ++t) {
      cp_async_wait<kStages - 2>();
      __syncthreads();
      if (t + kStages - 1 < run.n_tiles) issue_tile(t + kStages - 1);
      cp_async_commit();
      const uint32_t ks = base + (t % kStages) * 2 * kTileBytes;
      at.tile(a, ks, ks + kTileBytes, run.lo + t * kBlockN, run.hi, warp, lane);
    }
    cp_async_wait<0>();
    __syncthreads();
    at.finish(a, run, (float*)smem, sm_ml, warp, lane);
  }
}

// Folds the partial results of one (sequence, head) into (o, lse), thread d taking dimension d, for the exchange across ranks and the entry
// point that allocates nothing (one rank: decode_local_finish_kernel). All of the block's
// threads call it; `s_w` is kD floats of shared memory. The weights are taken once, by a thread per place, and the loads
// of eight places are in flight together (two serial passes over 64 places took most of 24 us).
__device__ __forceinline__ void combine_splits(const float* p, int splits, float* s_w, float& o, float& lse) {
  const int d = threadIdx.x;
  __shared__ float s_m[kD / 32];
  float m = -INFINITY;
  for (int s = d; s < splits; s += kD) m = fmaxf(m, __ldcg(p + (size_t)s * (kD + 1) + kD));
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, k));
  __syncthreads();
  if ((d & 31) == 0) s_m[d >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kD / 32; ++w) m = fmaxf(m, s_m[w]);
  float l = 0.f, acc = 0.f;
  for (int s0 = 0; s0 < splits; s0 += kD) {
    const int n = min(kD, splits - s0);
    __syncthreads();
    if (d < n) {
      const float ls = __ldcg(p + (size_t)(s0 + d) * (kD + 1) + kD);
      s_w[d] = ls == -INFINITY ? 0.f : exp2f(ls - m);
    }
    __syncthreads();
    for (int s = 0; s < n; s += 8) {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = s + k < n && s_w[s + k] != 0.f ? __ldcg(p + (size_t)(s0 + s + k) * (kD + 1) + d) : 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (s + k < n) { l += s_w[s + k]; acc += s_w[s + k] * v[k]; }
    }
  }
  o = l > 0.f ? acc / l : 0.f;
  lse = l > 0.f ? m + log2f(l) : -INFINITY;
}

// ------------------------------------------------------------------------------ exchange + merge
struct ExchangeArgs {
  DeviceContext ctx;
  const float* partial;     // [B, Hq, splits, D+1]
  float* gathered;          // heap: [2][W][Bmax][Hq][D+1]
  int32_t* flags;           // heap: [2][W][Bmax][Hq]
  int32_t* state;           // heap: [0] call counter, [1] finished CTAs
  void* out;                // [B, Hq, D] 16-bit
  float* out_lse;           // optional [B, Hq] natural-log lse of the full attention
  int B, Bmax, Hq, splits;
  int is_fp16;
};

__global__ void __launch_bounds__(kD) decode_exchange_kernel(const __grid_constant__ ExchangeArgs a) {
  const DeviceContext& ctx = a.ctx;
  const int W = ctx.world;
  const int call = *(volatile int32_t*)&a.state[0];
  const int buf = call & 1;
  const int32_t tag = (call >> 1) + 1;
  const int items = a.B * a.Hq;
  const int d = threadIdx.x;
  __shared__ float s_w[64], s_part[kD];
  __shared__ int s_ok;
  // phase A: combine local splits, push to every rank
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int b = it / a.Hq, h = it - b * a.Hq;
    float o, lse;
    combine_splits(a.partial + (size_t)it * a.splits * (kD + 1), a.splits, s_part, o, lse);
    float* slot = a.gathered + ((((size_t)buf * W + ctx.rank) * a.Bmax + b) * a.Hq + h) * (kD + 1);
    int32_t* flag = a.flags + (((size_t)buf * W + ctx.rank) * a.Bmax + b) * a.Hq + h;
    for (int i = 0; i < W; ++i) {
      int r = ctx.rank + i;
      if (r >= W) r -= W;
      float* dst = ctx.remote(slot, r);
      dst[d] = o;
      if (d == 0) dst[kD] = lse;
    }
    __syncthreads();
    if (d < W) {
      int r = ctx.rank + d;
      if (r >= W) r -= W;
      fence_sys();
      st_release_sys(ctx.remote(flag, r), tag);
    }
  }
  // phase B: wait for every source rank, merge
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int b = it / a.Hq, h = it - b * a.Hq;
    if (d == 0) s_ok = 1;
    __syncthreads();
    if (d < W) {
      const int32_t* flag = a.flags + (((size_t)buf * W + d) * a.Bmax + b) * a.Hq + h;
      if (!wait_flag_ge(ctx, flag, tag)) s_ok = 0;
      const float* slot = a.gathered + ((((size_t)buf * W + d) * a.Bmax + b) * a.Hq + h) * (kD + 1);
      s_w[d] = __ldcv(slot + kD);
    }
    __syncthreads();
    if (!s_ok) break;
    float m = -INFINITY;
    for (int r = 0; r < W; ++r) m = fmaxf(m, s_w[r]);
    float l = 0.f, acc = 0.f;
    for (int r = 0; r < W; ++r) {
      const float w = s_w[r] == -INFINITY ? 0.f : exp2f(s_w[r] - m);
      const float* slot = a.gathered + ((((size_t)buf * W + r) * a.Bmax + b) * a.Hq + h) * (kD + 1);
      l += w;
      acc += w * __ldcv(slot + d);
    }
    const float o = l > 0.f ? acc / l : 0.f;
    if (a.is_fp16) ((__half*)a.out)[(size_t)it * kD + d] = __float2half_rn(o);
    else ((__nv_bfloat16*)a.out)[(size_t)it * kD + d] = __float2bfloat16_rn(o);
    if (a.out_lse && d == 0) a.out_lse[it] = l > 0.f ? (m + log2f(l)) / kLog2e : -INFINITY;
    __syncthreads();
  }
  __syncthreads();
  if (d == 0) {
    __threadfence();
    if (atomicAdd(&a.state[1], 1) == (int)gridDim.x - 1) {
      a.state[1] = 0;
      a.state[0] = call + 1;
      __threadfence();
    }
  }
}

// Finish without a peer: fold this rank's partials into (o, lse). With one rank that is the whole result; with
// exchange == 2 it is what a decode over a KV shard returns when the cross-rank merge is done elsewhere, e.g. by an
// all-gather of the partial results as in the reference's RCCL baseline
// (examples/benchmark/reference/flash_decode_rccl/flash_decode_layer_rccl.py:100-130).
// A block per (sequence, head); kGroups threads per column share its places, and a thread's loads are all in flight together: first the
// places' weights, then the values that have one. Few heads with many places wait for latency only (one sequence of 32768 positions, 64
// heads with 37 places each: 3.8 us with one thread per column and eight loads in flight); with many heads one
// thread per column reads what there is to read.
template <int kGroups, int kAhead>
__global__ void __launch_bounds__(kD * kGroups) decode_local_finish_kernel(const float* partial, void* out, float* out_lse, int splits, int is_fp16) {
  const int it = blockIdx.x, d = threadIdx.x % kD, g = threadIdx.x / kD;
  __shared__ float s_o[kGroups][kD];
  __shared__ float2 s_ml[kGroups];
  ptx::pdl_wait();                                         // the partials are complete from here on
  const float* p = partial + (size_t)it * splits * (kD + 1);
  float m = -INFINITY, l = 0.f, acc = 0.f;
  for (int s0 = g; s0 < splits; s0 += kGroups * kAhead) {
    float w[kAhead], v[kAhead], top = m;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const int s = s0 + k * kGroups;
      w[k] = s < splits ? __ldcg(p + (size_t)s * (kD + 1) + kD) : -INFINITY;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {                     // (a place that no run filled holds no numbers)
      v[k] = w[k] != -INFINITY ? __ldcg(p + (size_t)(s0 + k * kGroups) * (kD + 1) + d) : 0.f;
      top = fmaxf(top, w[k]);
    }
    if (top == -INFINITY) continue;
    // (a place whose weight vanishes counts nothing, whatever it holds: no zero is multiplied by an infinity)
    const float keep = exp2f(m - top);
    m = top; l *= keep; acc = keep * (keep != 0.f ? acc : 0.f);
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const float e = exp2f(w[k] - m);
      l += e; acc += e * (e != 0.f ? v[k] : 0.f);
    }
  }
  if constexpr (kGroups > 1) {
    s_o[g][d] = acc;
    if (d == 0) s_ml[g] = make_float2(m, l);
    __syncthreads();
    if (g) return;
    float top = -INFINITY;
#pragma unroll
    for (int k = 0; k < kGroups; ++k) top = fmaxf(top, s_ml[k].x);
    l = acc = 0.f;
#pragma unroll
    for (int k = 0; k < kGroups; ++k) {
      const float e = s_ml[k].x == -INFINITY ? 0.f : exp2f(s_ml[k].x - top);
      l += s_ml[k].y * e; acc += (e != 0.f ? s_o[k][d] : 0.f) * e;
    }
    m = top;
  }
  const float o = l > 0.f ? acc / l : 0.f;
  if (is_fp16) ((__half*)out)[(size_t)it * kD + d] = __float2half_rn(o);
  else ((__nv_bfloat16*)out)[(size_t)it * kD + d] = __float2bfloat16_rn(o);
  if (out_lse && d == 0) out_lse[it] = l > 0.f ? (m + log2f(l)) / kLog2e : -INFINITY;
}

int decode_sms() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// Split-K pass over `a.B` sequences, in launches of up to kMaxSeqs, on two CTAs per SM.
template <bool kTma>
int launch_splitk(DecodeArgs a, cudaStream_t s) {
  constexpr int smem = kTma ? kDecodeSmemTma : kDecodeSmem;
  auto pick = [&](auto fp16, auto rows8) -> void (*)(const DecodeArgs) {
    return kTma ? decode_splitk_tma_kernel<decltype(fp16)::value, decltype(rows8)::value>
                : decode_splitk_kernel<decltype(fp16)::value, decltype(rows8)::value>;
  };
  using Y = std::true_type;
  using N = std::false_type;
  auto* kern = a.is_fp16 ? (a.group <= 8 ? pick(Y{}, Y{}) : pick(Y{}, N{})) : (a.group <= 8 ? pick(N{}, Y{}) : pick(N{}, N{}));
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -20;
  const int sms = decode_sms();
  const int total = a.B;
  for (int b0 = 0; b0 < total; b0 += kMaxSeqs) {
    DecodeArgs p = a;
    p.B = total - b0 < kMaxSeqs ? total - b0 : kMaxSeqs;
    p.q = a.q + (size_t)b0 * a.Hq * kD;
    p.block_table = a.block_table + (size_t)b0 * a.max_blocks;
    p.kv_lens = a.kv_lens + b0;
    p.partial = a.partial + (size_t)b0 * a.Hq * a.splits * (kD + 1);
    if (const int r = launch_pdl(kern, dim3(2 * sms), kWarps * 32 + (kTma ? 32 : 0), smem, s, p)) return r;
  }
  return 0;
}

}  // namespace

extern "C" {

typedef struct IrisDecodeDesc {
  IrisCtx ctx;
  const void* q; const void* k_cache; const void* v_cache;
  const int32_t* block_table; const int32_t* kv_lens;
  float* partial;
  float* gathered; int32_t* flags; int32_t* state;
  void* out; float* out_lse;
  int32_t B, Bmax, Hq, Hkv, D, page, max_blocks, splits;
  float sm_scale, soft_cap;
  int32_t dtype;
  int32_t exchange;   // 0: only the local split-K pass, 1: also combine + exchange + merge, 2: combine locally (out, lse of this rank's shard)
  int32_t num_blocks; // pages in each cache tensor (0: unknown, the TMA path is not used)
} IrisDecodeDesc;

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// 2-D map over a cache seen as [num_blocks * page positions, Hkv * D] 16-bit elements.
bool make_cache_map(CUtensorMap* m, const void* base, int dtype, uint64_t positions, uint64_t row_elems, uint32_t box_rows) {
  static EncodeTiledFn enc = nullptr;
  if (!enc) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) return false;
    enc = (EncodeTiledFn)p;
  }
  if (((uint64_t)base & 15) || ((row_elems * 2) & 15)) return false;
  cuuint64_t dims[2] = {row_elems, positions};
  cuuint64_t strides[1] = {row_elems * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = dtype == IRIS_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  return enc(m, dt, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

int iris_flash_decode(const IrisDecodeDesc* d, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (d->D != kD) return -3;
  if (d->Hq % d->Hkv) return -3;
  if (d->dtype != IRIS_BF16 && d->dtype != IRIS_F16) return -2;
  DecodeArgs a;
  a.q = (const __nv_bfloat16*)d->q; a.k_cache = (const __nv_bfloat16*)d->k_cache; a.v_cache = (const __nv_bfloat16*)d->v_cache;
  a.block_table = d->block_table; a.kv_lens = d->kv_lens; a.partial = d->partial;
  a.B = d->B; a.Hq = d->Hq; a.Hkv = d->Hkv; a.page = d->page; a.max_blocks = d->max_blocks; a.splits = d->splits;
  a.group = d->Hq / d->Hkv; a.head_groups = (a.group + 15) / 16;
  a.sm_scale = d->sm_scale; a.soft_cap = d->soft_cap; a.is_fp16 = d->dtype == IRIS_F16;
  a.status = d->ctx.status; a.box_rows = 0;
  // TMA fill when a 64-position tile is a whole number of page pieces
  bool tma = d->num_blocks > 0 && (d->page == 8 || d->page == 16 || d->page == 32 || d->page % 64 == 0);
  if (tma) {
    a.box_rows = d->page < kBlockN ? d->page : kBlockN;
    const uint64_t positions = (uint64_t)d->num_blocks * d->page, row = (uint64_t)d->Hkv * kD;
    tma = make_cache_map(&a.tmK, d->k_cache, d->dtype, positions, row, a.box_rows) &&
          make_cache_map(&a.tmV, d->v_cache, d->dtype, positions, row, a.box_rows);
  }
  const int r = tma ? launch_splitk<true>(a, s) : launch_splitk<false>(a, s);
  if (r) return r;
  if (!d->exchange) return 0;
  if (d->exchange == 2 || d->ctx.world <= 1) {
    const int items = d->B * d->Hq;
    if (items <= 2 * decode_sms() && d->splits > 8)      // (few heads: see the kernel)
      return launch_pdl(decode_local_finish_kernel<4, 10>, dim3(items), 4 * kD, 0, s, (const float*)d->partial, d->out, d->out_lse, (int)d->splits, a.is_fp16);
    return launch_pdl(decode_local_finish_kernel<1, 8>, dim3(items), kD, 0, s, (const float*)d->partial, d->out, d->out_lse, (int)d->splits, a.is_fp16);
  }
  ExchangeArgs x;
  memcpy(&x.ctx, &d->ctx, sizeof(DeviceContext));
  if (x.ctx.world > 64) return -4;
  x.partial = d->partial; x.gathered = d->gathered; x.flags = d->flags; x.state = d->state;
  x.out = d->out; x.out_lse = d->out_lse; x.B = d->B; x.Bmax = d->Bmax; x.Hq = d->Hq; x.splits = d->splits;
  x.is_fp16 = a.is_fp16;
  int items = d->B * d->Hq;
  const int most = 8 * decode_sms();
  int grid2 = items < most ? items : most;         // every CTA resident: pushes precede all waits anyway
  decode_exchange_kernel<<<grid2, kD, 0, s>>>(x);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // extern "C"

// ------------------------------------------------------------------ entry point that allocates nothing
// See flash_decode_static.h. The split-K kernel above is launched unchanged with its partial
// results directed into the file-scope array below; a small kernel then folds the splits into
// the output. Host code never uses `g_decode_static_scratch` as an address: the name is only a
// handle on the host side, the device address comes from cudaGetSymbolAddress.
namespace {

static __device__ __align__(256) unsigned char g_decode_static_scratch[IRIS_DECODE_STATIC_SCRATCH_BYTES];

constexpr int kStaticMaxDevices = 64;
float* g_static_scratch_addr[kStaticMaxDevices] = {};
std::mutex g_static_setup_mutex;

__global__ void __launch_bounds__(kD) decode_local_combine_kernel(const float* partial, void* out, int splits, int is_fp16) {
  const int it = blockIdx.x, d = threadIdx.x;
  __shared__ float s_part[kD];
  float o, lse;
  combine_splits(partial + (size_t)it * splits * (kD + 1), splits, s_part, o, lse);
  if (is_fp16) ((__half*)out)[(size_t)it * kD + d] = __float2half_rn(o);
  else ((__nv_bfloat16*)out)[(size_t)it * kD + d] = __float2bfloat16_rn(o);
}

void static_err(char* err, int32_t errlen, const char* msg) {
  if (err && errlen > 0) snprintf(err, (size_t)errlen, "%s", msg);
}

}  // namespace

extern "C" uint64_t iris_flash_decode_static_scratch_needed(int32_t B, int32_t Hq, int32_t splits, int32_t D) {
  return (uint64_t)B * (uint64_t)Hq * (uint64_t)splits * (uint64_t)(D + 1);
}

extern "C" int iris_flash_decode_static(const void* q, const void* k_cache, const void* v_cache, const int32_t* block_table,
                                        const int32_t* kv_lens, void* out, int32_t B, int32_t Hq, int32_t Hkv, int32_t D,
                                        int32_t page, int32_t max_blocks, int32_t splits, float sm_scale, float soft_cap,
                                        int32_t dtype, void* stream, char* err, int32_t errlen) {
  cudaStream_t s = (cudaStream_t)stream;
  if (D != kD || Hkv <= 0 || Hq % Hkv || B <= 0 || splits <= 0 || page <= 0) {
    static_err(err, errlen, "iris_flash_decode_static: head_dim must be 128, q_heads a multiple of kv_heads, sizes positive");
    return -3;
  }
  if (dtype != IRIS_BF16 && dtype != IRIS_F16) {
    static_err(err, errlen, "iris_flash_decode_static: dtype must be fp16 (0) or bf16 (1)");
    return -2;
  }
  const uint64_t need = iris_flash_decode_static_scratch_needed(B, Hq, splits, D) * sizeof(float);
  if (need > IRIS_DECODE_STATIC_SCRATCH_BYTES) {
    char msg[256];
    snprintf(msg, sizeof(msg),
             "iris_flash_decode_static: batch %d x q_heads %d x splits %d needs %llu bytes of scratch, the built-in array holds %u; "
             "lower splits or call iris_flash_decode with your own buffer",
             B, Hq, splits, (unsigned long long)need, IRIS_DECODE_STATIC_SCRATCH_BYTES);
    static_err(err, errlen, msg);
    return IRIS_DECODE_STATIC_TOO_LARGE;
  }
  // set-up, once per device: the array's address on the device that is current now
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kStaticMaxDevices) {
    static_err(err, errlen, "iris_flash_decode_static: no current CUDA device");
    return -4;
  }
  // The table below is per device: the array's address differs from GPU to GPU. One mutex covers the set-up, so
  // that two host threads making a device's first call agree.
  {
    std::lock_guard<std::mutex> guard(g_static_setup_mutex);
    if (!g_static_scratch_addr[dev]) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_decode_static_scratch);
      if (e != cudaSuccess || !p) {
        static_err(err, errlen, "iris_flash_decode_static: cudaGetSymbolAddress failed for the scratch array");
        return -5;
      }
      g_static_scratch_addr[dev] = (float*)p;
    }
  }
  float* scratch = g_static_scratch_addr[dev];

  DecodeArgs a;
  a.q = (const __nv_bfloat16*)q; a.k_cache = (const __nv_bfloat16*)k_cache; a.v_cache = (const __nv_bfloat16*)v_cache;
  a.block_table = block_table; a.kv_lens = kv_lens; a.partial = scratch;
  a.B = B; a.Hq = Hq; a.Hkv = Hkv; a.page = page; a.max_blocks = max_blocks; a.splits = splits;
  a.group = Hq / Hkv; a.head_groups = (a.group + 15) / 16;
  a.sm_scale = sm_scale; a.soft_cap = soft_cap; a.is_fp16 = dtype == IRIS_F16;
  a.status = nullptr; a.box_rows = 0;     // the cp.async instantiation: no tensor maps
  if (launch_splitk<false>(a, s)) {
    static_err(err, errlen, "iris_flash_decode_static: split-K kernel launch failed");
    return -21;
  }
  decode_local_combine_kernel<<<B * Hq, kD, 0, s>>>(scratch, out, splits, a.is_fp16);
  if (cudaGetLastError() != cudaSuccess) {
    static_err(err, errlen, "iris_flash_decode_static: combine kernel launch failed");
    return -21;
  }
  return 0;
}
