// Expert-sharded mixture-of-experts layer (reference: examples/31_expert_sharded_moe/*: topk.py,
// dispatch.py, grouped_matmul.py, fused_exp_matmul_ep_to_dp.py, combine.py, reduce.py).
//
// Launch sequence of one forward pass, all on one stream, no host round trips (the reference
// synchronises with .item() and a Python loop per expert, moe.py:262, ragged_metadata.py:52-78):
//   1 router     warp per token: top-k of the logits, softmax over the selected k, histogram
//   2 meta       one CTA: push this rank's expert histogram to every rank, cross-rank round, then
//                all offsets: where my rows for expert e start on e's owner, row range and tile
//                range of every local expert, expected arrivals
//   3 sort       (token, k) pairs bucketed by expert (list per expert)
//   4 dispatch + grouped GEMM 1 + SwiGLU, ONE kernel: communication CTAs walk the experts by local
//                index (so every rank's expert j fills up at the same time), stream each token row
//                HBM -> shared memory -> owner's inbox with bulk async copies and add the row
//                count to the owner's arrival counter for that expert; GEMM CTAs (tcgen05 main
//                loop) wait for an expert's arrivals, then multiply its rows by the expert's fused
//                gate|up weight and write silu(gate) * up
//                (the fusion the reference leaves as NotImplementedError, moe.py:285-286).
//                One rank: a gather kernel copies the rows into expert order first, and both grouped GEMMs are those
//                of moe_experts.cuh
//   5 grouped GEMM 2 + combine, ONE kernel: down projection whose epilogue stores every output row
//                straight into the (token, k) slot of the token's home rank; cross-rank round at exit
//   6 reduce     out[t] = sum_k weight[t, k] * slot[t, k]   (the reference's sum is unweighted)
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <math.h>
#include <string.h>

#include "gemm_host.cuh"
#include "quantize_common.cuh"
#include "moe_experts.cuh"

namespace {

constexpr int kMaxTopK = 16;
// One rank: token tiles of moe_experts.cuh. An expert has at most T rows, so up to 64 tokens every expert is one tile, and the
// smaller stages make a deeper ring; e4m3 needs TMEM columns for its scale cells, so its widest tile is 240.
constexpr int kSmallTokens = 64, kTile16 = 256, kTileFp8 = 240;

struct MoeDims {
  int T, K, E, El, D, F, capacity;
  int tile_rows;           // most rows of a token tile
};

// Device-resident metadata of one layer (all int32 unless noted; "heap" = symmetric heap).
struct MoeMeta {
  int32_t* topk_idx;       // [T, K]
  float* topk_w;           // [T, K]
  int32_t* counts_local;   // [E]      my tokens per expert
  int32_t* counts_all;     // heap [W, E]
  int32_t* cursor;         // [E]
  int32_t* list_off;       // [E + 1]  bucket boundaries in sorted_pairs
  int32_t* sorted_pairs;   // [T * K]
  int32_t* my_off;         // [E]      first inbox row (on the owner) of my rows for expert e
  int32_t* expert_rows;    // [El]     rows this rank receives per local expert
  int32_t* expert_row0;    // [El + 1] prefix of expert_rows
  int32_t* tile_prefix;    // [El + 1] prefix of ceil(rows / tile_rows)
  int32_t* expected_cum;   // [El]     arrivals expected so far (all calls)
  int32_t* arrived;        // heap [El] arrivals so far (all calls)
  long long* inbox_meta;   // heap [capacity]  (source rank << 32) | pair id
};

// ------------------------------------------------------------------------------------ 1 router
// One warp, one token: top-k of its E logits (kPer per lane), softmax over the k selected. Lane k < K returns with
// the k-th choice and its weight. A logit of -inf (a masked expert) or NaN ranks last but is an expert all the same:
// with fewer than K others it is chosen, lowest index first, so an index is always in range. The logits are ranked as integers
// of the same order (0 = no candidate, below -inf's), so a round is two warp reductions, the largest key and the lowest index
// that has it; ten dependent shuffles took 300 cycles a round.
template <int kPer>
__device__ __forceinline__ void route_token(const float* row, int E, int K, int lane, int& my_i, float& my_w) {
  uint32_t key[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const bool in = lane + i * 32 < E;
    float x = in ? row[lane + i * 32] : 0.f;
    x = x == x ? x + 0.f : -INFINITY;                              // (-0 ranks with +0)
    const uint32_t u = __float_as_uint(x);
    key[i] = in ? (u >> 31 ? ~u : u | 0x80000000u) : 0u;
  }
  float my_v = -INFINITY;
  my_i = 0;
  for (int k = 0; k < K; ++k) {
    uint32_t best = 0;
    int bi = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (key[i] > best) { best = key[i]; bi = lane + i * 32; }    // of equal ones the first: the lowest index
    const uint32_t m = __reduce_max_sync(0xffffffffu, best);
    const int e = (int)__reduce_min_sync(0xffffffffu, best == m && m ? (uint32_t)bi : 0x7fffffffu);
    if (lane == k) { my_v = __uint_as_float(m >> 31 ? m & 0x7fffffffu : ~m); my_i = e; }
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (lane + i * 32 == e) key[i] = 0;
  }
  const float ex = __expf(my_v - __shfl_sync(0xffffffffu, my_v, 0));
  float sum = 0.f;
  for (int k = 0; k < K; ++k) sum += __shfl_sync(0xffffffffu, ex, k);
  my_w = ex / sum;
}

// Blocks walk the tokens and count their choices in shared memory; a block adds its histogram to the global one
// once per expert. With one global atomic per (token, k) the counters were the bottleneck: 4096 tokens, 32 experts,
// top-8: 36 us, now 11.
template <int kPer>
__global__ void __launch_bounds__(512) router_topk_kernel(const float* logits, MoeDims dm, MoeMeta m) {
  ptx::pdl_wait();
  ptx::pdl_trigger();
  __shared__ int32_t hist[1024];
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int e = threadIdx.x; e < dm.E; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  for (int t = blockIdx.x * wpb + (threadIdx.x >> 5); t < dm.T; t += gridDim.x * wpb) {
    int my_i;
    float my_w;
    route_token<kPer>(logits + (size_t)t * dm.E, dm.E, dm.K, lane, my_i, my_w);
    if (lane < dm.K) {
      m.topk_idx[(size_t)t * dm.K + lane] = my_i;
      m.topk_w[(size_t)t * dm.K + lane] = my_w;
      atomicAdd(&hist[my_i], 1);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < dm.E; e += blockDim.x)
    if (hist[e]) atomicAdd(&m.counts_local[e], hist[e]);
}

// ------------------------------------------------------------------------------------ 2 meta
__global__ void __launch_bounds__(1024) moe_meta_kernel(const __grid_constant__ DeviceContext ctx, SyncBlock* sb, MoeDims dm,
                                                          MoeMeta m) {
  ptx::pdl_wait();
  ptx::pdl_trigger();
  const int W = ctx.world, E = dm.E, El = dm.El;
  const int32_t e0 = read_epoch(sb);
  __shared__ int s_ok;
  // publish my histogram on every rank, then one cross-rank round
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    const int32_t c = m.counts_local[i];
    for (int r = 0; r < W; ++r) *ctx.remote(m.counts_all + (size_t)ctx.rank * E + i, r) = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    bool ok = true;
    if (W > 1) {
      __threadfence_system();
      barrier_signal(ctx, sb);
      ok = barrier_wait(ctx, sb, e0 + 1);
    }
    sb->epoch = e0 + 1;
    s_ok = ok ? 1 : 0;
  }
  __syncthreads();
  if (!s_ok) return;
  // per global expert: total rows, my offset inside the owner's block
  __shared__ int32_t tot[1024];
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int t = 0;
    for (int s = 0; s < W; ++s) t += __ldcv(m.counts_all + (size_t)s * E + e);
    tot[e] = t;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int owner = e / El;
    int off = 0;
    for (int e2 = owner * El; e2 < e; ++e2) off += tot[e2];
    for (int s = 0; s < ctx.rank; ++s) off += __ldcv(m.counts_all + (size_t)s * E + e);
    m.my_off[e] = off;
    m.cursor[e] = 0;
  }
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) { m.list_off[e] = acc; acc += m.counts_local[e]; }
    m.list_off[E] = acc;
    int rows = 0, tiles = 0;
    for (int j = 0; j < El; ++j) {
      const int r = tot[ctx.rank * El + j];
      m.expert_rows[j] = r;
      m.expert_row0[j] = rows;
      m.tile_prefix[j] = tiles;
      m.expected_cum[j] += r;
      rows += r;
      tiles += expert_tiles(r, dm.tile_rows);
    }
    m.expert_row0[El] = rows;
    m.tile_prefix[El] = tiles;
    if (rows > dm.capacity) ctx.fail(kBadTranslate);   // more rows routed here than the inbox holds
  }
}

// ------------------------------------------------------------------------------------ 3 sort
// A block counts its pairs per expert in shared memory, reserves that many places of each bucket with one global
// atomic per expert, and places its pairs behind them (32768 pairs, 32 experts: 11 us with an atomic per pair, now 4).
// With one rank the bucket position is also the pair's inbox row: it is kept in `pos_of` for the gather.
__global__ void __launch_bounds__(256) moe_sort_kernel(MoeDims dm, MoeMeta m, int32_t* pos_of) {
  ptx::pdl_wait();
  ptx::pdl_trigger();      // not earlier: the gather reads the tokens before its own wait: see launch_pdl.cuh
  __shared__ int32_t cnt[1024], base[1024];
  for (int e = threadIdx.x; e < dm.E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  int e = 0, local = 0;
  if (p < dm.T * dm.K) {
    e = m.topk_idx[p];
    local = atomicAdd(&cnt[e], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < dm.E; i += blockDim.x)
    if (cnt[i]) base[i] = m.list_off[i] + atomicAdd(&m.cursor[i], cnt[i]);
  __syncthreads();
  if (p < dm.T * dm.K) {
    const int pos = base[e] + local;
    m.sorted_pairs[pos] = p;
    if (pos_of) pos_of[p] = pos;
  }
}
__global__ void moe_clear_kernel(MoeDims dm, MoeMeta m) {
  ptx::pdl_wait();
  ptx::pdl_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < dm.E) m.counts_local[i] = 0;
}

// ------------------------------------------------------------------------------------ 1-3 in one block (one rank)
// One rank and few tokens: routing, offsets and sort in one launch instead of four, whose latency is all they cost
// (64 tokens, 32 experts: 18 us in four kernels, now 12). With more tokens the work of a single block would be the longer.
constexpr int kPrepMaxTokens = 256;
template <int kPer>
__global__ void __launch_bounds__(1024) moe_prep_kernel(const float* logits, const __grid_constant__ DeviceContext ctx, MoeDims dm,
                                                        MoeMeta m, int32_t* pos_of) {
  ptx::pdl_wait();
  ptx::pdl_trigger();      // not earlier: the gather reads the tokens before its own wait: see launch_pdl.cuh
  __shared__ int32_t hist[1024], off[1024], w_rows[32], w_tiles[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  hist[tid] = 0;
  __syncthreads();
  for (int t = warp; t < dm.T; t += 32) {
    int my_i;
    float my_w;
    route_token<kPer>(logits + (size_t)t * dm.E, dm.E, dm.K, lane, my_i, my_w);
    if (lane < dm.K) {
      const size_t p = (size_t)t * dm.K + lane;
      m.topk_idx[p] = my_i;
      m.topk_w[p] = my_w;
      pos_of[p] = atomicAdd(&hist[my_i], 1);       // place inside the expert's rows
    }
  }
  __syncthreads();
  // exclusive prefix sums of rows and token tiles over the experts, one expert per thread
  const int rows = tid < dm.E ? hist[tid] : 0, tiles = expert_tiles(rows, dm.tile_rows);
  int pr = rows, pt = tiles;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int ur = __shfl_up_sync(0xffffffffu, pr, o), ut = __shfl_up_sync(0xffffffffu, pt, o);
    if (lane >= o) { pr += ur; pt += ut; }
  }
  if (lane == 31) { w_rows[warp] = pr; w_tiles[warp] = pt; }
  __syncthreads();
  for (int w = 0; w < warp; ++w) { pr += w_rows[w]; pt += w_tiles[w]; }
  if (tid < dm.E) {
    off[tid] = pr - rows;
    m.expert_rows[tid] = rows;
    m.expert_row0[tid] = pr - rows;
    m.tile_prefix[tid] = pt - tiles;
    if (tid == dm.E - 1) {
      m.expert_row0[dm.E] = pr;
      m.tile_prefix[dm.E] = pt;
      if (pr > dm.capacity) ctx.fail(kBadTranslate);     // more rows routed here than the inbox holds
    }
  }
  __syncthreads();
  for (int p = tid; p < dm.T * dm.K; p += blockDim.x) {
    const int pos = off[m.topk_idx[p]] + pos_of[p];
    m.sorted_pairs[pos] = p;
    pos_of[p] = pos;
  }
}

// ------------------------------------------------------------------------------------ 4' gather (one rank)
// With one rank every pair's row stays here, so nothing is sent: the token rows are copied into expert order by a
// kernel of their own and the grouped GEMM runs on every SM. The communication CTAs of the multi-rank form cost the
// GEMM 16 of 148 SMs for its whole run, and with few tokens their chain of one release per expert was what it waited
// for (64 tokens, 32 experts, e4m3: stage 1 306 us with them and 199 without; 4096 tokens bf16: 1808 us and 1538, plus 89 for
// this copy, which is bound by the 470 MB it writes). A block reads a piece of one token's row once and stores it to the
// token's K rows.
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint8_t* x, uint8_t* inbox, int row16,
                                                         const int32_t* pos_of, int K, int capacity) {
  __shared__ int32_t dst[kMaxTopK];
  const int t = blockIdx.x;
  // the tokens were complete before the kernel in front got past its own pdl_wait: the first piece is read while it runs (16 tokens,
  // 16 experts of 2048 x 1024: 45.0 -> 43.9 us a pass; quantising e4m3 rows that early was slower, 30.6 -> 31.5)
  const uint4* src = (const uint4*)x + (size_t)t * row16;
  const int c0 = blockIdx.y * blockDim.x + threadIdx.x;
  uint4 v = c0 < row16 ? __ldcg(src + c0) : make_uint4(0, 0, 0, 0);
  ptx::pdl_wait();
  ptx::pdl_trigger();      // not earlier: stage 1 reads weights and tables before its own wait: see launch_pdl.cuh
  if (threadIdx.x < K) dst[threadIdx.x] = pos_of[(size_t)t * K + threadIdx.x];
  __syncthreads();
  for (int c = c0; c < row16; c += gridDim.y * blockDim.x) {
    if (c != c0) v = __ldcg(src + c);
    for (int k = 0; k < K; ++k)
      if (dst[k] < capacity) ((uint4*)inbox)[(size_t)dst[k] * row16 + c] = v;
  }
}

// The same for e4m3 rows, from the 16-bit tokens: half a warp quantises one 128-column block of a token, stores the values to
// the token's K rows and the scale byte, four times, to its cell of the scale atoms of each row's tile ([tile][K block][atoms]).
__global__ void __launch_bounds__(256) moe_gather_quant_kernel(const __nv_bfloat16* x, uint8_t* inbox, uint8_t* inbox_sf, int atoms, MoeDims dm, MoeMeta m,
                                                               const int32_t* pos_of) {
  ptx::pdl_wait();
  ptx::pdl_trigger();      // not earlier: stage 1 reads weights and tables before its own wait: see launch_pdl.cuh
  __shared__ int32_t dst[kMaxTopK], tile[kMaxTopK], cell[kMaxTopK];
  const int t = blockIdx.x, half = threadIdx.x >> 4, sub = threadIdx.x & 15, D = dm.D, K = dm.K, kblocks = D / 128;
  if (threadIdx.x < K) {
    const int p = t * K + threadIdx.x, e = m.topk_idx[p], pos = pos_of[p], first = m.tile_prefix[e];
    const int row0 = m.expert_row0[e], per = expert_tile_rows(m.expert_row0[e + 1] - row0, m.tile_prefix[e + 1] - first);
    const int i = (pos - row0) / per;
    dst[threadIdx.x] = pos;
    tile[threadIdx.x] = first + i;
    cell[threadIdx.x] = sf_cell(pos - row0 - i * per);
  }
  __syncthreads();
  const int kb = blockIdx.y * 16 + half, c = kb * 128 + sub * 8;       // D is a multiple of 256: whole blocks
  Raw8<__nv_bfloat16> raw;
  raw.load(x + (size_t)t * D + c, c < D ? 8 : 0, 2);
  const int e = block_exponent(raw);
  if (c >= D) return;
  const uint2 v = quantised8(raw, e);
  for (int k = 0; k < K; ++k) {
    if (dst[k] >= dm.capacity) continue;
    *(uint2*)(inbox + (size_t)dst[k] * D + c) = v;
    if (sub == 0) *(uint32_t*)(inbox_sf + ((size_t)tile[k] * kblocks + kb) * (atoms * 512) + cell[k]) = (uint32_t)(e + 127) * 0x01010101u;
  }
}

// ------------------------------------------------------------------ 4/5 grouped GEMM policies
// kStage 1: A = inbox rows (dispatch runs in the communication CTAs of the same kernel), B = fused
// gate|up weight, SwiGLU epilogue into H. kStage 2: A = H, B = down weight, the epilogue sends
// every row to its token's home rank.
// kFp8: block-scaled e4m3. Tokens travel as e4m3 rows plus one scale byte per 128 columns; the inbox rows of
// a tile arrive one by one, so the producer warp puts the tile's scale atoms together from those bytes
// (kSfaFromRows). Stage 1's SwiGLU epilogue writes H as e4m3 with one scale byte per row and 128 columns
// (kQuantOut), which stage 2 reads the same way. Weights carry 128 x 128 block scales packed per expert.
template <int kStage, bool kFp8 = false>
struct GroupedGemm : Common {
  static constexpr bool kBulkEpilogue = false;
  static constexpr bool kSwiGLU = kStage == 1;
  static constexpr bool kSfaFromRows = kFp8;
  static constexpr bool kQuantOut = kFp8 && kStage == 1;
  static constexpr int kEsz = kFp8 ? 1 : 2;        // bytes per element of the tokens / of H
  const uint8_t* a_sf;     // fp8: scale bytes of this GEMM's A rows, [capacity][a_sf_ld] (inbox_sf or H_sf)
  int a_sf_ld;
  const uint8_t* x_sf;     // fp8 stage 1: scale bytes of this rank's tokens [T][a_sf_ld] (dispatch source)
  uint8_t* inbox_sf;       // fp8 stage 1: heap [capacity][a_sf_ld]
  uint8_t* h_sf;           // fp8 stage 1: [capacity][h_sf_ld] scale bytes of H
  int h_sf_ld;
  int sfb_per_expert;      // fp8: scale atoms of B per expert (tiles_n * kblocks * sfb_atoms)
  DeviceContext ctx;
  SyncBlock* sb;
  MoeDims dm;
  MoeMeta meta;
  const uint8_t* x;        // [T, D] tokens of this rank (stage 1: dispatch source)
  uint8_t* inbox;          // heap [capacity, D]
  uint8_t* H;              // [capacity, F]
  uint8_t* comb;           // heap [T * K, D]
  int n_comm_ctas;
  int k_per_expert;        // rows of B per expert (K of this GEMM)
  int n_per_expert;        // columns of B per expert when B is stored [El * N, K] (K-major)
  int b_kmajor;

  struct State {
    int j = -1;            // local expert of the current tile
    int key = -1;          // expert whose arrivals were confirmed
    int row0 = 0, rows_end = 0;
    unsigned long long* tab = nullptr;   // stage 2: destination row pointers of this warp's 32 rows
    uint32_t sf_cur[4] = {0, 0, 0, 0};   // fp8 producer: scale bytes of rows lane + 32 a for K blocks [4 g, 4 g + 4)
    uint32_t sf_nxt[4] = {0, 0, 0, 0};   //               and for the next four
  };
  IRIS_D int num_tiles() const { return meta.tile_prefix[dm.El] * tiles_n; }
  // tile -> (virtual m index = global 128-row tile counter, n tile); experts in order
  IRIS_D void tile(int t, int& tm, int& tn) const {
    tm = t / tiles_n;
    tn = t - tm * tiles_n;
  }
  IRIS_D int expert_of(int tm) const {
    int j = 0;
    while (j + 1 < dm.El && meta.tile_prefix[j + 1] <= tm) ++j;
    return j;
  }
  // The same asked by a whole converged warp, 32 experts per load and vote: the producer's search stands in front of
  // every tile's loads, and one dependent load per expert lasted longer than its ring.
  IRIS_D int expert_of_warp(int tm) const {
    const int lane = threadIdx.x & 31;
    int j = 0;
    for (int base = 0; base + 1 < dm.El; base += 32) {
      const int e = base + lane;
      const int n = __popc(__ballot_sync(0xffffffffu, e + 1 < dm.El && meta.tile_prefix[e + 1] <= tm));
      j += n;
      if (n < 32) break;
    }
    return j;
  }
  IRIS_D bool a_source(State& st, int tm, int kb, ASource& s) const {
    if (kb == 0) {
      st.j = expert_of_warp(tm);
      st.row0 = meta.expert_row0[st.j] + (tm - meta.tile_prefix[st.j]) * kBM;
      if (kStage == 1 && ctx.world > 1 && st.key != st.j) {     // one rank: the gather kernel ran before
        if (!wait_flag_ge(ctx, meta.arrived + st.j, meta.expected_cum[st.j])) return false;
        st.key = st.j;
        ptx::fence_proxy_async();
      }
    }
    s.map = &tmA; s.x = kb * bk; s.y = st.row0;
    if (b_kmajor) { s.bk = kb * bk; s.bn0 += st.j * n_per_expert; }
    else s.bk = st.j * k_per_expert + kb * bk;
    s.sf_map = nullptr; s.sf_row = 0;
    s.sfb_off = st.j * sfb_per_expert;
    return true;
  }
  // fp8: the scale atom of (128-row tile at st.row0, K block kb). Lane l owns rows l, l + 32, l + 64, l + 96:
  // their scale bytes come four K blocks at a time (one 32-bit load per row, the following group prefetched),
  // and the lane writes bytes [16 l, 16 l + 16) of the atom: for each of its rows the byte of this block, four times.
  IRIS_D void sfa_fill(State& st, int, int kb, uint8_t* atom, int lane) const {
    auto ld = [&](int a, int k) -> uint32_t {
      const int row = min(st.row0 + lane + 32 * a, dm.capacity - 1);
      return __ldcg((const uint32_t*)(a_sf + (size_t)row * a_sf_ld + k));
    };
    if (kb == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) { st.sf_cur[a] = ld(a, 0); st.sf_nxt[a] = 4 < a_sf_ld ? ld(a, 4) : 0; }
    } else if ((kb & 3) == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) { st.sf_cur[a] = st.sf_nxt[a]; st.sf_nxt[a] = kb + 4 < a_sf_ld ? ld(a, kb + 4) : 0; }
    }
    const int sh8 = (kb & 3) * 8;
    uint4 v;
    v.x = ((st.sf_cur[0] >> sh8) & 0xffu) * 0x01010101u;
    v.y = ((st.sf_cur[1] >> sh8) & 0xffu) * 0x01010101u;
    v.z = ((st.sf_cur[2] >> sh8) & 0xffu) * 0x01010101u;
    v.w = ((st.sf_cur[3] >> sh8) & 0xffu) * 0x01010101u;
    *(uint4*)(atom + lane * 16) = v;
  }
  // fp8 stage 1: 32 e4m3 values of H, and the row's scale byte for the tile's 128 columns
  IRIS_D void store_q32(State& st, int row, int col, uint4 a, uint4 b) const {
    if (row >= st.rows_end || col >= dm.F) return;
    uint4* p = (uint4*)(H + (size_t)row * dm.F + col);
    p[0] = a; p[1] = b;
  }
  IRIS_D void store_row_scale(State& st, int row, int n_tile, uint32_t byte) const {
    if (row < st.rows_end) h_sf[(size_t)row * h_sf_ld + n_tile] = (uint8_t)byte;
  }
  IRIS_D int row_origin(State& st, int) const { return st.row0; }
  IRIS_D void begin_tile(State& st, int tm, int, uint8_t* warp_scratch) const {
    st.j = expert_of(tm);
    st.row0 = meta.expert_row0[st.j] + (tm - meta.tile_prefix[st.j]) * kBM;
    st.rows_end = min(meta.expert_row0[st.j] + meta.expert_rows[st.j], dm.capacity);
    if (kStage == 2) {
      st.tab = (unsigned long long*)warp_scratch;
      const int lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3;
      const int row = st.row0 + quarter * 32 + lane;
      unsigned long long ptr = 0;
      if (row < st.rows_end) {
        const long long mt = ctx.world > 1 ? meta.inbox_meta[row] : (long long)meta.sorted_pairs[row];
        const int src = (int)(mt >> 32), pair = (int)(mt & 0xffffffffll);
        ptr = (unsigned long long)ctx.remote(comb + (size_t)pair * dm.D * 2, src);      // the combine buffer stays 16-bit
      }
      __syncwarp();
      st.tab[lane] = ptr;
      __syncwarp();
    }
  }
  IRIS_D void store16(State& st, int row, int col, uint4 v) const {
    if (row >= st.rows_end) return;
    if (kStage == 1) {
      if (col < dm.F) *(uint4*)(H + ((size_t)row * dm.F + col) * 2) = v;
    } else {
      const int quarter = (threadIdx.x >> 5) & 3;
      const unsigned long long p = st.tab[row - st.row0 - quarter * 32];
      if (p && col < dm.D) *(uint4*)(p + (size_t)col * 2) = v;
    }
  }
  IRIS_D void tile_done(State&, int, int) const {}

  // Dispatch (stage 1 only): groups (local expert j, destination) in j-major order, the order in
  // which the GEMM CTAs consume the experts. Every communication CTA pushes its slice of the rows
  // of EVERY group, so the first expert's rows are complete after 1 / El of the dispatch instead
  // of after a whole group per CTA. Rows go HBM -> shared memory -> destination inbox by bulk
  // async copies driven by one thread; the 8-byte routing record of each row is stored by the
  // other threads; each CTA adds its slice's row count to the expert's arrival counter.
  static constexpr int kSlot = 16 * 1024;
  IRIS_D void comm_main(uint8_t* smem_raw, int smem_bytes) const {
    if (kStage != 1) return;
    const int c = blockIdx.x - n_gemm_ctas;
    const int W = ctx.world;
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    const uint32_t row_bytes = (uint32_t)dm.D * kEsz;
    const int pieces = (int)((row_bytes + kSlot - 1) / kSlot);      // pieces per row
    int nb = (smem_bytes - 1024) / kSlot;
    if (nb > 12) nb = 12;
    uint64_t* bars = (uint64_t*)(smem + (size_t)nb * kSlot);
    if (threadIdx.x == 0) {
      for (int i = 0; i < nb; ++i) ptx::mbar_init(&bars[i], 1);
      ptx::fence_mbar_init();
      ptx::fence_proxy_async();
    }
    __syncthreads();
    int seq = 0;   // pieces issued so far (ring slot / parity)
    for (int g = 0; g < dm.El * W; ++g) {
      const int j = g / W;
      int r = ctx.rank + g % W;
      if (r >= W) r -= W;
      const int e = r * dm.El + j;
      const int n_all = meta.list_off[e + 1] - meta.list_off[e];
      const int i0 = (int)((long long)n_all * c / n_comm_ctas), i1 = (int)((long long)n_all * (c + 1) / n_comm_ctas);
      const int n = i1 - i0;
      if (n == 0) continue;                      // uniform over the CTA
      const int lo = meta.list_off[e] + i0;
      const int dst0 = meta.my_off[e] + i0;
      uint8_t* dst_inbox = ctx.remote(inbox, r);
      long long* dst_meta = ctx.remote(meta.inbox_meta, r);
      // routing records
      for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (dst0 + i < dm.capacity) dst_meta[dst0 + i] = ((long long)ctx.rank << 32) | (long long)meta.sorted_pairs[lo + i];
      if constexpr (kFp8) {       // and the rows' scale bytes, 16 at a time
        uint8_t* dst_sf = ctx.remote(inbox_sf, r);
        const int per_row = a_sf_ld / 16;
        for (int u = threadIdx.x; u < n * per_row; u += blockDim.x) {
          const int i = u / per_row, c16 = u - i * per_row;
          if (dst0 + i >= dm.capacity) continue;
          const int tok = meta.sorted_pairs[lo + i] / dm.K;
          *(uint4*)(dst_sf + (size_t)(dst0 + i) * a_sf_ld + c16 * 16) = *(const uint4*)(x_sf + (size_t)tok * a_sf_ld + c16 * 16);
        }
      }
      if (threadIdx.x == 0) {
        const int total = n * pieces;
        auto src_of = [&](int q) -> const uint8_t* {
          const int i = q / pieces, k = q - i * pieces;
          const int pair = meta.sorted_pairs[lo + i];
          return x + (size_t)(pair / dm.K) * row_bytes + (size_t)k * kSlot;
        };
        auto len_of = [&](int q) -> uint32_t {
          const int k = q % pieces;
          return min((uint32_t)kSlot, row_bytes - (uint32_t)k * kSlot);
        };
        auto issue = [&](int q) {
          const int slot = (seq + q) % nb;
          ptx::mbar_expect_tx(&bars[slot], len_of(q));
          ptx::bulk_load(smem + (size_t)slot * kSlot, src_of(q), len_of(q), &bars[slot]);
        };
        int next = min(nb, total);
        for (int q = 0; q < next; ++q) issue(q);
        bool ok = true;
        for (int q = 0; q < total; ++q) {
          const int slot = (seq + q) % nb;
          if (!ptx::mbar_wait(&bars[slot], (uint32_t)(((seq + q) / nb) & 1), kPipeTimeoutNs)) { fail(kTimeoutPipeline); ok = false; break; }
          const int i = q / pieces, k = q - i * pieces;
          if (dst0 + i < dm.capacity)
            ptx::bulk_store(dst_inbox + (size_t)(dst0 + i) * row_bytes + (size_t)k * kSlot, smem + (size_t)slot * kSlot, len_of(q));
          ptx::bulk_commit();
          if (q == total - 1) ptx::bulk_wait<0>();
          else ptx::bulk_wait_read<1>();
          const int free_upto = q == total - 1 ? q : q - 1;
          while (next <= free_upto + nb && next < total) issue(next++);
        }
        seq += total;
        if (ok) {
          ptx::fence_proxy_async();
        }
      }
      __syncthreads();   // routing records of all threads + data of thread 0 precede the release below
      if (threadIdx.x == 0) {
        fence_sys();
        red_release_sys_add(ctx.remote(meta.arrived + j, r), n);
      }
    }
  }
  IRIS_D void post_main() const {
    if (kStage == 2) {
      grid_exit_barrier(ctx, sb, read_epoch(sb), 0);
    }
  }
};

// ------------------------------------------------------------------------------------ 6 reduce
// Bound by the K rows it reads per token. One thread per eight columns of a token, the loads of all K rows issued
// before the first is used (64 tokens of 7168, top-8: 12 us with one block per token, now 5; 4096 tokens: 80 us, the time
// its 530 MB take).
__global__ void __launch_bounds__(128) moe_reduce_kernel(const __nv_bfloat16* comb, const float* w, __nv_bfloat16* out,
                                                         int T, int K, int D) {
  ptx::pdl_wait();
  ptx::pdl_trigger();
  __shared__ float s_w[kMaxTopK];
  const int t = blockIdx.x;
  if (threadIdx.x < K) s_w[threadIdx.x] = w[(size_t)t * K + threadIdx.x];
  __syncthreads();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 8;
  if (c >= D) return;
  const __nv_bfloat16* rows = comb + (size_t)t * K * D + c;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int k0 = 0; k0 < K; k0 += 8) {
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k0 + i < K) v[i] = __ldcg((const uint4*)(rows + (size_t)(k0 + i) * D));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (k0 + i >= K) break;
      const float wk = s_w[k0 + i];
      const __nv_bfloat162* h = (const __nv_bfloat162*)&v[i];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 f = __bfloat1622float2(h[q]);
        acc[2 * q] += wk * f.x;
        acc[2 * q + 1] += wk * f.y;
      }
    }
  }
  uint4 o;
  __nv_bfloat162* oh = (__nv_bfloat162*)&o;
#pragma unroll
  for (int q = 0; q < 4; ++q) oh[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
  *(uint4*)(out + (size_t)t * D + c) = o;
}

}  // namespace

extern "C" {

typedef struct IrisMoeDesc {
  IrisCtx ctx;
  int32_t T, K, E, El, D, F, capacity, comm_ctas;
  const void* x;            // [T, D] bf16
  const float* logits;      // [T, E]
  const void* w13;          // [El, D, 2F] bf16, columns in blocks of [gate 128 | up 128]
  const void* w2;           // [El, F, D] bf16
  void* out;                // [T, D] bf16
  void* inbox; void* H; void* comb;
  void* sync_meta; void* sync_gemm2;
  int32_t* topk_idx; float* topk_w;
  int32_t* counts_local; int32_t* counts_all; int32_t* cursor; int32_t* list_off; int32_t* sorted_pairs; int32_t* my_off;
  int32_t* expert_rows; int32_t* expert_row0; int32_t* tile_prefix; int32_t* expected_cum; int32_t* arrived;
  void* inbox_meta;
  int32_t weights_kmajor;   // 1: w13 is [El, 2F, D] and w2 is [El, D, F] (each expert's weight transposed: K contiguous)
  // Block-scaled e4m3 mode (fp8 != 0; weights_kmajor must be 1): x is the e4m3 form of the tokens [T, D] bytes,
  // w13 / w2 are e4m3, inbox is [capacity, D] bytes, H is [capacity, F] bytes; comb and out stay bf16.
  int32_t fp8;
  int32_t sf_ld1;           // bytes per row of x_sf / inbox_sf: >= D / 128, multiple of 16
  int32_t sf_ld2;           // bytes per row of H_sf: >= F / 128, multiple of 16
  const void* x_sf;         // [T, sf_ld1] one UE8M0 byte per token and 128 columns
  void* inbox_sf;           // heap [capacity, sf_ld1]
  void* H_sf;               // [capacity, sf_ld2]
  const void* w13_sf;       // scale atoms of w13: [El][2F / 256][D / 128][2][512]
  const void* w2_sf;        // scale atoms of w2:  [El][ceil(D / 224)][F / 128][2][512]
  int32_t* pos_of;          // [T * K] one rank only: inbox row of each (token, k) pair
  // One rank, e4m3: the bf16 tokens [T, D], quantised on the way into the inbox (x and x_sf are not read). inbox_sf and H_sf
  // are then scale atoms per token tile, iris_moe_sf_bytes(T, K, E, D or F) bytes each; w13_sf is [El][F / 128][D / 128][512], an
  // atom's first 256 bytes from the gate block's scale and the rest from the up block's; w2_sf is [El][D / 256][F / 128][2][512].
  const void* x16;
} IrisMoeDesc;

// One rank: up to this many tokens a call is 5 kernels, above it 8.
int iris_moe_prep_max_tokens(void) { return kPrepMaxTokens; }

// One rank, e4m3: bytes of the scale atoms of the token tiles of up to T tokens, for rows of `cols` columns.
long long iris_moe_sf_bytes(int T, int K, int E, int cols) {
  const long long small = T < kSmallTokens ? T : kSmallTokens;                          // a call may have fewer tokens: E tiles of one atom
  const long long tiles = (long long)T * K / kTileFp8 + E;
  const long long big = T > kSmallTokens ? tiles * 2 : 0, few = small > 0 ? E : 0;
  return (big > few ? big : few) * 512 * ceil_div(cols, 128);
}

int iris_moe_forward(const IrisMoeDesc* d, void* stream_) {
  cudaStream_t s = (cudaStream_t)stream_;
  if (d->K > kMaxTopK || d->E > 1024 || d->E % d->ctx.world || d->D % 64 || d->F % 128 || d->D % 256 || d->K > d->E || d->K < 1) return -3;
  if (d->T <= 0) return -21;
  DeviceContext ctx;
  memcpy(&ctx, &d->ctx, sizeof(ctx));
  const bool one_rank = ctx.world <= 1, km = d->weights_kmajor != 0;
  const bool experts = one_rank && km;          // the pair kernel of moe_experts.cuh
  const bool small = d->T <= kSmallTokens;
  const int tile_rows = !experts ? kBM : small ? kSmallTokens : d->fp8 ? kTileFp8 : kTile16;
  MoeDims dm{d->T, d->K, d->E, d->El, d->D, d->F, d->capacity, tile_rows};
  MoeMeta m{d->topk_idx, d->topk_w, d->counts_local, d->counts_all, d->cursor, d->list_off, d->sorted_pairs, d->my_off,
            d->expert_rows, d->expert_row0, d->tile_prefix, d->expected_cum, d->arrived, (long long*)d->inbox_meta};
  const int sms = sm_count();
  int32_t* pos_of = one_rank ? d->pos_of : nullptr;
  if (d->fp8 && !km) return -3;
  if (one_rank && (!pos_of || ((uintptr_t)d->x & 15) || ((uintptr_t)d->x16 & 15) || (d->fp8 && !d->x16))) return -11;
  // On one rank every kernel is launched behind its predecessor without waiting for it to finish (64 tokens, 32 experts,
  // e4m3: 243 us in all, 262 when each waited).
  auto go = [&](auto kern, dim3 grid, int block, auto... args) {
    if (experts) return launch_pdl(kern, grid, block, 0, s, args...);
    kern<<<grid, block, 0, s>>>(args...);
    return 0;
  };
  if (one_rank && d->T <= kPrepMaxTokens) {
    auto* prep = d->E <= 32 ? moe_prep_kernel<1> : d->E <= 64 ? moe_prep_kernel<2> : d->E <= 128 ? moe_prep_kernel<4>
                 : d->E <= 256 ? moe_prep_kernel<8> : moe_prep_kernel<32>;
    if (const int r = go(prep, dim3(1), 1024, d->logits, ctx, dm, m, pos_of)) return r;
  } else {
    if (const int r = go(moe_clear_kernel, dim3((d->E + 255) / 256), 256, dm, m)) return r;
    const int warps = d->T > 16 * sms ? 16 : 4;      // warps per block: few tokens spread over more SMs
    const int blocks = ceil_div(d->T, warps) < sms ? ceil_div(d->T, warps) : sms;
    auto* router = d->E <= 32 ? router_topk_kernel<1> : d->E <= 64 ? router_topk_kernel<2> : d->E <= 128 ? router_topk_kernel<4>
                   : d->E <= 256 ? router_topk_kernel<8> : router_topk_kernel<32>;
    int r = go(router, dim3(blocks), warps * 32, d->logits, dm, m);
    if (!r) r = go(moe_meta_kernel, dim3(1), 1024, ctx, (SyncBlock*)d->sync_meta, dm, m);
    if (!r) r = go(moe_sort_kernel, dim3(ceil_div(d->T * d->K, 256)), 256, dm, m, pos_of);
    if (r) return r;
  }
  if (one_rank) {
    if (d->fp8) {
      const int r = go(moe_gather_quant_kernel, dim3(d->T, ceil_div(d->D, 2048)), 256, (const __nv_bfloat16*)d->x16, (uint8_t*)d->inbox, (uint8_t*)d->inbox_sf,
                       small ? 1 : 2, dm, m, (const int32_t*)pos_of);
      if (r) return r;
    } else {
      const int row16 = d->D * 2 / 16;
      int split = ceil_div(4 * sms, d->T);
      if (split > ceil_div(row16, 256)) split = ceil_div(row16, 256);
      const int r = go(moe_gather_kernel, dim3(d->T, split), 256, (const uint8_t*)d->x, (uint8_t*)d->inbox, row16, (const int32_t*)pos_of, d->K, d->capacity);
      if (r) return r;
    }
  }
  if (cudaGetLastError() != cudaSuccess) return -21;

  const int comm = one_rank ? 0 : (d->comm_ctas > 0 ? d->comm_ctas : 16);
  auto common = [&](auto& pol, int bn, int N, int Kdim, bool f8) {
    pol.sh = Shape{d->capacity, N, Kdim};
    pol.tiles_m = 0; pol.tiles_n = ceil_div(N, bn); pol.group_m = 1;
    pol.bf16 = 1; pol.bn = bn; pol.fp8 = f8; pol.bk = f8 ? 128 : kBK; pol.kblocks = ceil_div(Kdim, pol.bk);
    pol.sfb_atoms = f8 ? ceil_div(bn, 128) : 0; pol.c_bulk = 0;
    pol.bias_row = nullptr; pol.bias_col = nullptr; pol.status = d->ctx.status; pol.timeline = nullptr;
    pol.ctx = ctx; pol.dm = dm; pol.meta = m;
    pol.inbox = (uint8_t*)d->inbox; pol.H = (uint8_t*)d->H; pol.comb = (uint8_t*)d->comb;
    pol.b_kmajor = km;
    pol.a_sf = nullptr; pol.a_sf_ld = 0; pol.x_sf = nullptr; pol.inbox_sf = nullptr; pol.h_sf = nullptr; pol.h_sf_ld = 0;
    pol.sfb_per_expert = pol.tiles_n * pol.kblocks * pol.sfb_atoms;
  };
  if (experts) {
    ExpertArgs a;
    a.row0 = m.expert_row0; a.tiles = m.tile_prefix; a.pairs = m.sorted_pairs;
    a.status = d->ctx.status; a.El = d->El; a.capacity = d->capacity;
    const int max_tiles = small ? d->E : d->T * d->K / tile_rows + d->E;
    const ExpertProblem up{d->w13, d->w13_sf, d->inbox, d->inbox_sf, 2 * d->F, d->D, max_tiles};
    const ExpertProblem down{d->w2, d->w2_sf, d->H, d->H_sf, d->D, d->F, max_tiles};
    a.out = (uint8_t*)d->H; a.out_sf = (uint8_t*)d->H_sf; a.ldo = d->F;
    int r = d->fp8 ? (small ? launch_experts<ExpertCfg<1, true, kSmallTokens>>(a, up, s) : launch_experts<ExpertCfg<1, true, kTileFp8>>(a, up, s))
                   : (small ? launch_experts<ExpertCfg<1, false, kSmallTokens>>(a, up, s) : launch_experts<ExpertCfg<1, false, kTile16>>(a, up, s));
    if (r) return r;
    a.out = (uint8_t*)d->comb; a.out_sf = nullptr; a.ldo = d->D;
    r = d->fp8 ? (small ? launch_experts<ExpertCfg<2, true, kSmallTokens>>(a, down, s) : launch_experts<ExpertCfg<2, true, kTileFp8>>(a, down, s))
               : (small ? launch_experts<ExpertCfg<2, false, kSmallTokens>>(a, down, s) : launch_experts<ExpertCfg<2, false, kTile16>>(a, down, s));
    if (r) return r;
  } else if (d->fp8) {
    if (!km || d->sf_ld1 % 16 || d->sf_ld2 % 16 || d->sf_ld1 * 128 < d->D || d->sf_ld2 * 128 < d->F || d->D % 128 || d->F % 128) return -3;
    {
      GroupedGemm<1, true> pol;
      common(pol, 256, 2 * d->F, d->D, true);
      int r = make_map(&pol.tmA, d->inbox, IRIS_F8E4M3, d->capacity, d->D, d->D, 128, kBM);
      if (r) return r;
      r = make_map(&pol.tmB, d->w13, IRIS_F8E4M3, (uint64_t)d->El * 2 * d->F, d->D, d->D, 128, 256);
      if (r) return r;
      r = make_sf_map(&pol.tmSFB, d->w13_sf, (uint64_t)d->El * pol.sfb_per_expert, pol.sfb_atoms);
      if (r) return r;
      pol.tmSFA = pol.tmSFB;      // unused: A's atoms are built from the rows' scale bytes
      pol.n_gemm_ctas = sms - comm; pol.sb = nullptr;
      pol.x = (const uint8_t*)d->x; pol.n_comm_ctas = comm; pol.k_per_expert = d->D; pol.n_per_expert = 2 * d->F;
      pol.a_sf = (const uint8_t*)d->inbox_sf; pol.a_sf_ld = d->sf_ld1; pol.x_sf = (const uint8_t*)d->x_sf;
      pol.inbox_sf = (uint8_t*)d->inbox_sf; pol.h_sf = (uint8_t*)d->H_sf; pol.h_sf_ld = d->sf_ld2;
      r = launch<Config<256, true, 4, false, true, 1, 0>>(pol, sms, s);
      if (r) return r;
    }
    {
      GroupedGemm<2, true> pol;
      common(pol, 224, d->D, d->F, true);
      int r = make_map(&pol.tmA, d->H, IRIS_F8E4M3, d->capacity, d->F, d->F, 128, kBM);
      if (r) return r;
      r = make_map(&pol.tmB, d->w2, IRIS_F8E4M3, (uint64_t)d->El * d->D, d->F, d->F, 128, 224);
      if (r) return r;
      r = make_sf_map(&pol.tmSFB, d->w2_sf, (uint64_t)d->El * pol.sfb_per_expert, pol.sfb_atoms);
      if (r) return r;
      pol.tmSFA = pol.tmSFB;
      pol.n_gemm_ctas = sms; pol.sb = (SyncBlock*)d->sync_gemm2;
      pol.x = nullptr; pol.n_comm_ctas = 0; pol.k_per_expert = d->F; pol.n_per_expert = d->D;
      pol.a_sf = (const uint8_t*)d->H_sf; pol.a_sf_ld = d->sf_ld2;
      r = launch<Config<224, true, 4, false, true, 2>>(pol, sms, s);
      if (r) return r;
    }
  } else {
  {
    GroupedGemm<1> pol;
    common(pol, 256, 2 * d->F, d->D, false);
    int r = make_map(&pol.tmA, d->inbox, IRIS_BF16, d->capacity, d->D, d->D, kBK, kBM);
    if (r) return r;
    if (km) r = make_map(&pol.tmB, d->w13, IRIS_BF16, (uint64_t)d->El * 2 * d->F, d->D, d->D, kBK, 256);
    else r = make_map(&pol.tmB, d->w13, IRIS_BF16, (uint64_t)d->El * d->D, 2 * d->F, 2 * d->F, 64, 64);
    if (r) return r;
    pol.n_gemm_ctas = sms - comm; pol.sb = nullptr;
    pol.x = (const uint8_t*)d->x; pol.n_comm_ctas = comm; pol.k_per_expert = d->D; pol.n_per_expert = km ? 2 * d->F : 0;
    r = km ? launch<Config<256, true, 4>>(pol, sms, s) : launch<Config<256, false, 4>>(pol, sms, s);
    if (r) return r;
  }
  {
    GroupedGemm<2> pol;
    common(pol, 256, d->D, d->F, false);
    int r = make_map(&pol.tmA, d->H, IRIS_BF16, d->capacity, d->F, d->F, kBK, kBM);
    if (r) return r;
    if (km) r = make_map(&pol.tmB, d->w2, IRIS_BF16, (uint64_t)d->El * d->D, d->F, d->F, kBK, 256);
    else r = make_map(&pol.tmB, d->w2, IRIS_BF16, (uint64_t)d->El * d->F, d->D, d->D, 64, 64);
    if (r) return r;
    pol.n_gemm_ctas = sms; pol.sb = (SyncBlock*)d->sync_gemm2;
    pol.x = nullptr; pol.n_comm_ctas = 0; pol.k_per_expert = d->F; pol.n_per_expert = km ? d->D : 0;
    r = km ? launch<Config<256, true, 4>>(pol, sms, s) : launch<Config<256, false, 4>>(pol, sms, s);
    if (r) return r;
  }
  }
  const int r = go(moe_reduce_kernel, dim3(d->T, ceil_div(d->D, 1024)), 128, (const __nv_bfloat16*)d->comb, (const float*)d->topk_w, (__nv_bfloat16*)d->out,
                   d->T, d->K, d->D);
  if (r) return r;
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // extern "C"
