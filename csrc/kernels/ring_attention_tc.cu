// Ring attention with tcgen05 attention CTAs (the communication CTAs are those of
// ring_attention_common.cuh). One attention CTA works on items of TWO tiles of 128 queries that share their
// K/V head and walks the key blocks in arrival order in tiles of 128 keys:
//
//   warp 0      TMA producer: the item's two Q tiles, then K and V tiles (two stages each) from this rank's own
//               K/V or from the ring-buffer slot of the block's origin, after the slot's arrival counter has
//               been seen (acquire, bounded)
//   warp 1      MMA issuer: per query tile i, S_i = Q_i K^T (tcgen05.mma, M 128, N 128, K 128) and
//               O_i += P_i V (P from TMEM). Issue order PV_0(j), S_0(j+1), PV_1(j), S_1(j+1): the tensor pipe
//               works for one query tile while the softmax of the other runs
//   warps 4..7  softmax of query tile 0, warps 8..11 of tile 1, one thread per query row (216 registers each, the
//               issuers give theirs up). Per tile: tcgen05.ld of
//               the 128 scores, row maximum, P = exp2(s - max) (one packed FMA and one packed add per two scores,
//               one ex2.approx each) written as packed 16-bit pairs over the first 64 columns of the SAME S
//               buffer (the tensor pipe runs its MMAs in issue order, so S(j+1) does not overwrite P(j) before
//               P V has read it). After a row's first tiles the maximum that P is taken against moves only when the new one
//               exceeds it by more than 2^8: then the O row in TMEM is rescaled (tcgen05.ld / st). P and the row sums stay
//               below 2^8 times their usual range, the fp32 sums and the final division are exact in that factor.
//
// What bounds it: per tile of 128 x 128 the two MMAs take 1024 cycles of the tensor pipe and the 16384 exponentials
// 1024 cycles of the MUFU. With one query tile per CTA and two threads per row (the previous split) the softmax of a tile
// lay open next to its MMAs and the two threads of a row met in shared memory twice: about 3000 cycles per tile
// (8192 tokens, 32 / 8 heads, causal, bf16: 736 us). Two tiles in turn, one thread per row: 549 us, with the MMAs issued eight
// to a statement 511 (both with their inputs in L2, the second is 554 from HBM), with the loads' waits out of the chain 540 from
// HBM; 3000 tokens, full attention, fp16, which the mma.sync kernel took before: 603, 187, 178, 174 us.
// An item's start and end cost about 9000 cycles each time, next to 3500 a pair of tiles: with its tiles counted in closed form instead of by walking
// and the output stored by rows 554 -> 541 us, 3000 tokens 180 -> 176 (both under the power cap); three-operand maxima: by keys, 2304
// tokens, 8 heads, causal 31.1 -> 29.2. A pair of tiles now (cycles, one tile's chain): load 150, maximum 410, exponentials 1350, P 190,
// to the issuing warp 100, P V and S until the next softmax sees it 1290. Outside this chain remain about 20 k cycles an item (of 928 k cycles an SM 8192 tokens
// spend 785 k in it, of 316 k 3000 tokens 251 k): the softmax warps rescale O early on, read it, scale and store it, and only then take the next item's scores.
// Slower were: 64-key halves with S double-buffered (more MMAs to issue: 746), P released to the MMAs in halves (541 -> 572 under the power cap), part of the
// exponentials as a polynomial on the FMA pipe (the softmax warps are short of issue slots).
// The two tiles are two query heads of one K/V head group where the group is even (same keys, no work done twice or
// for padding), else two neighbouring tiles of 128 queries of one head. Items are handed out longest first, in
// alternating direction, so that a causal mask leaves no CTA with the long items at the end.
//
// Few query tiles (kByKeys; at most one per SM, under a causal mask on one rank two): an item is ONE query tile, and its key tiles go
// in turn to the CTA's two places, each with its own S, O, maximum and sum; at the end each place's warps merge 64 columns of the
// two O in TMEM. With the softmax of one place only, softmax, P V and S of a tile were a serial chain, slower than the
// previous split of this kernel (8 heads, causal, us, that / one place / by keys: 512 tokens 14.6 / 15.6 / 11.7, 1024 tokens
// 19.5 / 22.9 / 16.4, 2304 tokens 34.8 / 41.7 / 27.1). What a short sequence spends outside its tiles counts too: K, V and Q have a
// producer warp each, the tensor maps are prefetched, and the output goes out by rows through shared memory.
//
// Sequences that are not a multiple of 128: the last tile's rows and keys past the end come back as zeros from TMA
// (the ring buffer is mapped block by block for that), its scores are masked and its rows are not stored.
//
// TMEM: S0 / P0 columns [0, 128), S1 / P1 [128, 256), O0 [256, 384), O1 [384, 512). Shared memory: Q 2 x 32 KB,
// K 2 x 32 KB, V 2 x 32 KB, output rows 16 KB. Every wait (mbarriers, arrival counters) is bounded.
#include "ring_attention_common.cuh"

#include "iris/gemm/sm100_mainloop.cuh"
#include "launch_pdl.cuh"
#include <type_traits>

using namespace iris;
using namespace iris_ring;
using iris::gemm::desc_kmajor;
using iris::gemm::desc_mnmajor;
using iris::gemm::make_idesc;

namespace {

constexpr int kTQ = 128;                 // queries per item = TMEM lanes
constexpr int kTK = 128;                 // keys per tile
constexpr int kTcThreads = 384;          // three warpgroups: issuers (two of four warps work), softmax of query tile 0, of tile 1
constexpr int kHalf = 128 * 128;         // bytes of a [128 rows][64 columns] 16-bit half tile
constexpr int kTile = 2 * kHalf;         // 32 KB
constexpr int kKvStages = 2;
constexpr int kStageOut = 32 * 64;       // bytes a softmax warp stages its output rows in, 32 columns at a time
// Q tiles, K and V stages, barriers, (m, l) of both places (by keys), output rows
constexpr int kTcSmem = 1024 + kTile * 2 + kTile * 2 * kKvStages + 256 + 2 * 128 * 8 + 8 * kStageOut;
constexpr float kRescaleAt = 8.f;        // log2 of how far a row's maximum may run ahead of the one P is taken against
// ... while the tile's number among its row's is below this it may not: a row's largest weight is exactly 1 then and loses nothing when P
// is rounded, which counts most where few keys share the weight. Error against 64 bits (2-norm) of 8192 tokens, causal, bf16: 2.13e-3
// with kRescaleAt everywhere, 2.10e-3 with 8, 2.09e-3 when O is always rescaled (the kernel with one query tile did that);
// time with inputs in L2 467, 484, 530 us. By keys (short rows) always: 512 tokens 2.25e-3 -> 2.18e-3, within 3 % of the time.
constexpr int kExactTiles = 8;
constexpr uint64_t kWaitNs = 4000000000ull;
static_assert(kTcSmem <= 227 * 1024, "shared memory budget");

struct TcArgs {
  RingArgs a;
  int by_head;           // 1: an item's two query tiles are two heads of one group, 0: two neighbouring tiles of one head
  CUtensorMap tmQ;       // [S, Hq * D], box 64 x 128
  CUtensorMap tmKown;    // [1][S, Hkv * D], box 64 x 128 x 1
  CUtensorMap tmVown;    // [1][S, Hkv * D], box 64 x 64 x 1
  CUtensorMap tmKbuf;    // ring buffer seen as [2 * W * 2][S, Hkv * D], box 64 x 128 x 1
  CUtensorMap tmVbuf;    // same, box 64 x 64 x 1
};

__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The eight MMAs of one 128 x 128 x 128 product, issued by one elected lane of a converged warp in one statement: K steps
// of 16, whose descriptors lie constant distances apart (in 16-byte units). One elect, one add per operand: with the
// descriptor of every step computed from its address and an elect each, an MMA cost the issuing warp about 100 cycles and this
// warp, not the tensor pipe (64 cycles per MMA) or the softmax, set the pace.
// S = Q K^T: both operands [128 rows][64 + 64 columns] in shared memory, K-major.
__device__ __forceinline__ void mma_s_elect(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a;\n\t.reg .b64 b;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.s64 a, %1, 0;\n\tadd.s64 b, %2, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t"
      "add.s64 a, %1, 2;\n\tadd.s64 b, %2, 2;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 4;\n\tadd.s64 b, %2, 4;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 6;\n\tadd.s64 b, %2, 6;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 1024;\n\tadd.s64 b, %2, 1024;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 1026;\n\tadd.s64 b, %2, 1026;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 1028;\n\tadd.s64 b, %2, 1028;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "add.s64 a, %1, 1030;\n\tadd.s64 b, %2, 1030;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
      "}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// O += P V: P from TMEM (lane = row, 16-bit pairs along K per column), V in 64-key halves, MN-major.
__device__ __forceinline__ void mma_pv_elect(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q, t;\n\t.reg .b32 a;\n\t.reg .b64 b;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
      "add.s32 a, %1, 0;\n\tadd.s64 b, %2, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, p;\n\t"
      "add.s32 a, %1, 8;\n\tadd.s64 b, %2, 128;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "add.s32 a, %1, 16;\n\tadd.s64 b, %2, 256;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "add.s32 a, %1, 24;\n\tadd.s64 b, %2, 384;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "add.s32 a, %1, 32;\n\tadd.s64 b, %2, 1024;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "add.s32 a, %1, 40;\n\tadd.s64 b, %2, 1152;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "add.s32 a, %1, 48;\n\tadd.s64 b, %2, 1280;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "add.s32 a, %1, 56;\n\tadd.s64 b, %2, 1408;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [a], b, %3, t;\n\t"
      "}" ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 3-D tiled load by one elected lane of a converged warp (see the *_elect forms of ptx.cuh).
__device__ __forceinline__ void tma_load_3d_elect(uint32_t smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
      "@q cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}" ::"r"(smem_dst),
      "l"(m), "r"(ptx::smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}

// One item: two query tiles (qt[i], head h[i]) of one K/V head. n_q: how many of them exist (an odd number of
// query tiles leaves the last item with one). By keys: one query tile, whose key tiles the two places share, and one item per CTA.
struct Item {
  int qt[2], h[2], kvh, n_q;
};
template <bool kByKeys>
struct ItemOrder {
  int items, rounds, stride, c, per_q, q_tiles, Hq, group;
  bool by_head;
  __device__ ItemOrder(const RingArgs& a, int by_head_) {
    q_tiles = (a.S + kTQ - 1) / kTQ;
    Hq = a.Hq;
    group = a.Hq / a.Hkv;
    by_head = !kByKeys && by_head_ != 0;
    per_q = by_head ? Hq / 2 : Hq;
    items = (by_head || kByKeys ? q_tiles : (q_tiles + 1) / 2) * per_q;
    stride = gridDim.x - a.n_comm;
    c = blockIdx.x - a.n_comm;
    rounds = (items + stride - 1) / stride;
  }
  // the CTA's item of a round; false when the last round has none for it. Longest items (late queries) first.
  __device__ bool get(int round, Item& it) const {
    const int idx = round * stride + ((round & 1) ? stride - 1 - c : c);
    if (idx >= items) return false;
    const int q = items / per_q - 1 - idx / per_q, hh = idx % per_q;
    if (by_head) {
      it.qt[0] = it.qt[1] = q;
      it.h[0] = 2 * hh; it.h[1] = 2 * hh + 1;
      it.n_q = 2;
    } else if (kByKeys) {
      it.qt[0] = it.qt[1] = q;
      it.h[0] = it.h[1] = hh;
      it.n_q = 2;
    } else {
      it.qt[0] = 2 * q; it.qt[1] = 2 * q + 1;
      it.h[0] = it.h[1] = hh;
      it.n_q = it.qt[1] < q_tiles ? 2 : 1;
    }
    it.kvh = it.h[0] / group;
    return true;
  }
};

// The key tiles of one item, in the order every role walks them: blocks in arrival order (own,
// r-1, r-2, ...), tiles inside a block in order; causal items skip what lies after their queries. A tile is
// visited when one of the item's query tiles needs it; needs(i) says which. By keys, place 0 takes the first, third, ... tile of
// the walk and place 1 the others.
//
// Contiguous layout: rank r holds tokens [r*S, (r+1)*S). A causal item of query tile qt takes all
// tiles of earlier blocks, tiles 0..qt of its own block (the last one masked on the diagonal) and
// nothing of later blocks - so the last rank does W times the work of the first.
// Zigzag layout: the sequence is cut into 2W chunks of S/2 tokens and rank r holds chunks r and
// 2W-1-r (its block = [chunk r | chunk 2W-1-r]). Under a causal mask a query of chunk r sees
// chunks 0..r, a query of chunk 2W-1-r sees every first-half chunk and the second-half chunks
// of origins >= r: every rank does the same amount of work.
template <bool kByKeys>
struct TileWalk {
  int W, r, T, causal, zigzag;
  int qt[2], n_q;
  int step = 0, t = -1, origin = 0;
  int b0 = 0;                              // second range of a block starts here (first range ends at or before it)
  int a1[2], b1[2];                        // query tile i takes [0, a1[i]) and [b0, b1[i]) of the current block
  int ua1 = 0, ub1 = 0;                    // their union
  int n = -1;                              // tiles taken before this one (counted by keys only)
  bool first = false;                      // the current tile is the first one taken from its block
  __device__ TileWalk(const RingArgs& a, const Item& it)
      : W(a.ctx.world), r(a.ctx.rank), T((a.S + kTK - 1) / kTK), causal(a.causal), zigzag(a.zigzag), n_q(it.n_q) {
    qt[0] = it.qt[0]; qt[1] = it.qt[1];
    open_block();
  }
  __device__ void ranges() {
    const int Th = T / 2;
    b0 = causal && zigzag ? Th : T;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a1[i] = T; b1[i] = b0;                 // (b1[i] >= b0 always)
      if (i >= n_q) { a1[i] = 0; continue; }
      if (!causal) continue;
      if (!zigzag) a1[i] = origin > r ? 0 : origin == r ? qt[i] + 1 : T;
      else if (qt[i] < Th) a1[i] = origin > r ? 0 : origin == r ? qt[i] + 1 : Th;   // query chunk r: first halves of origins <= r
      else {                                                                        // query chunk 2W-1-r: every first half, second halves of origins >= r
        a1[i] = Th;
        b1[i] = origin > r ? T : origin == r ? qt[i] + 1 : b0;
      }
    }
    ua1 = max(a1[0], a1[1]); ub1 = max(b1[0], b1[1]);
  }
  __device__ void open_block() {
    for (; step < W; ++step) {
      origin = r - step;
      if (origin < 0) origin += W;
      ranges();
      if (ua1 > 0 || ub1 > b0) { t = -1; return; }
    }
  }
  // tiles of the whole walk: query tile 0's, query tile 1's, and all. (Counted by walking, at 93 cycles a tile, they held back the
  // first product of an item of 63 tiles by 6000 cycles.)
  __device__ void count(int& n0, int& n1, int& all) {
    n0 = n1 = all = 0;
    for (step = 0; step < W; ++step) {
      origin = r - step;
      if (origin < 0) origin += W;
      ranges();
      n0 += a1[0] + b1[0] - b0; n1 += a1[1] + b1[1] - b0; all += ua1 + ub1 - b0;
    }
  }
  // advances to the next tile; false when the item is finished
  __device__ bool next() {
    while (step < W) {
      first = t < 0;
      if (t < 0) t = ua1 > 0 ? 0 : b0;
      else if (++t == ua1 && ub1 > b0) t = b0;
      if (t < ua1 || (t >= b0 && t < ub1)) {
        if (kByKeys) ++n;
        return true;
      }
      ++step;
      open_block();
    }
    return false;
  }
  // (selected, not indexed: an index that is not a constant would put the arrays in local memory)
  __device__ bool needs(int i) const { return kByKeys ? (n & 1) == i : t < (i ? a1[1] : a1[0]) || (t >= b0 && t < (i ? b1[1] : b1[0])); }
  __device__ bool diagonal(int i) const { return causal && origin == r && t == (i ? qt[1] : qt[0]); }
};

// kScaleFirst: a scale that is not positive is applied before the mask and the maximum (0 times a masked -inf is NaN, a negative
// factor turns maximum and mask round); a positive one changes neither and goes into the exponentials' FMA.
template <bool kFp16, bool kScaleFirst, bool kByKeys>
__device__ void attn_main_tc(const TcArgs& g, uint8_t* smem_raw, int call) {
  using TileWalk = ::TileWalk<kByKeys>;
  const RingArgs& a = g.a;
  const DeviceContext& ctx = a.ctx;
  const int W = ctx.world, r = ctx.rank;
  const int par = call & 1;
  const int32_t target = ((call >> 1) + 1) * a.n_comm;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* q_s = smem;                                   // [2][kTile]
  uint8_t* k_s = q_s + 2 * kTile;                        // [stages][kTile]
  uint8_t* v_s = k_s + kKvStages * kTile;
  uint64_t* bars = (uint64_t*)(v_s + kKvStages * kTile);
  uint64_t* q_full = bars;              // [2] the item's Q tile i has landed
  uint64_t* q_free = bars + 2;          // [2] every S MMA of the item has read Q tile i
  uint64_t* k_full = bars + 4;          // [2]
  uint64_t* k_empty = bars + 6;         // [2]
  uint64_t* v_full = bars + 8;          // [2]
  uint64_t* v_empty = bars + 10;        // [2]
  uint64_t* s_full = bars + 12;         // [2] by query tile: its S is complete (and its P V of the tile before)
  uint64_t* p_full = bars + 14;         // [2] by query tile: 4 softmax warps wrote P (and rescaled O)
  uint64_t* o_full = bars + 16;         // [2] the item's O_i is complete
  uint64_t* o_free = bars + 18;         // [2] 4 softmax warps have read the item's O_i
  uint32_t* tmem_slot = (uint32_t*)(bars + 20);
  float2* ml = (float2*)((uint8_t*)bars + 256);          // [2][128] by keys: a place's maximum and sum per row

  if (kByKeys && warp == 2 && lane < 3)     // the first loads of a short sequence would wait for the maps one by one
    ptx::prefetch_tmap(lane == 0 ? &g.tmQ : lane == 1 ? &g.tmKown : &g.tmVown);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&q_full[i], 1); ptx::mbar_init(&q_free[i], 1);
      ptx::mbar_init(&s_full[i], 1); ptx::mbar_init(&p_full[i], 4);
      ptx::mbar_init(&o_full[i], 1); ptx::mbar_init(&o_free[i], 4);
    }
    for (int i = 0; i < kKvStages; ++i) {
      ptx::mbar_init(&k_full[i], 1); ptx::mbar_init(&k_empty[i], 1);
      ptx::mbar_init(&v_full[i], 1); ptx::mbar_init(&v_empty[i], 1);
    }
    ptx::fence_mbar_init();
    ptx::fence_proxy_async();
  }
  if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, 512);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *(volatile uint32_t*)tmem_slot;
  if constexpr (kByKeys) ptx::pdl_trigger();
  const ItemOrder<kByKeys> order(a, g.by_head);

  // 72 + 216 + 216 = 3 x 168, what the block was launched with (the splits stand at the head of their branches:
  // the compiler gives each branch its own budget from there). The compiler still keeps a few words of walk state on the stack.
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  if (warp == 0 || (kByKeys && warp != 1)) {
    // ------------------------------------------------------------------ TMA producer (by keys three: warp 0 K, warp 2 V, warp 3 Q;
    // K is loaded as soon as its stage is read then, not behind V of the tile before, whose stage is free much later)
    unsigned arrived_mask = 1u << r;
    uint32_t n_tile = 0;                    // K/V tiles issued so far (barrier phases)
    uint32_t n_q[2] = {0, 0};               // Q tiles loaded so far, per place
    bool ok = true;
    Item item;
    for (int rd = 0; rd < order.rounds && ok; ++rd) {
      if (!order.get(rd, item)) continue;
      if (!kByKeys || warp == 3) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (i >= (kByKeys ? 1 : item.n_q) || !ok) break;          // (by keys both places use Q tile 0)
          if (!__all_sync(0xffffffffu, ptx::mbar_wait(&q_free[i], (n_q[i] & 1) ^ 1, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; break; }
          const uint32_t qd = ptx::smem_u32(q_s + i * kTile);
          ptx::mbar_expect_tx_elect(&q_full[i], kTile);
          ptx::tma_load_2d_elect(qd, &g.tmQ, &q_full[i], item.h[i] * kD, item.qt[i] * kTQ);
          ptx::tma_load_2d_elect(qd + kHalf, &g.tmQ, &q_full[i], item.h[i] * kD + 64, item.qt[i] * kTQ);
          ++n_q[i];
        }
        if (kByKeys) continue;
      }
      TileWalk w(a, item);
      while (ok && w.next()) {
        if (w.first && !((arrived_mask >> w.origin) & 1u)) {
          int seen = 1;
          if (lane == 0) seen = wait_flag_ge(ctx, a.flags + (size_t)par * W + w.origin, target) ? 1 : 0;
          seen = __shfl_sync(0xffffffffu, seen, 0);
          if (!seen) { ok = false; break; }
          ptx::fence_proxy_async();
          arrived_mask |= 1u << w.origin;
        }
        const int st = n_tile % kKvStages;
        const uint32_t ph = ((n_tile / kKvStages) & 1) ^ 1;
        const bool own = w.origin == r;
        const CUtensorMap* mk = own ? &g.tmKown : &g.tmKbuf;
        const CUtensorMap* mv = own ? &g.tmVown : &g.tmVbuf;
        const int zk = own ? 0 : (par * W + w.origin) * 2;       // ring buffer blocks: (parity, origin, K | V)
        const int zv = own ? 0 : zk + 1;
        const int pos0 = w.t * kTK;
        const uint32_t kd = ptx::smem_u32(k_s + st * kTile);
        const uint32_t vd = ptx::smem_u32(v_s + st * kTile);
        if (!kByKeys || warp == 0) {
          if (!__all_sync(0xffffffffu, ptx::mbar_wait(&k_empty[st], ph, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; break; }
          ptx::mbar_expect_tx_elect(&k_full[st], kTile);
          tma_load_3d_elect(kd, mk, &k_full[st], item.kvh * kD, pos0, zk);
          tma_load_3d_elect(kd + kHalf, mk, &k_full[st], item.kvh * kD + 64, pos0, zk);
        }
        if (!kByKeys || warp == 2) {
          if (!__all_sync(0xffffffffu, ptx::mbar_wait(&v_empty[st], ph, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; break; }
          ptx::mbar_expect_tx_elect(&v_full[st], kTile);
#pragma unroll
          for (int kh = 0; kh < 2; ++kh)
#pragma unroll
            for (int nb = 0; nb < 2; ++nb)
              tma_load_3d_elect(vd + kh * kHalf + nb * 8192, mv, &v_full[st], item.kvh * kD + nb * 64, pos0 + kh * 64, zv);
        }
        ++n_tile;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    const uint32_t idesc_s = make_idesc(kTK, !kFp16, false);     // B = K tile, K-major
    const uint32_t idesc_o = make_idesc(kD, !kFp16, true);       // B = V tile, [keys, d] row-major
    // The warp stays converged: every lane computes the warp-uniform operands and each tensor-core instruction
    // elects its issuing lane (issued from inside `if (lane == 0)` they cost about 100 cycles apiece). Votes and
    // the warp reduction make the loop state and the TMEM base uniform for the compiler too.
    const uint32_t tmem_u = __reduce_or_sync(0xffffffffu, tmem_base);
    uint32_t n_k = 0, n_v = 0;                     // K / V tiles taken so far
    uint32_t n_qi[2] = {0, 0}, n_p[2] = {0, 0};    // items / P tiles per query tile so far
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t phase) {
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(bar, phase, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; }
      return ok;
    };
    Item item;
    for (int rd = 0; rd < order.rounds && ok; ++rd) {
      if (!order.get(rd, item)) continue;
      if constexpr (kByKeys) {
        // S of the walk's tiles j + 1 and j + 2 is issued while the softmax works on tile j
        int n, n0, n1;
        TileWalk(a, item).count(n0, n1, n);
        if (!wait(&q_full[0], 0)) break;
        const uint32_t qb = ptx::smem_u32(q_s);
        auto wait_k = [&]() { return wait(&k_full[n_k % kKvStages], (n_k / kKvStages) & 1); };
        auto issue_s = [&](int i) {
          const int st = n_k % kKvStages;
          ptx::tc_fence_after();
          mma_s_elect(tmem_u + i * 128, desc_kmajor(qb), desc_kmajor(ptx::smem_u32(k_s + st * kTile)), idesc_s, 0);
          ptx::mma_commit_elect(&s_full[i]);
          ptx::mma_commit_elect(&k_empty[st]);
          ++n_k;
        };
        if (!wait_k()) break;
        issue_s(0);
        if (n > 1) {
          if (!wait_k()) break;
          issue_s(1);
        }
        for (int j = 0; j < n; ++j) {
          const int i = j & 1, st = j % kKvStages;
          // (P's wait comes last, see below)
          if (!wait(&v_full[st], (j / kKvStages) & 1) || (j + 2 < n && !wait_k()) || !wait(&p_full[i], (j >> 1) & 1)) break;
          ptx::tc_fence_after();
          mma_pv_elect(tmem_u + 256 + i * 128, tmem_u + i * 128, desc_mnmajor(ptx::smem_u32(v_s + st * kTile)), idesc_o, j >= 2);
          if (j >= n - 2) ptx::mma_commit_elect(&o_full[i]);
          ptx::mma_commit_elect(&v_empty[st]);
          if (j + 2 < n) issue_s(i);
        }
        break;
      }
      int left_s[2], left_pv[2], all;               // S and P V MMAs of the item still to be issued, per query tile
      TileWalk(a, item).count(left_s[0], left_s[1], all);
      left_pv[0] = left_s[0]; left_pv[1] = left_s[1];
      const int total[2] = {left_s[0], left_s[1]};
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (i < item.n_q && ok) wait(&q_full[i], n_qi[i] & 1);
      auto issue_s = [&](int i, int st) {
        ptx::tc_fence_after();
        const uint32_t qb = ptx::smem_u32(q_s + i * kTile), kb = ptx::smem_u32(k_s + st * kTile);
        mma_s_elect(tmem_u + i * 128, desc_kmajor(qb), desc_kmajor(kb), idesc_s, 0);
        ptx::mma_commit_elect(&s_full[i]);
        if (--left_s[i] == 0) ptx::mma_commit_elect(&q_free[i]);
      };
      auto issue_pv = [&](int i, int st) {
        ptx::tc_fence_after();
        const uint32_t vb = ptx::smem_u32(v_s + st * kTile);
        const bool clear = left_pv[i] == total[i];
        // P: 16 keys = 8 columns of 16-bit pairs at the start of the tile's S buffer
        mma_pv_elect(tmem_u + 256 + i * 128, tmem_u + i * 128, desc_mnmajor(vb), idesc_o, !clear);
        if (--left_pv[i] == 0) ptx::mma_commit_elect(&o_full[i]);
      };
      TileWalk cur(a, item), nxt(a, item);
      bool has = cur.next(), has_n = nxt.next();
      // S of the first tile
      if (ok && has && wait(&k_full[n_k % kKvStages], (n_k / kKvStages) & 1)) {
        const int st = n_k % kKvStages;
        if (cur.needs(0)) issue_s(0, st);
        if (cur.needs(1)) issue_s(1, st);
        ptx::mma_commit_elect(&k_empty[st]);
        ++n_k;
      }
      while (ok && has) {
        has_n = nxt.next();
        const int vst = n_v % kKvStages, kst = n_k % kKvStages;
        // (the loads' waits stand in front of P's: a wait costs this warp some 200 cycles even when it is over, and what follows P
        // is the chain that sets the pace. 8192 tokens, 32 / 8 heads, causal, inputs in L2: 485 us with them behind it, now 467.)
        if (!wait(&v_full[vst], (n_v / kKvStages) & 1) || (has_n && !wait(&k_full[kst], (n_k / kKvStages) & 1))) break;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          if (cur.needs(i)) {
            if (!wait(&p_full[i], n_p[i] & 1)) break;
            // the previous item's O must have been read out before this item's first P V overwrites it
            if (left_pv[i] == total[i] && !wait(&o_free[i], (n_qi[i] & 1) ^ 1)) break;
            issue_pv(i, vst);
            ++n_p[i];
          }
          if (cur.needs(i) && (i == 1 || !cur.needs(1))) ptx::mma_commit_elect(&v_empty[vst]);      // the tile's last P V
          if (has_n && nxt.needs(i)) {
            issue_s(i, kst);
          }
        }
        if (!ok) break;
        ++n_v;
        if (has_n) { ptx::mma_commit_elect(&k_empty[kst]); ++n_k; }
        has = has_n;
        cur.next();
      }
      ++n_qi[0];
      if (item.n_q > 1) ++n_qi[1];
    }
  }
  } else {
    // ------------------------------------------------------------------ softmax / correction / epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    const int quarter = warp & 3;
    const int i = (warp - 4) >> 2;                            // query tile of the item
    const int row = quarter * 32 + lane;                      // query row inside the tile
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const uint32_t s_addr = lane_addr + i * 128, o_addr = lane_addr + 256 + i * 128;
    const float scale2 = kScaleFirst ? 1.f : a.sm_scale * kLog2e;
    const unsigned long long scale_pair = pack_f32x2(scale2, scale2);
    uint32_t n_item = 0, n_tile = 0;
    bool ok = true;
    Item item;
    // The warp's 32 rows go out through shared memory, 32 columns (64 bytes) of a row by four lanes: with a row per lane every
    // 16-byte store instruction touched 32 lines, and an item's output took 3700 cycles. 16-byte pieces, XORed by half the
    // row so that eight rows written and two rows read together meet different banks.
    uint8_t* stage = (uint8_t*)(ml + 2 * 128) + (warp - 4) * kStageOut;
    auto put_rows = [&](const uint32_t (&o)[32], int c, int q_tile, int h) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        *(uint4*)(stage + lane * 64 + ((e ^ ((lane >> 1) & 3)) << 4)) =
            make_uint4(pack2<kFp16>(__uint_as_float(o[8 * e]), __uint_as_float(o[8 * e + 1])), pack2<kFp16>(__uint_as_float(o[8 * e + 2]), __uint_as_float(o[8 * e + 3])),
                       pack2<kFp16>(__uint_as_float(o[8 * e + 4]), __uint_as_float(o[8 * e + 5])), pack2<kFp16>(__uint_as_float(o[8 * e + 6]), __uint_as_float(o[8 * e + 7])));
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int rr = k * 8 + (lane >> 2), e = lane & 3, pos = q_tile * kTQ + quarter * 32 + rr;
        if (pos < a.S)
          *(uint4*)(a.out + ((size_t)pos * a.Hq + h) * kD * 2 + c * 64 + e * 16) = *(const uint4*)(stage + rr * 64 + ((e ^ ((rr >> 1) & 3)) << 4));
      }
      __syncwarp();
    };
    for (int rd = 0; rd < order.rounds && ok; ++rd) {
      if (!order.get(rd, item)) continue;
      if (i >= item.n_q) continue;
      const int qpos = (i ? item.qt[1] : item.qt[0]) * kTQ + row;                // position inside this rank's block
      const int head = i ? item.h[1] : item.h[0];
      float m_run = -INFINITY;                                // what P is taken against (log2 units)
      unsigned long long l_pair[2] = {0ull, 0ull};            // the row sum, in four parts
      int j = 0;
      TileWalk w(a, item);
      while (w.next()) {
        if (!w.needs(i)) continue;
        if (!__all_sync(0xffffffffu, ptx::mbar_wait(&s_full[i], n_tile & 1, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; break; }
        ptx::tc_fence_after();
        uint32_t s[128];
#pragma unroll
        for (int c = 0; c < 4; ++c) ptx::tmem_ld_32x32(s_addr + c * 32, *reinterpret_cast<uint32_t (*)[32]>(&s[c * 32]));
        ptx::tmem_ld_wait();
        if constexpr (kScaleFirst) {
#pragma unroll
          for (int c = 0; c < 128; ++c) s[c] = __float_as_uint(__uint_as_float(s[c]) * (a.sm_scale * kLog2e));
        }
        // causal mask on the diagonal tile, keys past the end of the block in its last tile
        int lim = a.S - 1 - w.t * kTK;
        if (w.diagonal(i)) lim = min(lim, qpos - w.t * kTK);
        if (__any_sync(0xffffffffu, lim < kTK - 1)) {
#pragma unroll
          for (int c = 0; c < 128; ++c)
            if (c > lim) s[c] = 0xff800000u;     // -inf
        }
        float mx4[4];             // four chains: the maximum is latency bound otherwise
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = max3(__uint_as_float(s[u]), __uint_as_float(s[4 + u]), __uint_as_float(s[8 + u]));
#pragma unroll
        for (int c = 12; c + 7 < 128; c += 8) {
#pragma unroll
          for (int u = 0; u < 4; ++u) mx4[u] = max3(mx4[u], __uint_as_float(s[c + u]), __uint_as_float(s[c + 4 + u]));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) mx4[u] = fmaxf(mx4[u], __uint_as_float(s[124 + u]));
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale2;     // (the first tile holds a key the row sees)
        float alpha = 1.f;
        if (j == 0) m_run = mx;
        else if (mx > m_run + (kByKeys || j < kExactTiles ? 0.f : kRescaleAt)) { alpha = ex2_approx(m_run - mx); m_run = mx; }
        // rescale O when some row of this warp moved its maximum (this tile's S was issued after the previous tile's
        // P V, and its barrier covers both: O holds every earlier tile)
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
          const unsigned long long al = pack_f32x2(alpha, alpha);
#pragma unroll
          for (int u = 0; u < 2; ++u) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(l_pair[u]) : "l"(al));
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t o[32];
            ptx::tmem_ld_32x32(o_addr + c * 32, o);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st_32x32(o_addr + c * 32, o);
          }
        }
        // p = exp2(s * scale - max): packed FMA for two scores at a time, one ex2.approx each, packed sums. P goes over
        // the first 64 columns of the tile's S buffer: every thread of the row (this one) has read its scores
        const float neg_m = fminf(-m_run, 3e38f);      // finite where every key so far scores -inf: their P is 0, not NaN
        const unsigned long long negm_pair = pack_f32x2(neg_m, neg_m);
        unsigned long long rs[2] = {0ull, 0ull};
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t pw[32];        // 64 probabilities as 16-bit pairs
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int c = hf * 64 + 2 * e;
            unsigned long long sp, xp;
            asm("mov.b64 %0, {%1, %2};" : "=l"(sp) : "r"(s[c]), "r"(s[c + 1]));
            asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(xp) : "l"(sp), "l"(scale_pair), "l"(negm_pair));
            float x0, x1;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(xp));
            const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
            asm("add.rn.f32x2 %0, %0, %1;" : "+l"(rs[e & 1]) : "l"(pack_f32x2(p0, p1)));
            pw[e] = pack2<kFp16>(p0, p1);
          }
          tmem_st_32x32(s_addr + hf * 32, pw);
        }
        tmem_st_wait();                         // P (and a rescaled O) are in TMEM before the MMA is told
        ptx::tc_fence_before();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&p_full[i]);
#pragma unroll
        for (int u = 0; u < 2; ++u) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(l_pair[u]) : "l"(rs[u]));
        ++n_tile;
        ++j;
      }
      if (!ok && !kByKeys) break;                             // (by keys the other place waits for this one at a barrier)
      // ---- item epilogue: the row sum, the last P V, O / sum -> 16-bit -> global
      float l_all = 0.f;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float x0, x1;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(l_pair[u]));
        l_all += x0 + x1;
      }
      if constexpr (kByKeys) {
        // Both places' warps of a quarter reach the same TMEM lanes, so each merges 64 columns of the two O; only the
        // rows' maxima and sums go through shared memory. An item of one key tile is place 0's alone.
        const int n = w.n + 1;
        const bool both = n > 1, mine = both || i == 0;
        ml[i * 128 + row] = make_float2(m_run, l_all);
        for (int k = 0; k < (both ? 2 : 1); ++k)
          if (ok && !__all_sync(0xffffffffu, ptx::mbar_wait(&o_full[k], 0, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; }
        ptx::named_barrier(1, 256);
        ptx::tc_fence_after();
        if (ok && mine) {
          float m = m_run, l = l_all, w_own = 1.f, w_other = 0.f;
          if (both) {
            const float2 other = ml[(i ^ 1) * 128 + row];
            m = fmaxf(m_run, other.x);
            w_own = m_run == -INFINITY ? 0.f : ex2_approx(m_run - m);
            w_other = other.x == -INFINITY ? 0.f : ex2_approx(other.x - m);
            l = l_all * w_own + other.y * w_other;
          }
          const float inv = l > 0.f ? 1.f / l : 0.f;
          w_own *= inv; w_other *= inv;
          const uint32_t other_addr = lane_addr + 256 + (i ^ 1) * 128;
          const int c0 = both ? 2 * i : 0, c1 = both ? c0 + 2 : 4;
#pragma unroll 1
          for (int c = c0; c < c1; ++c) {
            uint32_t o[32], o2[32];
            ptx::tmem_ld_32x32(o_addr + c * 32, o);
            if (both) ptx::tmem_ld_32x32(other_addr + c * 32, o2);
            ptx::tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 32; ++e) {
              float f = __uint_as_float(o[e]) * w_own;
              if (both) f += __uint_as_float(o2[e]) * w_other;
              o[e] = __float_as_uint(f);
            }
            put_rows(o, c, item.qt[0], head);
          }
          if (a.lse && i == 0 && qpos < a.S) a.lse[(size_t)qpos * a.Hq + head] = l > 0.f ? (m + log2f(l)) / kLog2e : -INFINITY;
        }
        break;
      }
      if (!__all_sync(0xffffffffu, ptx::mbar_wait(&o_full[i], n_item & 1, kWaitNs))) { ctx.fail(kTimeoutPipeline); ok = false; break; }
      ptx::tc_fence_after();
      const float inv = l_all > 0.f ? 1.f / l_all : 0.f;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        ptx::tmem_ld_32x32(o_addr + c * 32, o);
        ptx::tmem_ld_wait();
        if (c == 3) {                           // O is in registers: the next item's first P V may overwrite it
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&o_free[i]);
        }
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * inv);
        put_rows(o, c, i ? item.qt[1] : item.qt[0], head);
      }
      if (a.lse && qpos < a.S) a.lse[(size_t)qpos * a.Hq + head] = l_all > 0.f ? (m_run + log2f(l_all)) / kLog2e : -INFINITY;
      ++n_item;
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  if (warp == 1) ptx::tmem_dealloc(tmem_base, 512);
}

template <bool kFp16, bool kScaleFirst, bool kByKeys>
__global__ void __launch_bounds__(kTcThreads, 1) ring_attention_tc_kernel(const __grid_constant__ TcArgs g) {
  extern __shared__ __align__(128) uint8_t smem[];
  if constexpr (kByKeys) ptx::pdl_wait();      // (see the launch)
  const int call = *(volatile int32_t*)&g.a.state[0];
  if ((int)blockIdx.x < g.a.n_comm) comm_main(g.a, smem, kTcSmem, call);
  else attn_main_tc<kFp16, kScaleFirst, kByKeys>(g, smem, call);
  finish_call(g.a, call);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// blocks x [rows, cols] of 16-bit elements (blocks = 0: a 2-D map of one), box 64 x box_rows x 1: rows past the end of a block
// come back as zeros.
bool make_map16(CUtensorMap* m, const void* base, bool fp16, uint64_t blocks, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  static EncodeTiledFn enc = nullptr;
  if (!enc) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) return false;
    enc = (EncodeTiledFn)p;
  }
  if (((uint64_t)base & 15) || ((cols * 2) & 15)) return false;
  cuuint64_t dims[3] = {cols, rows, blocks};
  cuuint64_t strides[2] = {cols * 2, rows * cols * 2};
  cuuint32_t box[3] = {64, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, blocks ? 3 : 2, (void*)base, dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

namespace iris_ring {

int launch_ring_attention_tc(const RingArgs& a, cudaStream_t stream) {
  if (a.S <= 0) return 1;
  // One rank, one key tile: nothing to share or overlap, and the mma.sync CTAs with their 64 x 64 tiles are through earlier. Measured,
  // us, here / mma.sync, 8 heads, full attention: 32 tokens 7.8 / 6.2, 64 tokens 8.9 / 7.2, 128 tokens 7.9 / 8.4 (32 heads 9.0 / 8.8),
  // 129 tokens 9.3 / 10.0, 200 tokens 9.5 / 11.5, 256 tokens 9.3 / 11.7.
  if (a.ctx.world == 1 && !a.zigzag && a.S <= kTK) return 1;
  const int W = a.ctx.world;
  TcArgs g;
  g.a = a;
  const bool f16 = a.is_fp16 != 0;
  const uint64_t kvc = (uint64_t)a.Hkv * kD;
  if ((uint64_t)a.out & 15) return 1;    // output rows are written with 16-byte stores
  if (!make_map16(&g.tmQ, a.q, f16, 0, a.S, (uint64_t)a.Hq * kD, kTQ)) return 1;
  if (!make_map16(&g.tmKown, a.k, f16, 1, a.S, kvc, kTK)) return 1;
  if (!make_map16(&g.tmVown, a.v, f16, 1, a.S, kvc, 64)) return 1;
  if (W > 1) {
    if (!make_map16(&g.tmKbuf, a.kv_buf, f16, 4ull * W, a.S, kvc, kTK)) return 1;
    if (!make_map16(&g.tmVbuf, a.kv_buf, f16, 4ull * W, a.S, kvc, 64)) return 1;
  } else {
    g.tmKbuf = g.tmKown;
    g.tmVbuf = g.tmVown;
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int q_tiles = (a.S + kTQ - 1) / kTQ;
  // Key tiles shared by the places while every query tile can have an SM. Under a causal mask also when it takes two turns: the
  // second ones are the short ones, and of two-tile items there would be fewer than SMs (us, two-tile items / by keys:
  // 8 heads 2432 tokens 44.7 / 29.2, 4608 tokens 78.5 / 54.1, 32 heads 1024 tokens 26.2 / 26.2, 1280 tokens, 320 tiles 30.9 / 35.4;
  // full attention, 8 heads 2432 tokens 47.4 / 52.8). The turns need CTAs that wait for nobody: one rank.
  const int tiles = q_tiles * a.Hq;
  const bool by_keys = tiles <= sms - a.n_comm || (W == 1 && a.causal && tiles <= 2 * sms);
  g.by_head = (a.Hq / a.Hkv) % 2 == 0;
  const int items = by_keys ? tiles : g.by_head ? q_tiles * (a.Hq / 2) : (q_tiles + 1) / 2 * a.Hq;
  // one CTA per SM (212 KB of shared memory), all resident; by keys a CTA per item, which the SMs take in order (longest first)
  int attn = sms - a.n_comm;
  if (by_keys || attn > items) attn = items;
  if (attn < 1) return 1;
  const int grid = a.n_comm + attn;
  const bool scale_first = !(a.sm_scale > 0.f);
  auto pick = [&](auto fp16, auto first) -> void (*)(const TcArgs) {
    return by_keys ? ring_attention_tc_kernel<decltype(fp16)::value, decltype(first)::value, true>
                   : ring_attention_tc_kernel<decltype(fp16)::value, decltype(first)::value, false>;
  };
  using Y = std::true_type;
  using N = std::false_type;
  auto* kern = f16 ? (scale_first ? pick(Y{}, Y{}) : pick(Y{}, N{})) : (scale_first ? pick(N{}, Y{}) : pick(N{}, N{}));
  const int smem = kTcSmem;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -20;
  // Short calls start behind the stream's last kernel (512 tokens, 8 heads, causal 16.4 -> 15.6 us); the long ones have nothing to gain
  // (8192 tokens, 32 / 8 heads, causal 551 -> 558).
  if (W == 1 && by_keys) return launch_pdl(kern, dim3(grid), kTcThreads, smem, stream, g);
  kern<<<grid, kTcThreads, smem, stream>>>(g);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // namespace iris_ring
