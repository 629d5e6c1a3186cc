// Block-sparse attention on INT8 Q/K and an FP16 copy of the FP8 V carrier, for
// sm_100a.
//
// An item is a 128-row query tile of one head and that tile's list of 64-row KV tiles (or a part of
// it).  One CTA per SM walks item after item:
//   S = Q8 . K8^T      tcgen05.mma kind::i8, 128x64x128, Q8 in TMEM, int32 in TMEM
//   P = exp2(c*S - m)  FP32 in registers, one thread per query row, m an integer
//   O += P16 . V16     tcgen05.mma kind::f16, 128x128x64, P in TMEM, fp32 in TMEM
// V16 holds the E4M3 codes as FP16 (exact), so the product is that of the FP8
// carrier; P is rounded once to FP16 (relative error up to 2^-11).
//
// Why FP16 P.  The tensor pipe takes the same time for one 16-bit product as for two
// 8-bit products (the two E4M3 terms of attn_tc.cu), but a softmax thread needs one
// packed conversion per pair of scores instead of a mask, a residual and two
// conversions per score.  BF16 would do as well for speed and never overflow, but its
// eight bits lose precision: against 64-bit arithmetic on the same carriers the
// outputs of 11 layers (1960 to 33272 tokens, 10 to 100 %) were off by 1.64e-3 to 1.67e-3
// (relative 2-norm) with BF16, 1.19e-3 to 1.31e-3 with two E4M3 terms, 2.1e-4 to 2.3e-4
// with FP16.
//
// FP16 ends at 2^16 and 2^-24, and there is no running maximum: it would put two serial
// phases (maximum, O rescale) into every tile.  Instead m is fixed by the first two
// tiles: their row maximum becomes 2^-5, which leaves the rows 21 bits of room above
// and puts the last unit 19 bits below (two E4M3 terms: 16 to 19 bits below the largest
// score).  A row whose sum over a tile passes 65504 leaves that tile out (P = 0), and
// the tile is noted; when the list is through, O and the row sums are brought to a new m
// and the noted tiles, and only those, are walked again.  The walk begins in the middle of
// the list: a routed list has the context in front, and the tiles that were selected for
// their scores are the better measure.  Of 16 layers with scores of 4 bits standard
// deviation, held over groups of 64 tokens, 2 to 14 % of the query tiles (27 % in a dense one of
// 24792 tokens) came round again, with 0.03 to 0.5 % of all tiles; with the first tile of
// the list and 2^-7 it was 17 to 61 % and 1.5 to 9 %.  What it costs at 24 heads x 33272
// tokens, 30 %, launches in a row: 2.82 ms on inputs with a rank-8 part; 3.00 with one row of every query
// tile 48 bits ahead in every 40th tile; 3.43 with a third of the rows ahead in every tenth;
// two E4M3 terms take 4.4 to 4.5 ms of each.  All but the first two tiles of a list
// ahead is the worst: two walks, three where a sum overflows (120 bits): 24 heads x 9872,
// dense, 0.85 ms, then 2.21 and 2.86, where two E4M3 terms take 1.31, 1.12 and 1.10.
//
// Without a running maximum the tiles of a row are independent but for the sum: the sixteen
// softmax warps form four groups, group g takes every fourth tile, and each scheduler has one
// warp of every group, in its own phase of wait / load / exponentials / store.
//
// TMEM (all 512 columns): O 128, Q8 2 x 32 (A operand of QK^T, copied from shared memory by the tensor
// pipe; the next item's rows arrive while this one's are used), P 4 x 32 (one per group), S 3 x 64.  QK^T runs up
// to three tiles ahead of the groups, P.V behind them in the order of the list, and no tile waits for
// another one's P.V.  Two CTAs of 256 columns an SM, as before, have room for S or P of two tiles each:
// QK^T(j+2) had to wait for P.V(j), and a group's softmax, its P.V and its next QK^T were one chain.
// One query tile an SM also ends twice as soon, which evens out what the last CTAs do.
//
// Warp roles: warps 0-15 softmax/epilogue (TMEM lanes 32*(w%4).., group w/4), 16 K loader, 17 QK^T
// issuer, 18 P.V issuer and TMEM owner, 19 V loader.  The last four are one thread each but for
// fetching the list: what such a thread does for a tile is a chain of dependent instructions, and with
// votes of the whole warp, or K and V from one thread, that chain was as long as a tile takes (600 cycles).
//
// A CTA that is nearly through with an item takes over one that has not started (clusterlaunchcontrol), the long
// ones first; the next item's Q, scales and first tile indices are fetched under the last tiles of this one.
//
// Dense rows (query tiles that see every key) are cut into parts where they would outlast
// all others by more than the parts cost: see split_dense_rows.  Each part is an item with its own reference point; it
// leaves its sums in memory and the part that comes last adds them up, in the order of
// the list, so that the result does not depend on which one that was.
//
// What bounds it: per tile and SM the ex2 pipe needs 512 cycles, the tensor pipe 453 (measured: 144 for QK^T with A
// in TMEM, 258 with A in shared memory, 309 for P.V; at the nominal rates 384 in all), the softmax warps with their loads, stores
// and barriers 565 (in a loop of their own; 572 beside issuing warps).  By the SM clock a tile takes 640 in the middle of a list:
// the groups wait for one another's slots and for the slowest quarter of a group.  From an item's last P to the first
// P of the next one it was 7600 cycles.  Cycles of a launch with the epilogue at the item's end, all first tiles in the loop / now, thousands:
// 24 heads x 33272 tokens at 30 % 4856 / 4596; 24 x 9872 dense 1379 / 1298; 3 x 33272 at 30 % 621 / 595; 7 x 10384 at 15 % 113 / 108;
// 24 x 5000 at 10 % 141 / 119.  In time, launches of many layers in a row: 1.03 to 1.05 of it is gained, as the power cap sets the clock
// (1.49 GHz for the first of these after 200 launches, 1.75 for one by itself).
// Tried and slower on the earlier form: a polynomial
// for a share of the exponentials, two threads per row, one group per CTA.  Parts added up by a kernel of their own: 13 instead
// of 27 tiles' time for a part, but another main loop by ptxas' choice, 3 to 8 % slower for every launch.  On this form: groups kept
// out of step by a barrier inside the exponentials (every form 5 to 45 % slower: it cuts the loop's schedule), waits of the
// loading and issuing threads that sleep (1 to 13 % slower), eight orders of the exponentials' source (alike, or 1 % slower).
#include <type_traits>

#include "attn_common.cuh"
#include "tma.cuh"

namespace h3s {

constexpr int kHGroups = 4;  // of softmax warps; a group takes every fourth tile
constexpr int kHSoftmaxWarps = 4 * kHGroups;
constexpr int kHKeyLoader = kHSoftmaxWarps, kHScoreIssuer = kHSoftmaxWarps + 1, kHValueIssuer = kHSoftmaxWarps + 2,
              kHValueLoader = kHSoftmaxWarps + 3;
constexpr int kHWarps = kHSoftmaxWarps + 4, kHThreads = kHWarps * 32;
constexpr int kHScoreSlots = 3;
constexpr int kHMaxKStages = 5, kHMaxVStages = 8;
constexpr int kHTmemCols = 512, kHTmemQ = 128, kHTmemP = 192, kHTmemS = 320;  // O from 0
constexpr uint32_t kHKBytes = H3S_KV_TILE * H3S_HEAD_DIM;      // 8192
constexpr uint32_t kHVBytes = H3S_HEAD_DIM * H3S_KV_TILE * 2;  // 16384
constexpr uint32_t kHQBytes = H3S_Q_TILE * H3S_HEAD_DIM;       // 16384
constexpr int kHBlock = 16;  // tiles of a list that are fetched at a time
constexpr int kHMeta = 32;   // tiles whose scale is kept: a block and those before it that are loaded but not taken yet
constexpr float kHSumLimit = 65504.f;  // of a row over one tile: no P above it can have overflowed FP16
constexpr float kHFirstBits = 5.f;     // the reference tiles' row maximum becomes 2^-5 ...
constexpr float kHMostBits = 15.f;     // ... P may grow to 2^15 ...
constexpr float kHAgainBits = 8.f;     // ... and the largest sum of a row that did not fit becomes 2^8 at most
constexpr int kHNoted = 2048;          // bits of the note of tiles left out, each for 2^n neighbours of a longer list

enum { kAgainNoted = 1, kAgainFar = 2 };

// Beside the code of a wait: whose item it was about.  Constants, as what stands behind a wait is code in the loops.
constexpr int kInScoreIssuer = kHScoreIssuer << 8, kInValueIssuer = kHValueIssuer << 8, kItemBefore = 1 << 15;

// What the warps need to know of an item: left by the K loader, so that its place in the launch is worked out once
struct alignas(16) HalfItem {
  float v_scale[H3S_HEAD_DIM];
  int number;  // of the launch, -1: no more
  int head, tq, n_iter;
  int dense_row, part;  // of an item that is a part; -1 otherwise
};

struct alignas(16) HalfShared {
  uint4 next_reply;            // of the request for another item
  uint64_t next_ready;         // ... has arrived
  uint64_t q_full, q_free;     // the next item's Q rows are in shared memory, have been copied to TMEM
  uint64_t k_full[kHMaxKStages], k_empty[kHMaxKStages];
  uint64_t v_full[kHMaxVStages], v_empty[kHMaxVStages];
  uint64_t s_full[kHGroups];       // QK^T of a tile has completed; by group and not by slot, whose last user is another
                                   // group: a wait must never be two uses ahead
  uint64_t s_taken[kHScoreSlots];  // S of a tile is in registers
  uint64_t p_full[kHGroups];       // P of a tile is in TMEM
  uint64_t pv_done[kHGroups];      // P.V of a tile has completed: P may be written again
  uint64_t o_full, o_free;     // every P.V of a pass has completed; the softmax warps have read or scaled O
  uint64_t first_max;          // the reference tiles' row maxima are in `first`
  uint64_t pass_end;           // the rows' values of a pass are in `row`, `noted` is complete; all warps arrive and wait
  uint64_t staged;             // softmax warps only: the output tile is in shared memory (and steps before that)
  uint32_t tmem_base;
  int abort_word;              // code of the wait that ran out, 256 times the warp it was in (softmax: 0), kItemBefore
  int stopped[kHWarps];        // turn (of three) of the item that a warp ended at
  int finish;                  // of an item that is a part: this CTA writes the output tile
  int again[4];                // per item in turn.  kAgainNoted: some row has left out a tile; kAgainFar: its sum
                               // there does not tell the maximum
  HalfItem item[3];            // in turn: an epilogue may still read the last one when the one after next is known
  struct { int n_valid; float scale; } tile[kHMeta];  // keys of a tile inside the sequence, and the factor of its scores
  int block[2][kHBlock];            // the next tiles of the list, for the threads that load K and V
  uint32_t noted[2][kHNoted / 32];  // tiles of the list that some row has left out, per item in turn
  float first[2][H3S_Q_TILE];
  float over[kHGroups][H3S_Q_TILE];    // largest sum that a row has left out
  float row[2][kHGroups][H3S_Q_TILE];  // values the threads of a row give each other at a pass's end, in turn
};

// The output tile has room of its own, so that the next item's tiles can arrive under it
template <typename OutT>
struct HalfLayout {
  static constexpr int kKStages = sizeof(OutT) == 4 ? 3 : 5, kVStages = sizeof(OutT) == 4 ? 6 : 8;
  static constexpr uint32_t kOffK = 0;
  static constexpr uint32_t kOffV = kOffK + kKStages * kHKBytes;
  static constexpr uint32_t kOffQ = kOffV + kVStages * kHVBytes;
  static constexpr uint32_t kOffOut = kOffQ + kHQBytes;
  static constexpr uint32_t kOffShared = kOffOut + H3S_Q_TILE * H3S_HEAD_DIM * sizeof(OutT);
  static constexpr uint32_t kBytes = kOffShared + sizeof(HalfShared) + 1024;  // alignment slack
  static_assert(kKStages + kHScoreSlots < kHBlock && kKStages <= kHMaxKStages && kVStages <= kHMaxVStages && kBytes <= 227 * 1024, "attention shared memory exceeds the per-CTA limit");
};

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// Row sum and, with kPack, FP16 P of 64 scores.  The int32 scores become fp32 without a
// conversion instruction: for |s| < 2^22, bits(12582912.0f) + s are the bits of
// the float 12582912 + s exactly, and the offset is folded into the constants of
// the FMA that follows: P = exp2(c*f + bias) = exp2(c*s - m).  The folded constant is
// rounded, by 2^-24 of c*12582912: nothing for attention scores, but a factor of two from c = 1 on
// (scores of 2^20 bits).  With kExact the offset is taken off first and `bias` is -m.
template <bool kPack, bool kExact>
__device__ __forceinline__ float exp_sum(const uint32_t (&s)[H3S_KV_TILE], float c, float bias,
                                         uint32_t (&packed)[H3S_KV_TILE / 2]) {
  const float2 c2 = make_float2(c, c), bias2 = make_float2(bias, bias);
  float2 sum_a = make_float2(0.f, 0.f), sum_b = make_float2(0.f, 0.f);
#pragma unroll
  for (int i = 0; i < H3S_KV_TILE / 2; ++i) {
    float2 f = make_float2(__uint_as_float(s[2 * i] + kIntBiasBits), __uint_as_float(s[2 * i + 1] + kIntBiasBits));
    if (kExact) f = add2(f, make_float2(-kIntBias, -kIntBias));
    const float2 x = fma2(c2, f, bias2);
    const float2 p = make_float2(fast_exp2(x.x), fast_exp2(x.y));
    if (i & 1) sum_b = add2(sum_b, p); else sum_a = add2(sum_a, p);
    if (kPack) packed[i] = pack_half2(p.x, p.y);
  }
  sum_a = add2(sum_a, sum_b);
  return sum_a.x + sum_a.y;
}

__device__ __forceinline__ int max_score(const uint32_t (&s)[H3S_KV_TILE]) {
  int a = __vimax3_s32(s[0], s[1], s[2]), b = __vimax3_s32(s[3], s[4], s[5]);
#pragma unroll
  for (int i = 6; i + 3 < H3S_KV_TILE; i += 4) {
    a = __vimax3_s32(a, s[i], s[i + 1]);
    b = __vimax3_s32(b, s[i + 2], s[i + 3]);
  }
  return max(__vimax3_s32(a, s[H3S_KV_TILE - 2], s[H3S_KV_TILE - 1]), b);
}

// 32 floats -> 16 (bf16, fp16) or 32 words
template <typename OutT>
__device__ __forceinline__ void pack_columns(const uint32_t (&o)[32], uint32_t (&packed)[8 * sizeof(OutT)]) {
#pragma unroll
  for (int e = 0; e < 32; e += 4 / static_cast<int>(sizeof(OutT))) {
    const float lo = __uint_as_float(o[e]);
    if constexpr (std::is_same<OutT, float>::value) {
      packed[e] = __float_as_uint(lo);
    } else if constexpr (std::is_same<OutT, __half>::value) {
      packed[e / 2] = pack_half2(lo, __uint_as_float(o[e + 1]));
    } else {
      const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, __uint_as_float(o[e + 1]));
      packed[e / 2] = *reinterpret_cast<const uint32_t *>(&pair);
    }
  }
}

// Number of tiles the noted bits stand for (whole warp)
__device__ __forceinline__ int noted_tiles(const uint32_t *noted, int n_iter, int coarse, int lane) {
  const uint32_t last = static_cast<uint32_t>(n_iter - 1) >> coarse;
  int bits = 0;
  for (int w = lane; w < kHNoted / 32; w += 32) bits += __popc(noted[w]);
  bits = __reduce_add_sync(0xffffffffu, bits) << coarse;
  const bool ends = (noted[last >> 5] >> (last & 31)) & 1u;  // the last bit may stand for fewer
  return bits - (ends ? static_cast<int>((last + 1) << coarse) - n_iter : 0);
}

// Item `w` of a launch: dense (long) rows first, then the routed rows
struct HalfWork {
  int head, tq;
  int dense_row, part;  // running number of a dense row, part of its list where it is cut (-1: not)
  bool dense;
  int first_tile, n_iter;
  const int32_t *route_row;
};

__device__ __forceinline__ HalfWork work_item(const AttnParams &prm, int w) {
  HalfWork it;
  const int n_sparse = prm.route != nullptr ? prm.q_stop - prm.q_start : 0;
  const int n_dense = prm.q_tiles - n_sparse;
  const int dense_items = prm.heads * n_dense * prm.parts;
  it.dense = w < dense_items;
  it.dense_row = it.first_tile = 0;
  it.part = -1;
  it.route_row = nullptr;
  if (it.dense) {
    it.dense_row = w / prm.parts;
    const int part = w - it.dense_row * prm.parts;
    if (prm.parts > 1) it.part = part;
    it.head = it.dense_row / n_dense;
    const int i = it.dense_row - it.head * n_dense;
    it.tq = (n_sparse == 0 || i < prm.q_start) ? i : prm.q_stop + (i - prm.q_start);
    it.first_tile = part * prm.kv_tiles / prm.parts;  // even parts
    it.n_iter = (part + 1) * prm.kv_tiles / prm.parts - it.first_tile;
  } else {
    const int v = w - dense_items;
    it.head = v / n_sparse;
    const int i = v - it.head * n_sparse;
    it.tq = prm.q_start + i;
    it.n_iter = prm.route_len;
    it.route_row = prm.route + (static_cast<int64_t>(it.head) * n_sparse + i) * prm.route_len;
  }
  return it;
}

// The i-th tile that is walked
__device__ __forceinline__ int list_position(int i, int n_iter) {
  return i + n_iter / 2 < n_iter ? i + n_iter / 2 : i + n_iter / 2 - n_iter;
}

// A bit of the note stands for 2^n tiles
__device__ __forceinline__ int note_scale(int n_iter) { return 32 - __clz((n_iter - 1) / kHNoted); }

template <typename OutT>
__global__ void __launch_bounds__(kHThreads, 1)
sparse_attn_half_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                        const AttnParams prm) {
  using L = HalfLayout<OutT>;
  extern __shared__ unsigned char smem_dyn[];
  // SWIZZLE_128B tiles need 1024-byte alignment
  // (offset arithmetic, so that the compiler still sees shared memory)
  unsigned char *smem = smem_dyn + ((1024u - (ptx::smem_u32(smem_dyn) & 1023u)) & 1023u);
  HalfShared &sh = *reinterpret_cast<HalfShared *>(smem + L::kOffShared);
  volatile int *abort_word = &sh.abort_word;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  HalfWork work = work_item(prm, blockIdx.x);  // the first; more are asked for.  The loaders' own: the others read `sh.item`
  int n_iter = work.n_iter;

  // ---- setup ----
  let_next_start();
  if (threadIdx.x == 0) {
    ptx::mbar_init(&sh.next_ready, 1);
    ptx::mbar_init(&sh.q_full, 1);
    ptx::mbar_init(&sh.q_free, 1);
    for (int i = 0; i < L::kKStages; ++i) {
      ptx::mbar_init(&sh.k_full[i], 1);
      ptx::mbar_init(&sh.k_empty[i], 1);
    }
    for (int i = 0; i < L::kVStages; ++i) {
      ptx::mbar_init(&sh.v_full[i], 1);
      ptx::mbar_init(&sh.v_empty[i], 1);
    }
    for (int i = 0; i < kHScoreSlots; ++i) ptx::mbar_init(&sh.s_taken[i], 4);
    for (int g = 0; g < kHGroups; ++g) {
      ptx::mbar_init(&sh.s_full[g], 1);
      ptx::mbar_init(&sh.p_full[g], 4);
      ptx::mbar_init(&sh.pv_done[g], 1);
    }
    ptx::mbar_init(&sh.o_full, 1);
    ptx::mbar_init(&sh.o_free, kHSoftmaxWarps);
    ptx::mbar_init(&sh.first_max, 8);
    ptx::mbar_init(&sh.pass_end, kHWarps);
    ptx::mbar_init(&sh.staged, kHSoftmaxWarps);
    sh.abort_word = 0;
    sh.finish = 0;
    for (int i = 0; i < 4; ++i) sh.again[i] = 0;
    sh.item[0].number = blockIdx.x;
    sh.item[0].head = work.head;
    sh.item[0].tq = work.tq;
    sh.item[0].dense_row = work.dense_row;
    sh.item[0].part = work.part;
    ptx::fence_mbar_init();
  }
  if (threadIdx.x < 2 * kHNoted / 32) (&sh.noted[0][0])[threadIdx.x] = 0u;
  if (warp == kHValueIssuer) {
    ptx::tmem_alloc(&sh.tmem_base, kHTmemCols);
    ptx::tmem_relinquish();
  }
  wait_for_previous();
  if (threadIdx.x < H3S_HEAD_DIM) sh.item[0].v_scale[threadIdx.x] = load_written(prm.v_scale + work.head * H3S_HEAD_DIM + threadIdx.x);
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_o = sh.tmem_base;

  // Passes of an item: one over the list; where tiles were left out another one over those,
  // with a pass for the rows' true maxima in between where a sum has overflowed.  Every warp
  // arrives at `pass_end` and waits for it, so all agree on the tiles and the next item.
  // `done` counts the tiles of earlier items and passes, `passes` the passes, `items` the items:
  // slots and parities run on.
  bool ok = true;
  int done = 0, passes = 0;
  uint32_t items = 0;
  auto last_pass = [&]() {
    const int again = *static_cast<volatile int *>(&sh.again[items & 3]);
    return again == 0 ? 0 : again & kAgainFar ? 2 : 1;
  };
  auto arrive_pass = [&]() {
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&sh.pass_end);
  };
  auto wait_pass = [&]() {
    return warp_wait(&sh.pass_end, passes & 1u, abort_word, kAbortPass | warp << 8, 4 * prm.wait_budget_ns);
  };
  auto end_pass = [&]() {
    arrive_pass();
    return wait_pass();
  };
  auto count_noted = [&]() { return noted_tiles(sh.noted[items & 1], n_iter, note_scale(n_iter), lane); };
  // after an item's last pass: the next one, if there is one
  auto next_item = [&]() {
    ++items;
    const HalfItem &next = sh.item[items % 3u];
    n_iter = next.n_iter;
    return next.number >= 0;
  };

  if (warp == kHKeyLoader || warp == kHValueLoader) {
    // =================== K and V loaders ===================
    // Both walk the list: the whole warp fetches a block of tile indices, one block ahead of
    // their use, and one thread then loads those tiles.  The K loader also leaves the tiles'
    // scales in shared memory for the softmax warps, asks for the next item and, while this one's
    // last tiles are worked on, fetches that one's Q rows and scales.
    const bool keys = warp == kHKeyLoader;
    const CUtensorMap *map = keys ? &map_k : &map_v;
    if (lane == 0) {
      ptx::prefetch_tensormap(map);
      if (keys) ptx::prefetch_tensormap(&map_q);
    }
    // what an item's q_scale and k_scale are multiplied with: 1 / sqrt(128) / ln 2
    auto scale_of = [&](const HalfWork &it) {
      return load_written(prm.q_scale + it.head * prm.q_tiles + it.tq) * (0.08838834764831845f * 1.4426950408889634f);
    };
    float item_scale = keys ? scale_of(work) : 0.f, coming_scale = 0.f;
    int next_tile = 0;  // of the block of the list that comes next, one per lane
    float next_scale = 0.f;
    auto fetch = [&](const HalfWork &it, int position) {
      next_tile = it.dense ? it.first_tile + position : load_written(it.route_row + position);
      if (keys) next_scale = load_written(prm.k_scale + static_cast<int64_t>(it.head) * prm.kv_tiles + next_tile);
    };
    auto fetch_block = [&](const HalfWork &it, int i) {  // from the i-th tile on
      fetch(it, list_position(min(i + lane % kHBlock, it.n_iter - 1), it.n_iter));
    };
    auto load_q = [&](const HalfWork &it) {
      if (lane == 0) {
        ptx::mbar_arrive_expect_tx(&sh.q_full, kHQBytes);
        ptx::tma_load_3d(smem + L::kOffQ, &map_q, &sh.q_full, 0, it.tq * H3S_Q_TILE, it.head);
      }
      __syncwarp();
    };
    int *block = sh.block[keys ? 0 : 1];
    uint64_t *full = keys ? sh.k_full : sh.v_full, *empty = keys ? sh.k_empty : sh.v_empty;
    unsigned char *ring = smem + (keys ? L::kOffK : L::kOffV);
    const int stages = keys ? L::kKStages : L::kVStages;
    const uint32_t bytes = keys ? kHKBytes : kHVBytes;
    uint32_t seq = 0;    // tiles so far
    int stage = 0;       // state of the loading thread ...
    uint32_t round = 1;  // ... parity of the ring's previous use
    int drop = prm.drop_kv_load;  // running number of the tile that is not loaded, -1: none
    // the fetched block's first `tiles` tiles into the next stages; `meanwhile` may fetch again
    auto load_block = [&](int tiles, auto meanwhile) {
      if (lane < tiles) block[lane] = next_tile;
      if (keys && lane < tiles) {
        auto &tile = sh.tile[(seq + lane) % kHMeta];
        tile.n_valid = prm.sequence - next_tile * H3S_KV_TILE;
        tile.scale = item_scale * next_scale;
      }
      seq += tiles;
      __syncwarp();
      meanwhile();
      bool fine = true;
      if (ptx::elect_one()) {
        const int head = work.head;
        for (int i = 0; i < tiles; ++i) {
          const int t = block[i];
          fine = ptx::mbar_wait(&empty[stage], round, abort_word, kAbortKvEmpty | warp << 8, 4 * prm.wait_budget_ns);
          if (!fine) break;
          if (drop != 0) {
            ptx::mbar_arrive_expect_tx(&full[stage], bytes);
            ptx::tma_load_3d(ring + stage * bytes, map, &full[stage], keys ? 0 : t * H3S_KV_TILE * 2, keys ? t * H3S_KV_TILE : 0, head);
          }
          if (drop >= 0) --drop;
          if (++stage == stages) { stage = 0; round ^= 1u; }
        }
      }
      __syncwarp();
      return __all_sync(0xffffffffu, fine) != 0;
    };
    if (keys) load_q(work);
    fetch_block(work, 0);
    HalfWork coming = work;
    while (ok) {
      if (prm.drop_last_v_load && !keys) drop = work.n_iter - 1;
      for (int i = 0; ok && i < work.n_iter; i += kHBlock) {
        if (keys && i + kHBlock >= work.n_iter) {
          // Not before the last block: an item that is taken over waits until this one is through, while other
          // SMs run out of work.  7 heads x 10384 tokens at 15 %, 21 long rows that are not cut: 81 us when it was asked for
          // at once, 75 so; one head of 33272 at 10 % in parts 82 and 77.
          if (lane == 0) {
            ptx::fence_proxy_async_smem();  // the last reply has been read
            ptx::mbar_arrive_expect_tx(&sh.next_ready, sizeof(sh.next_reply));
            ptx::request_block(&sh.next_reply, &sh.next_ready);
          }
          __syncwarp();
        }
        ok = load_block(min(kHBlock, work.n_iter - i), [&]() { if (i + kHBlock < work.n_iter) fetch_block(work, i + kHBlock); });
      }
      ok = ok && warp_wait(&sh.next_ready, items & 1u, abort_word, kAbortNextItem | warp << 8, 4 * prm.wait_budget_ns);
      if (!ok) break;
      const int next = ptx::granted_block(&sh.next_reply);
      if (next >= 0) {
        coming = work_item(prm, next);
        fetch_block(coming, 0);
        if (keys) {
          HalfItem &to = sh.item[(items + 1) % 3u];
          coming_scale = scale_of(coming);
          if (lane == 0) {
            to.head = coming.head;
            to.tq = coming.tq;
            to.n_iter = coming.n_iter;
            to.dense_row = coming.dense_row;
            to.part = coming.part;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) to.v_scale[i * 32 + lane] = load_written(prm.v_scale + coming.head * H3S_HEAD_DIM + i * 32 + lane);
          ok = warp_wait(&sh.q_free, items & 1u, abort_word, kAbortQFree | warp << 8, 4 * prm.wait_budget_ns);
          if (!ok) break;
          load_q(coming);
        }
      }
      if (keys && lane == 0) sh.item[(items + 1) % 3u].number = next;
      ok = end_pass();
      ++passes;
      if (!ok) break;
      const int final_pass = last_pass();
      if (final_pass > 0) {
        const int first_tile = next_tile;  // of the next item, put aside
        const float first_scale = next_scale;
        const int count = count_noted(), coarse = note_scale(work.n_iter);
        const uint32_t *noted = sh.noted[items & 1];
        for (int pass = 1; ok && pass <= final_pass; ++pass) {
          int cursor = 0;
          for (int i = 0; ok && i < count; ++i) {
            for (;;) {  // the next noted tile; there is one, i < count
              const int bit = cursor >> coarse;
              const uint32_t w = noted[bit >> 5] >> (bit & 31);
              if (w & 1u) break;
              cursor = (w != 0u ? bit + __ffs(w) - 1 : ((bit >> 5) + 1) << 5) << coarse;
            }
            fetch(work, list_position(cursor++, work.n_iter));
            ok = load_block(1, []() {});
          }
          ok = ok && end_pass();
          ++passes;
        }
        next_tile = first_tile;
        next_scale = first_scale;
      }
      if (!ok || next < 0) break;
      ++items;
      work = coming;
      n_iter = work.n_iter;
      item_scale = coming_scale;
    }
  } else if (warp == kHScoreIssuer) {
    // =================== QK^T issuer ===================
    constexpr uint32_t idesc_qk = ptx::umma_idesc(2, 1, 1, H3S_Q_TILE, H3S_KV_TILE);
    const uint64_t k_desc0 = ptx::umma_desc_kmajor(ptx::smem_u32(smem + L::kOffK), 1024, ptx::kSwizzle128);
    const uint64_t q_desc = ptx::umma_desc_kmajor(ptx::smem_u32(smem + L::kOffQ), 1024, ptx::kSwizzle128);
    int stage = 0, slot = 0;  // state of the issuing thread
    uint32_t round = 0, slot_round = 0;
    while (ok) {
      const uint32_t tmem_q = tmem_o + kHTmemQ + (items & 1) * 32;
      ok = warp_wait(&sh.q_full, items & 1u, abort_word, kAbortQFull | kInScoreIssuer, prm.wait_budget_ns);
      if (!ok) break;
      if (ptx::elect_one()) {
#pragma unroll
        for (int k = 0; k < H3S_HEAD_DIM / 32; ++k) ptx::tmem_copy_256b(tmem_q + k * 8, q_desc + 2 * k);
        ptx::tc_commit(&sh.q_free);
      }
      __syncwarp();
      int count = n_iter;
      for (int pass = 0;; ++pass) {
        arrive_pass();  // nothing of the pass's end depends on this warp
        if (ptx::elect_one()) {
          for (int i = 0; i < count; ++i) {
            ok = ptx::mbar_wait(&sh.k_full[stage], round, abort_word, kAbortKvFull | kInScoreIssuer, prm.wait_budget_ns) &&
                 ptx::mbar_wait(&sh.s_taken[slot], slot_round ^ 1u, abort_word, kAbortScoreSlot | kInScoreIssuer, 3 * prm.wait_budget_ns);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint64_t k_desc = k_desc0 + static_cast<uint64_t>(stage * (kHKBytes >> 4));
#pragma unroll
            for (int k = 0; k < H3S_HEAD_DIM / 32; ++k)
              ptx::umma_i8_ts(tmem_o + kHTmemS + slot * 64, tmem_q + k * 8, k_desc + 2 * k, idesc_qk, k > 0);
            ptx::tc_commit(&sh.s_full[(done + i) % kHGroups]);
            ptx::tc_commit(&sh.k_empty[stage]);
            if (++stage == L::kKStages) { stage = 0; round ^= 1u; }
            if (++slot == kHScoreSlots) { slot = 0; slot_round ^= 1u; }
          }
        }
        __syncwarp();
        ok = __all_sync(0xffffffffu, ok) != 0;
        done += count;
        ok = ok && wait_pass();
        ++passes;
        if (!ok || pass == last_pass()) break;
        if (pass == 0) count = count_noted();
      }
      if (!ok || !next_item()) break;
    }
  } else if (warp == kHValueIssuer) {
    // =================== P.V issuer ===================
    constexpr uint32_t idesc_pv = ptx::umma_idesc(1, 0, 0, H3S_Q_TILE, H3S_HEAD_DIM);
    const uint64_t v_desc0 = ptx::umma_desc_kmajor(ptx::smem_u32(smem + L::kOffV), 1024, ptx::kSwizzle128);
    int stage = 0;
    uint32_t round = 0;
    while (ok) {
      int count = n_iter;
      for (int pass = 0;; ++pass) {
        arrive_pass();  // nothing of the pass's end depends on this warp
        ok = warp_wait(&sh.o_free, (passes & 1u) ^ 1u, abort_word, kAbortOFree | kInValueIssuer, 4 * prm.wait_budget_ns);
        if (ok && ptx::elect_one()) {
          for (int i = 0; i < count; ++i) {
            const int j = done + i, g = j % kHGroups;
            ok = ptx::mbar_wait(&sh.v_full[stage], round, abort_word, kAbortKvFull | kInValueIssuer, prm.wait_budget_ns) &&
                 ptx::mbar_wait(&sh.p_full[g], (j / kHGroups) & 1u, abort_word, kAbortPFull | kInValueIssuer, 3 * prm.wait_budget_ns);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint64_t v_desc = v_desc0 + static_cast<uint64_t>(stage * (kHVBytes >> 4));
#pragma unroll
            for (int k = 0; k < H3S_KV_TILE / 16; ++k)
              ptx::umma_f16_ts(tmem_o, tmem_o + kHTmemP + g * 32 + k * 8, v_desc + 2 * k, idesc_pv,
                               (pass > 0 || i > 0 || k > 0) ? 1u : 0u);
            ptx::tc_commit(&sh.pv_done[g]);
            ptx::tc_commit(&sh.v_empty[stage]);
            if (i == count - 1) ptx::tc_commit(&sh.o_full);
            if (++stage == L::kVStages) { stage = 0; round ^= 1u; }
          }
        }
        __syncwarp();
        ok = __all_sync(0xffffffffu, ok) != 0;
        done += count;
        ok = ok && wait_pass();
        ++passes;
        if (!ok || pass == last_pass()) break;
        if (pass == 0) count = count_noted();
      }
      if (!ok || !next_item()) break;
    }
  } else {
    // =================== softmax + epilogue (warps 0-15) ===================
    const int quarter = warp & 3, group = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t tmem_p = tmem_o + kHTmemP + group * 32 + lane_addr;

    // scores of tile j -> registers, and the factor that belongs to them
    auto take = [&](uint32_t j, uint32_t (&s)[H3S_KV_TILE], float &c) {
      if (!warp_wait(&sh.s_full[group], (j / kHGroups) & 1u, abort_word, kAbortSFull, 2 * prm.wait_budget_ns)) return false;
      const uint32_t slot = j % kHScoreSlots;
      ptx::tc_fence_after();
      H3S_TMEM_LD64(tmem_o + kHTmemS + slot * 64 + lane_addr, s);
      // left in shared memory by the K loader before the stage was handed to the tensor
      // pipe; the entry is written again when P.V of this tile is long complete
      const int n_valid = sh.tile[j % kHMeta].n_valid;
      c = sh.tile[j % kHMeta].scale;
      ptx::tmem_wait_ld(s);
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.s_taken[slot]);
      // Keys beyond the sequence (ragged last tile only): the integer whose biased
      // bits are those of -inf, so that P becomes 0; it is also below every score.
      if (n_valid < H3S_KV_TILE) {
#pragma unroll
        for (int i = 0; i < H3S_KV_TILE; ++i)
          if (i >= n_valid) s[i] = 0xff800000u - kIntBiasBits;
      }
      return true;
    };
    // the group's P columns are free
    auto room = [&](uint32_t j) {
      return warp_wait(&sh.pv_done[group], ((j / kHGroups) & 1u) ^ 1u, abort_word, kAbortPvDone, 4 * prm.wait_budget_ns);
    };
    // behind `room`: the fence orders the store after P.V's reads of the same columns
    auto put = [&](const uint32_t (&packed)[H3S_KV_TILE / 2]) {
      ptx::tc_fence_after();
      H3S_TMEM_ST32(tmem_p, packed);
    };
    auto hand_over = [&]() {
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.p_full[group]);
    };
    auto leave_first = [&](int which, float value) {
      sh.first[which][row] = value;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.first_max);
    };
    auto first_reference = [&]() { return ceilf(fmaxf(sh.first[0][row], sh.first[1][row])) + kHFirstBits; };
    uint32_t staged_uses = 0;
    auto meet = [&]() {  // all softmax warps
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.staged);
      return warp_wait(&sh.staged, staged_uses++ & 1u, abort_word, kAbortStaged, 4 * prm.wait_budget_ns);
    };
    // every P.V of the pass that has ended
    auto all_products = [&](int whose = 0) {
      return warp_wait(&sh.o_full, (passes - 1) & 1u, abort_word, kAbortFinal | whose, 4 * prm.wait_budget_ns);
    };
    auto release_o = [&]() {
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.o_free);
    };

    // O / l * v_scale of an item whose sums are complete, 32 columns of a row to a thread
    auto normalise = [&](uint32_t (&o)[32], float sum, const HalfItem &from) {
      const float inv_l = 1.0f / sum;
      const float2 inv2 = make_float2(inv_l, inv_l);
      const float4 *v_scale = reinterpret_cast<const float4 *>(from.v_scale) + group * 8;
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        const float4 vs = v_scale[e / 4];
        // |o / l| <= 448: nothing overflows
        const float2 a = mul2(mul2(make_float2(__uint_as_float(o[e]), __uint_as_float(o[e + 1])), inv2), make_float2(vs.x, vs.y));
        const float2 b = mul2(mul2(make_float2(__uint_as_float(o[e + 2]), __uint_as_float(o[e + 3])), inv2), make_float2(vs.z, vs.w));
        o[e] = __float_as_uint(a.x); o[e + 1] = __float_as_uint(a.y);
        o[e + 2] = __float_as_uint(b.x); o[e + 3] = __float_as_uint(b.y);
      }
    };
    auto row_sum = [&]() {  // of the pass that has ended
      const float *sums = &sh.row[(passes - 1) & 1][0][row];
      return (sums[0] + sums[H3S_Q_TILE]) + (sums[2 * H3S_Q_TILE] + sums[3 * H3S_Q_TILE]);
    };
    // The epilogue of the item before, once this group's first tile of the next one is handed over: the softmax warps need
    // not wait for the last P.V, and the next P.V comes later.  Every warp by itself: its 32 rows of 32 columns
    // go through its own piece of shared memory to a TMA store, which also leaves out rows past the sequence.
    bool pending = false;
    auto finish_last = [&](const HalfItem &from) {
      pending = false;
      if (!all_products(kItemBefore)) return false;
      ptx::tc_fence_after();
      uint32_t o[32];
      H3S_TMEM_LD32(tmem_o + lane_addr + group * 32, o);
      ptx::tmem_wait_ld(o);
      release_o();
      normalise(o, row_sum(), from);
      constexpr int kRowBytes = 32 * static_cast<int>(sizeof(OutT)), kChunks = kRowBytes / 16;
      uint32_t packed[4 * kChunks];
      pack_columns<OutT>(o, packed);
      unsigned char *piece = smem + L::kOffOut + warp * (32 * kRowBytes);
      if (lane == 0) ptx::bulk_wait_read();  // the piece's last store has read it
      __syncwarp();
      // the map's swizzle: rows of 64 bytes take turns by pairs, rows of 128 bytes one by one
      const int turn = sizeof(OutT) == 4 ? lane & 7 : (lane >> 1) & 3;
#pragma unroll
      for (int k = 0; k < kChunks; ++k)
        *reinterpret_cast<uint4 *>(piece + lane * kRowBytes + ((k ^ turn) << 4)) =
            make_uint4(packed[4 * k], packed[4 * k + 1], packed[4 * k + 2], packed[4 * k + 3]);
      ptx::fence_proxy_async_smem();
      __syncwarp();
      const int first_row = from.tq * H3S_Q_TILE + quarter * 32;
      if (lane == 0 && first_row < prm.sequence) {
        ptx::tma_store_3d(&map_out, piece, group * kRowBytes, first_row, from.head);
        ptx::bulk_commit();
      }
      return true;
    };

    while (ok) {
      // Which of the four groups has the first tile depends on what the CTA has done before; sums are
      // added up in the order of the tiles all the same, so that a result does not depend on that.
      const int rank = (group - done) & (kHGroups - 1);
      float m = 0.f, l = 0.f;
      sh.over[group][row] = 0.f;
      if (rank == 1 && n_iter == 1) leave_first(1, -INFINITY);
      // One tile.  A group's first one is a case of its own, so that the loop over the others holds neither the maxima nor the
      // last item's epilogue: 24 heads x 33272 tokens at 30 % 4.89 -> 4.61 million cycles.
      auto walk = [&](int i, auto first) {
        uint32_t s[H3S_KV_TILE];
        float c;
        if (!take(done + i, s, c)) return false;
        if (decltype(first)::value) {
          if (i < 2) leave_first(i, c * static_cast<float>(max_score(s)));  // c > 0
          if (!warp_wait(&sh.first_max, items & 1u, abort_word, kAbortFirstMax, 2 * prm.wait_budget_ns)) return false;
          m = first_reference();
        }
        uint32_t packed[H3S_KV_TILE / 2];
        float sum = exp_sum<true, false>(s, c, -fmaf(c, kIntBias, m), packed);
        if (!room(done + i)) return false;
        put(packed);
        const bool out = !(sum <= kHSumLimit);
        if (__any_sync(0xffffffffu, out)) {  // these rows leave the tile out
          const bool far = __any_sync(0xffffffffu, sum == INFINITY || c > 1.f);  // no measure of the maximum
          ptx::tmem_wait_st();
          if (out) {
            sh.over[group][row] = fmaxf(sh.over[group][row], sum);
            sum = 0.f;
#pragma unroll
            for (int e = 0; e < H3S_KV_TILE / 2; ++e) packed[e] = 0u;
          }
          put(packed);
          if (lane == 0) {
            const int coarse = note_scale(n_iter);
            atomicOr(&sh.noted[items & 1][(i >> coarse) >> 5], 1u << ((i >> coarse) & 31));
            atomicOr(&sh.again[items & 3], far ? kAgainNoted | kAgainFar : kAgainNoted);
          }
        }
        l += sum;
        hand_over();
        return true;
      };
      if (rank < n_iter) {
        ok = walk(rank, std::true_type{});
        if (ok && pending) ok = finish_last(sh.item[(items + 2) % 3u]);
        if (ok) {
          for (int i = rank + kHGroups; i < n_iter; i += kHGroups)
            if (!walk(i, std::false_type{})) { ok = false; break; }
        }
      }
      if (!ok) break;
      if (rank >= n_iter) {  // a group without a tile: the last item is not finished, and there is no reference point yet
        ok = (!pending || finish_last(sh.item[(items + 2) % 3u])) &&
             warp_wait(&sh.first_max, items & 1u, abort_word, kAbortFirstMax, 2 * prm.wait_budget_ns);
        if (!ok) break;
        m = first_reference();
      }
      done += n_iter;
      sh.row[passes & 1][rank][row] = l;
      // the word of the item after next: its last readers (two items ago) have all been at a pass's end since
      if (threadIdx.x == 0) sh.again[(items + 2) & 3] = 0;
      ok = end_pass();
      ++passes;
      if (!ok) break;
      const int final_pass = last_pass();
      if (final_pass > 0) {
        const int count = count_noted();
        ok = all_products();
        float m_again = m;
        if (final_pass == 1) {
          const float most = fmaxf(fmaxf(sh.over[0][row], sh.over[1][row]), fmaxf(sh.over[2][row], sh.over[3][row]));
          const uint32_t bits = __float_as_uint(most);
          if (bits != 0u) m_again = m + (static_cast<float>(static_cast<int>(bits >> 23) - 126) - kHAgainBits);
        } else {
          release_o();
          float top = -INFINITY;
          for (int i = (group - done) & (kHGroups - 1); ok && i < count; i += kHGroups) {
            uint32_t s[H3S_KV_TILE];
            float c;
            ok = take(done + i, s, c) && room(done + i);
            if (!ok) break;
            top = fmaxf(top, c * static_cast<float>(max_score(s)));
            uint32_t none[H3S_KV_TILE / 2];  // O stays as it is
#pragma unroll
            for (int e = 0; e < H3S_KV_TILE / 2; ++e) none[e] = 0u;
            put(none);
            hand_over();
          }
          done += count;
          sh.row[passes & 1][rank][row] = top;
          ok = ok && end_pass();
          const float *tops = &sh.row[passes & 1][0][row];
          ++passes;
          top = fmaxf(fmaxf(tops[0], tops[H3S_Q_TILE]), fmaxf(tops[2 * H3S_Q_TILE], tops[3 * H3S_Q_TILE]));
          if (top > m + kHMostBits) m_again = ceilf(top) - kHAgainBits;
          ok = ok && all_products();
        }
        const float factor = fast_exp2(m - m_again);  // a power of two
        l *= factor;
        if (ok && __any_sync(0xffffffffu, m_again != m)) {
          ptx::tc_fence_after();
          uint32_t o[32];
          H3S_TMEM_LD32(tmem_o + lane_addr + group * 32, o);
          ptx::tmem_wait_ld(o);
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * factor);
          H3S_TMEM_ST32(tmem_o + lane_addr + group * 32, o);
          ptx::tmem_wait_st();
        }
        release_o();
        for (int i = (group - done) & (kHGroups - 1); ok && i < count; i += kHGroups) {
          uint32_t s[H3S_KV_TILE];
          float c;
          ok = take(done + i, s, c) && room(done + i);
          if (!ok) break;
          uint32_t packed[H3S_KV_TILE / 2];
          // the same sum as in the first pass, so the same tiles
          const bool out = !(exp_sum<false, false>(s, c, -fmaf(c, kIntBias, m), packed) <= kHSumLimit);
          const float sum = exp_sum<true, true>(s, c, -m_again, packed);
          if (out) {
            l += sum;
          } else {
#pragma unroll
            for (int e = 0; e < H3S_KV_TILE / 2; ++e) packed[e] = 0u;
          }
          put(packed);
          hand_over();
        }
        done += count;
        m = m_again;
        sh.row[passes & 1][rank][row] = l;
        ok = ok && end_pass();
        ++passes;
        if (!ok) break;
        // (this note's next item is the one after next, and its last reader has been at the pass's end)
        if (threadIdx.x < kHNoted / 32) sh.noted[items & 1][threadIdx.x] = 0u;
      }
      const HalfItem &work = sh.item[items % 3u];
      const bool split = work.part >= 0;
      if (!split && prm.out_map) {
        pending = true;
        if (next_item()) continue;
        ok = finish_last(sh.item[(items + 2) % 3u]);
        break;
      }

      // Parts of a row, and outputs that go to peers too: the softmax warps work together, at once
      l = row_sum();
      ok = all_products();
      if (!ok) break;
      ptx::tc_fence_after();
      uint32_t o[32];
      H3S_TMEM_LD32(tmem_o + lane_addr + group * 32, o);
      ptx::tmem_wait_ld(o);
      release_o();
      bool finish = true;
      if (split) {
        // Partial sums of part p: [32 groups of 4 columns][128 rows] float4, so that a warp's rows are
        // neighbours; then 128 row sums and 128 reference points.
        constexpr int kPartFloats = H3S_Q_TILE * (H3S_HEAD_DIM + 2);
        const float *parts_base = prm.partial + static_cast<int64_t>(work.dense_row) * prm.parts * kPartFloats;
        float *mine = const_cast<float *>(parts_base) + static_cast<int64_t>(work.part) * kPartFloats;
#pragma unroll
        for (int e = 0; e < 32; e += 4)
          __stcg(reinterpret_cast<float4 *>(mine) + (group * 8 + e / 4) * H3S_Q_TILE + row,
                 make_float4(__uint_as_float(o[e]), __uint_as_float(o[e + 1]), __uint_as_float(o[e + 2]),
                             __uint_as_float(o[e + 3])));
        if (group == 0) {
          __stcg(mine + H3S_Q_TILE * H3S_HEAD_DIM + row, l);
          __stcg(mine + H3S_Q_TILE * (H3S_HEAD_DIM + 1) + row, m);
        }
        __threadfence();
        ok = meet();
        if (ok && threadIdx.x == 0) {
          __threadfence();
          sh.finish = atomicAdd(prm.arrived + work.dense_row, 1u) == static_cast<unsigned int>(prm.parts - 1);
          __threadfence();
        }
        ok = ok && meet();
        if (!ok) break;
        finish = *static_cast<volatile int *>(&sh.finish) != 0;
        if (finish) {
          l = 0.f;
          float top = -INFINITY;  // largest reference point of the parts
          for (int p = 0; p < prm.parts; ++p)
            top = fmaxf(top, __ldcg(parts_base + p * kPartFloats + H3S_Q_TILE * (H3S_HEAD_DIM + 1) + row));
          for (int p = 0; p < prm.parts; ++p) {
            const float *at = parts_base + p * kPartFloats + H3S_Q_TILE * H3S_HEAD_DIM + row;
            l = fmaf(__ldcg(at), fast_exp2(__ldcg(at + H3S_Q_TILE) - top), l);
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) o[e] = 0u;
#pragma unroll 1
          for (int p = 0; p < prm.parts; ++p) {
            const float *at = parts_base + p * kPartFloats;
            // the reference points are integers: the factors are powers of two
            const float weight = fast_exp2(__ldcg(at + H3S_Q_TILE * (H3S_HEAD_DIM + 1) + row) - top);
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
              const float4 x = __ldcg(reinterpret_cast<const float4 *>(at) + (group * 8 + e / 4) * H3S_Q_TILE + row);
              o[e] = __float_as_uint(fmaf(x.x, weight, __uint_as_float(o[e])));
              o[e + 1] = __float_as_uint(fmaf(x.y, weight, __uint_as_float(o[e + 1])));
              o[e + 2] = __float_as_uint(fmaf(x.z, weight, __uint_as_float(o[e + 2])));
              o[e + 3] = __float_as_uint(fmaf(x.w, weight, __uint_as_float(o[e + 3])));
            }
          }
        }
      }
      if (finish) {
        // Staged through shared memory: the four warps of a row quarter each write eight of the quarter's rows as
        // contiguous lines, and what goes to the peers is made of lines too.
        normalise(o, l, work);
        constexpr int kRowBytes = H3S_HEAD_DIM * static_cast<int>(sizeof(OutT));
        constexpr int kChunks = 32 * static_cast<int>(sizeof(OutT)) / 16;
        unsigned char *out_tile = smem + L::kOffOut;
        uint32_t packed[4 * kChunks];
        pack_columns<OutT>(o, packed);
        // a warp's own store of an earlier item may still be reading its piece, and the warps write each other's
        if (lane == 0) ptx::bulk_wait_read();
        ok = meet();
        if (!ok) break;
        // the chunk index is XORed with the row so that the 32 rows of a warp do not collide on banks
#pragma unroll
        for (int k = 0; k < kChunks; ++k)
          *reinterpret_cast<uint4 *>(out_tile + row * kRowBytes + (((group * kChunks + k) ^ (row & 15)) << 4)) =
              make_uint4(packed[4 * k], packed[4 * k + 1], packed[4 * k + 2], packed[4 * k + 3]);
        ok = meet();
        if (!ok) break;
        store_rows<OutT>(prm, out_tile, work.head, work.tq, quarter * 32 + group * 8, 8, lane);
        if (prm.n_peer_out > 0) scatter_to_peers<OutT>(prm, out_tile, work.head, work.tq, kHSoftmaxWarps * 32);
      }
      if (!next_item()) break;
    }
    if (lane == 0) ptx::bulk_wait();  // the last stores, before the CTA's shared memory goes
  }

  // ---- teardown ----
  if (lane == 0) sh.stopped[warp] = items % 3u;
  __syncthreads();
  const int word = sh.abort_word, code = word & 255;
  if (code != 0) {
    // leave time for copies / MMAs still in flight before releasing TMEM and shared memory
    __nanosleep(200000);
    if (threadIdx.x == 0) {
      int turn = (sh.stopped[(word >> 8) & 31] + ((word & kItemBefore) != 0 ? 2 : 0)) % 3;
      if (sh.item[turn].number < 0) turn = (turn + 2) % 3;  // a warp that was through
      const HalfItem &at = sh.item[turn];
      report_status(prm.status, prm.status_mirror, code, at.number, at.head, at.tq);
    }
  }
  if (warp == kHValueIssuer) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_o, kHTmemCols);
  }
}

// E4M3 codes -> FP16 values: 16 per thread
__global__ void __launch_bounds__(256) v_half_kernel(const uint4 *__restrict__ v8, uint4 *__restrict__ v16, int64_t chunks) {
  let_next_start();
  wait_for_previous();
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= chunks) return;
  const uint4 codes = load_written(v8 + i);
  v16[2 * i] = e4m3x8_to_half(make_uint2(codes.x, codes.y));
  v16[2 * i + 1] = e4m3x8_to_half(make_uint2(codes.z, codes.w));
}

// Whether and how the dense rows' tile lists are cut.  A row longer than half of what an SM gets on average may end after
// everything else has, which parts even out; but parts are dear.  Beside its tiles (0.35 us each) a whole dense row takes an SM
// about as long as eight tiles, a routed one fifteen (most of it before its first tile), a part 28 and three for each
// part of its row: it writes 66 KB, waits until they are seen, and one of them reads them all back; and counters are cleared
// before the launch, which then starts behind the one before it.  So as many parts as end first by this estimate, every SM
// taking the next item as it gets free, and only if
//  - that is earlier than with whole rows, or
//  - it is no later, and the parts' own cost is under 1 % of the work (three heads of 33272 tokens at 30 %: 417 us, 410 whole), or
//  - nothing but dense rows is there, and dealt out evenly instead of in rounds the parts would end with the rows, by an older
//    estimate of their cost.  Whole rows are the faster ones at this last line (3 x 4000: 30 us, 45 in parts; 2 x 1537 15 and 23);
//    it stays because the tests of the parts take their shapes from it.
// Fitted to 228 shapes of 1 to 24 heads, launches in a row.  Measured, us, whole / in parts (how many), the one taken last:
//   dense   1 x 5000 34 / 28 (3), 1 x 9400 57 / 45 (2), 1 x 20000 224 / 185 (3); 2 x 9000 99 (4) / 57, 4 x 9000 177 (4) / 106,
//           6 x 1545 35 (3) / 15, 12 x 2000 56 (2) / 32, 1 x 33272 463 (4) / 401
//   routed  1 x 12512 at 30 % 74 / 34 (6), 3 x 6512 at 30 % 42 / 39 (2), 2 x 15000 at 15 % 87 / 46 (3), 1 x 33272 at 10 % 184 / 58 (5), at 30 %
//           202 / 134 (2); 4 x 2304 at 30 % 24 (6) / 19, 6 x 4256 33 (2) / 30, 24 x 5000 at 10 % 100 (4) / 75, 7 x 10384 at 15 % 74 (4) / 68
// It is wrong by most for 3 x 18181 at 20 % (107 whole, 96 in sixteen parts) and 4 x 8161 at 15 % (46 in three, 43 in four).
constexpr int kMinPartTiles = 6, kMaxParts = 16;
constexpr int kLongTiles = 8, kRoutedTiles = 15, kPartTiles = 28, kPerPartTiles = 3;
constexpr int kEvenLongTiles = 12, kEvenPartTiles = 27;

// When the last item ends, in tiles: `dense` ones of `dense_cost` first, then `routed` ones of `routed_cost`
static int64_t launch_span(int64_t dense, int64_t dense_cost, int64_t routed, int64_t routed_cost) {
  const int64_t late = dense % kSmCount, early = kSmCount - late;  // SMs that get one dense item more, and the others
  int64_t early_free = dense / kSmCount * dense_cost, late_free = early_free + dense_cost;
  int64_t end = late > 0 ? late_free : early_free;
  while (routed > 0) {
    const bool first = late == 0 || early_free <= late_free;
    int64_t &free = first ? early_free : late_free;
    routed -= first ? early : late;
    free += routed_cost;
    if (free > end) end = free;
  }
  return end;
}

static int split_dense_rows(int heads, int q_tiles, int kv_tiles, int n_sparse, int route_len) {
  const int64_t rows = static_cast<int64_t>(heads) * (q_tiles - n_sparse), routed = static_cast<int64_t>(heads) * n_sparse;
  if (rows == 0 || static_cast<int64_t>(kv_tiles) * kSmCount * 2 <= rows * kv_tiles + routed * route_len) return 1;
  const int64_t whole_cost = kv_tiles + kLongTiles, routed_cost = route_len + kRoutedTiles;
  const int64_t whole_span = launch_span(rows, whole_cost, routed, routed_cost), whole_work = rows * whole_cost + routed * routed_cost;
  int best = 1;
  int64_t best_span = 0, best_work = 0;
  bool even = false;
  for (int parts = 2; parts <= kMaxParts && kv_tiles / parts >= kMinPartTiles; ++parts) {
    const int part_tiles = ceil_div(kv_tiles, parts);
    const int64_t cost = part_tiles + kPartTiles + kPerPartTiles * parts, work = rows * parts * cost + routed * routed_cost;
    const int64_t span = launch_span(rows * parts, cost, routed, routed_cost);
    if (best == 1 || span < best_span) { best = parts; best_span = span; best_work = work; }
    const int64_t even_cost = part_tiles + kEvenPartTiles, share = rows * parts * even_cost / kSmCount;
    even = even || (routed == 0 && 100 * (share > even_cost ? share : even_cost) <= 103 * (kv_tiles + kEvenLongTiles));
  }
  if (best == 1) return 1;
  const bool earlier = best_span < whole_span;
  const bool free = best_span <= whole_span && 100 * best_work <= 101 * whole_work;
  return earlier || free || even ? best : 1;
}

static size_t split_bytes(int64_t dense_rows, int parts, size_t *arrived_bytes) {
  *arrived_bytes = (static_cast<size_t>(dense_rows) * sizeof(unsigned int) + 255) & ~static_cast<size_t>(255);
  return *arrived_bytes + static_cast<size_t>(dense_rows) * parts * H3S_Q_TILE * (H3S_HEAD_DIM + 2) * sizeof(float);
}

template <typename OutT>
static int launch_attn_half(const CUtensorMap &mq, const CUtensorMap &mk, const CUtensorMap &mv, const CUtensorMap &mo,
                            const AttnParams &prm, cudaStream_t stream) {
  constexpr int kBytes = static_cast<int>(HalfLayout<OutT>::kBytes);
  H3S_CHECK_CUDA(cudaFuncSetAttribute(sparse_attn_half_kernel<OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBytes));
  const int n_sparse = prm.route != nullptr ? prm.q_stop - prm.q_start : 0;
  const int items = prm.heads * ((prm.q_tiles - n_sparse) * prm.parts + n_sparse);
  H3S_CHECK_CUDA(launch_next(sparse_attn_half_kernel<OutT>, items, kHThreads, kBytes, stream, mq, mk, mv, mo, prm));
  return H3S_OK;
}

}  // namespace h3s

extern "C" int h3s_v_half(const uint8_t *v8t, void *v16t, int heads, int sequence, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(v8t != nullptr && v16t != nullptr, "v_half: NULL pointer");
  H3S_CHECK_ARG(heads > 0 && sequence > 0, "v_half: empty problem (heads=%d sequence=%d)", heads, sequence);
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(v8t) | reinterpret_cast<uintptr_t>(v16t)) & 15) == 0, "v_half: carriers must be 16-byte aligned");
  const int64_t chunks = static_cast<int64_t>(heads) * H3S_HEAD_DIM * (ceil_div(sequence, 128) * 128) / 16;
  H3S_CHECK_CUDA(launch_next(v_half_kernel, static_cast<unsigned>((chunks + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream),
                             reinterpret_cast<const uint4 *>(v8t), static_cast<uint4 *>(v16t), chunks));
  return H3S_OK;
}

extern "C" size_t h3s_sparse_attn_half_workspace_bytes(int heads, int sequence, int route_len, int q_start, int q_stop) {
  using namespace h3s;
  if (heads <= 0 || sequence <= 0) return 0;
  const int q_tiles = ceil_div(sequence, H3S_Q_TILE), kv_tiles = ceil_div(sequence, H3S_KV_TILE);
  const int n_sparse = route_len > 0 ? q_stop - q_start : 0;
  const int parts = split_dense_rows(heads, q_tiles, kv_tiles, n_sparse, route_len);
  size_t arrived_bytes;
  return parts > 1 ? split_bytes(static_cast<int64_t>(heads) * (q_tiles - n_sparse), parts, &arrived_bytes) : 0;
}

extern "C" int h3s_sparse_attn_half_fwd_mirrored(const int8_t *q8, const int8_t *k8, const void *v16t, const float *q_scale,
                                                 const float *k_scale, const float *v_scale, const int32_t *route,
                                                 int route_len, int q_start, int q_stop, void *out, void *const *peer_out,
                                                 int n_peer_out, int out_dtype, int64_t out_stride_h, int64_t out_stride_s,
                                                 int heads, int sequence, int flags, void *workspace, size_t workspace_bytes,
                                                 int32_t *status, int32_t *host_mirror, h3s_stream_t stream) {
  using namespace h3s;
  AttnParams prm;
  int rc = fill_attn_params(&prm, q8, k8, v16t, q_scale, k_scale, v_scale, route, route_len, q_start, q_stop, out,
                            peer_out, n_peer_out, out_dtype, out_stride_h, out_stride_s, heads, sequence, flags, status,
                            "sparse_attn_half_fwd");
  if (rc) return rc;
  const uint64_t S = static_cast<uint64_t>(sequence);
  const uint64_t row_bytes = static_cast<uint64_t>(ceil_div(sequence, 128)) * 128 * 2;
  CUtensorMap mq, mk, mv;
  rc = make_tensor_map_u8_3d(&mq, q8, H3S_HEAD_DIM, S, heads, H3S_HEAD_DIM, S * H3S_HEAD_DIM, H3S_HEAD_DIM,
                             H3S_Q_TILE, CU_TENSOR_MAP_SWIZZLE_128B, "sparse_attn_half_fwd Q map");
  if (rc) return rc;
  rc = make_tensor_map_u8_3d(&mk, k8, H3S_HEAD_DIM, S, heads, H3S_HEAD_DIM, S * H3S_HEAD_DIM, H3S_HEAD_DIM,
                             H3S_KV_TILE, CU_TENSOR_MAP_SWIZZLE_128B, "sparse_attn_half_fwd K map");
  if (rc) return rc;
  rc = make_tensor_map_u8_3d(&mv, v16t, row_bytes, H3S_HEAD_DIM, heads, row_bytes, row_bytes * H3S_HEAD_DIM,
                             H3S_KV_TILE * 2, H3S_HEAD_DIM, CU_TENSOR_MAP_SWIZZLE_128B, "sparse_attn_half_fwd V map");
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  prm.status_mirror = host_mirror;
  prm.parts = 1; prm.partial = nullptr; prm.arrived = nullptr;
  // One head's stride is never used and need not suit a map; with peers the tile is staged as a whole instead
  const uint64_t size = out_dtype == H3S_F32 ? 4 : 2;
  CUtensorMap mo;
  const uint64_t stride_s = static_cast<uint64_t>(out_stride_s) * size;
  const uint64_t stride_h = heads > 1 ? static_cast<uint64_t>(out_stride_h) * size : stride_s;
  prm.out_map = prm.out_map && n_peer_out == 0 && (flags & H3S_ATTN_PLAIN_STORES) == 0 &&
                make_tensor_map_u8_3d(&mo, out, H3S_HEAD_DIM * size, S, heads, stride_s, stride_h, 32 * size, 32,
                                      size == 4 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                                      "sparse_attn_half_fwd output map") == H3S_OK;
  if (!prm.out_map) mo = mq;
  if (workspace != nullptr) {
    const int n_sparse = route != nullptr ? q_stop - q_start : 0;
    const int parts = split_dense_rows(heads, prm.q_tiles, prm.kv_tiles, n_sparse, n_sparse ? route_len : 0);
    size_t arrived_bytes;
    const size_t need = split_bytes(static_cast<int64_t>(heads) * (prm.q_tiles - n_sparse), parts, &arrived_bytes);
    if (parts > 1) {
      H3S_CHECK_ARG(workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0,
                    "sparse_attn_half_fwd: the workspace must be 16-byte aligned and hold %zu bytes, got %zu", need, workspace_bytes);
      prm.parts = parts;
      prm.arrived = static_cast<unsigned int *>(workspace);
      prm.partial = reinterpret_cast<float *>(static_cast<unsigned char *>(workspace) + arrived_bytes);
      H3S_CHECK_CUDA(cudaMemsetAsync(workspace, 0, arrived_bytes, s));
    }
  }
  switch (out_dtype) {
    case H3S_F32: return launch_attn_half<float>(mq, mk, mv, mo, prm, s);
    case H3S_BF16: return launch_attn_half<__nv_bfloat16>(mq, mk, mv, mo, prm, s);
    default: return launch_attn_half<__half>(mq, mk, mv, mo, prm, s);
  }
}

extern "C" int h3s_sparse_attn_half_fwd(const int8_t *q8, const int8_t *k8, const void *v16t, const float *q_scale,
                                        const float *k_scale, const float *v_scale, const int32_t *route,
                                        int route_len, int q_start, int q_stop, void *out, void *const *peer_out,
                                        int n_peer_out, int out_dtype, int64_t out_stride_h, int64_t out_stride_s,
                                        int heads, int sequence, int flags, void *workspace, size_t workspace_bytes,
                                        int32_t *status, h3s_stream_t stream) {
  return h3s_sparse_attn_half_fwd_mirrored(q8, k8, v16t, q_scale, k_scale, v_scale, route, route_len, q_start, q_stop, out, peer_out,
                                           n_peer_out, out_dtype, out_stride_h, out_stride_s, heads, sequence, flags, workspace,
                                           workspace_bytes, status, nullptr, stream);
}
