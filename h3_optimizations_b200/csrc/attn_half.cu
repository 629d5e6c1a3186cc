// Block-sparse attention on INT8 Q/K and an FP16 copy of the FP8 V carrier, for
// sm_100a.
//
// One CTA owns one 128-row query tile of one head and walks that tile's list
// of 64-row KV tiles:
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
// tokens, 30 %: 3.09 to 3.26 ms on the inputs above; 3.29 to 3.48 with one row of every query
// tile 48 bits ahead in every 40th tile; 3.78 to 3.94 with a third of the rows ahead in every tenth;
// two E4M3 terms take 4.2 to 4.3 ms of each.  All but the first two tiles of a list
// ahead is the worst: two walks, three where a sum overflows (120 bits): 24 heads x 9872,
// dense, 0.83 ms, then 2.1 to 2.2 and 2.9, where two E4M3 terms take 1.13.
//
// Without a running maximum the tiles of a row are independent but for the sum:
// the eight softmax warps form two groups, group g takes tiles g, g+2, ..., and
// with two CTAs per SM four warps share a scheduler, each in its own phase of
// wait / load / exponentials / store.  With one group, or with two threads per row,
// the CTAs fall into step and both pipes idle a third of the time.
//
// TMEM (256 columns per CTA, two CTAs per SM): O 128, Q8 32 (A operand of QK^T:
// Q is read once instead of with every K tile, which takes a third off the
// shared-memory traffic), and three 32-column slots A B C.  S(j) is 64 columns:
// A+B for even j, B+C for odd j; P(j) is 32 columns: A for even, C for odd.
// QK^T(j) needs S(j-1) in registers (slot B) and P.V(j-2) complete.
//
// Warp roles: warps 0-7 softmax/epilogue (TMEM lanes 32*(w%4).., group w/4), warp 8
// TMA producer and QK^T issuer, warp 9 P.V issuer and TMEM owner.
//
// Dense rows (query tiles that see every key) are cut into parts where one of them is
// longer than what a CTA slot gets on average, i.e. where a few long rows would outlast
// all others: see split_dense_rows.  Each part is a CTA with its own reference point; it
// leaves its sums in memory and the part that comes last adds them up, in the order of
// the list, so that the result does not depend on which one that was.
//
// What bounds it: per tile and SM the ex2 pipe needs 512 cycles, the tensor pipe 453
// (measured: 144 for QK^T with A in TMEM, 258 with A in shared memory, 309 for P.V; at
// the nominal rates 384 in all), the remaining softmax instructions about 290 issue
// slots; a tile takes about 800.  24 heads x 33272 tokens at 30 %, launches in a row: 4.20 to
// 4.33 ms with two E4M3 terms, 3.09 to 3.26 ms here.  Tried and slower: a polynomial for a
// share of the exponentials, two threads per row, one group per CTA, scores of the next
// tile fetched between the halves of this one.
#include "attn_common.cuh"
#include "tma.cuh"

namespace h3s {

constexpr int kHStages = 4;  // tile i+2 is loaded when tile i-2 is done
constexpr int kHSoftmaxWarps = 8;
constexpr int kHThreads = (kHSoftmaxWarps + 2) * 32;
constexpr int kHTmemCols = 256;
constexpr uint32_t kHKBytes = H3S_KV_TILE * H3S_HEAD_DIM;      // 8192
constexpr uint32_t kHVBytes = H3S_HEAD_DIM * H3S_KV_TILE * 2;  // 16384
constexpr uint32_t kHOffK = 0;
constexpr uint32_t kHOffV = kHOffK + kHStages * kHKBytes;
constexpr uint32_t kHOffBar = kHOffV + kHStages * kHVBytes;
constexpr uint32_t kHSmemBytes = kHOffBar + 4096 + 1024;  // barriers/scalars + alignment slack
constexpr float kHSumLimit = 65504.f;  // of a row over one tile: no P above it can have overflowed FP16
constexpr float kHFirstBits = 5.f;     // the reference tiles' row maximum becomes 2^-5 ...
constexpr float kHMostBits = 15.f;     // ... P may grow to 2^15 ...
constexpr float kHAgainBits = 8.f;     // ... and the largest sum of a row that did not fit becomes 2^8 at most
constexpr int kHNoted = 2048;          // bits of the note of tiles left out, each for 2^n neighbours of a longer list

enum { kAgainNoted = 1, kAgainFar = 2 };

struct HalfShared {
  uint64_t q_ready;            // four softmax warps have put the Q rows into TMEM
  uint64_t kv_full[kHStages];
  uint64_t s_full[2];          // QK^T of tile j has completed (one per group)
  uint64_t s_taken[2];         // S(j) is in registers
  uint64_t p_full[2];          // P(j) is in TMEM
  uint64_t pv_done[2];         // P.V of tile j has completed: its stage and its slot are free
  uint64_t first_max;          // both groups have left their first tile's row maxima in `first`
  uint64_t first_exp;          // group 0 is through its first tile's exponentials
  uint64_t pass_end;           // the rows' values of a pass are in `row`, `noted` is complete; all warps wait,
                               // and the P.V warp arrives too: see there
  uint64_t staged;             // softmax warps only: the output tile is in shared memory (and steps before that)
  uint32_t tmem_base;
  int abort_word;
  int again;                   // kAgainNoted: some row has left out a tile; kAgainFar: its sum there does not tell the maximum
  int finish;                  // this CTA writes the output tile
  int tile_index[kHStages];    // KV tile held by each stage ...
  float tile_scale[kHStages];  // ... and its k_scale, written by the producer
  float v_scale[H3S_HEAD_DIM];
  uint32_t noted[kHNoted / 32];  // tiles of the list that some row has left out
  float first[2][H3S_Q_TILE];
  float row[2][2][H3S_Q_TILE];  // values the two threads of a row give each other, in turn
};
static_assert(sizeof(HalfShared) <= 4096, "barrier block too large");

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

// Number of tiles the noted bits stand for (whole warp)
__device__ __forceinline__ int noted_tiles(const uint32_t *noted, int n_iter, int coarse, int lane) {
  const uint32_t last = static_cast<uint32_t>(n_iter - 1) >> coarse;
  int bits = 0;
  for (int w = lane; w < kHNoted / 32; w += 32) bits += __popc(noted[w]);
  bits = __reduce_add_sync(0xffffffffu, bits) << coarse;
  const bool ends = (noted[last >> 5] >> (last & 31)) & 1u;  // the last bit may stand for fewer
  return bits - (ends ? static_cast<int>((last + 1) << coarse) - n_iter : 0);
}

template <typename OutT>
__global__ void __launch_bounds__(kHThreads, 2)
sparse_attn_half_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        const int8_t *__restrict__ q8, const AttnParams prm) {
  extern __shared__ unsigned char smem_dyn[];
  // SWIZZLE_128B tiles need 1024-byte alignment
  // (offset arithmetic, so that the compiler still sees shared memory)
  unsigned char *smem = smem_dyn + ((1024u - (ptx::smem_u32(smem_dyn) & 1023u)) & 1023u);
  HalfShared &sh = *reinterpret_cast<HalfShared *>(smem + kHOffBar);
  volatile int *abort_word = &sh.abort_word;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // ---- work item: dense (long) rows first, then the routed rows ----
  const int n_sparse = prm.route != nullptr ? prm.q_stop - prm.q_start : 0;
  const int n_dense = prm.q_tiles - n_sparse;
  int head, tq;
  int dense_row = 0, part = 0;  // running number of a dense row, part of its list
  bool dense;
  {
    const int w = blockIdx.x;
    const int dense_items = prm.heads * n_dense * prm.parts;
    if (w < dense_items) {
      dense = true;
      dense_row = w / prm.parts;
      part = w - dense_row * prm.parts;
      head = dense_row / n_dense;
      const int i = dense_row - head * n_dense;
      tq = (n_sparse == 0 || i < prm.q_start) ? i : prm.q_stop + (i - prm.q_start);
    } else {
      dense = false;
      const int v = w - dense_items;
      head = v / n_sparse;
      tq = prm.q_start + (v - head * n_sparse);
    }
  }
  const bool split = dense && prm.parts > 1;
  const int first_tile = part * prm.part_tiles;  // of a dense row's list
  const int n_iter = dense ? min(prm.part_tiles, prm.kv_tiles - first_tile) : prm.route_len;
  const int32_t *route_row =
      dense ? nullptr
            : prm.route + (static_cast<int64_t>(head) * n_sparse + (tq - prm.q_start)) * prm.route_len;

  // ---- setup ----
  if (threadIdx.x == 0) {
    ptx::mbar_init(&sh.q_ready, 4);
    for (int i = 0; i < kHStages; ++i) ptx::mbar_init(&sh.kv_full[i], 1);
    for (int g = 0; g < 2; ++g) {
      ptx::mbar_init(&sh.s_full[g], 1);
      ptx::mbar_init(&sh.s_taken[g], 4);
      ptx::mbar_init(&sh.p_full[g], 4);
      ptx::mbar_init(&sh.pv_done[g], 1);
    }
    ptx::mbar_init(&sh.first_max, kHSoftmaxWarps);
    ptx::mbar_init(&sh.first_exp, 4);
    ptx::mbar_init(&sh.pass_end, kHSoftmaxWarps + 1);
    ptx::mbar_init(&sh.staged, kHSoftmaxWarps);
    sh.abort_word = 0;
    sh.again = 0;
    sh.finish = 1;
    ptx::fence_mbar_init();
  }
  if (threadIdx.x < kHNoted / 32) sh.noted[threadIdx.x] = 0u;
  if (threadIdx.x < H3S_HEAD_DIM) sh.v_scale[threadIdx.x] = __ldg(prm.v_scale + head * H3S_HEAD_DIM + threadIdx.x);
  if (warp == kHSoftmaxWarps + 1) {
    ptx::tmem_alloc(&sh.tmem_base, kHTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_o = sh.tmem_base;         // 128 columns, fp32
  const uint32_t tmem_q = tmem_o + 128;         // 32 columns, four int8 codes each
  const uint32_t tmem_s = tmem_o + 160;         // slots A B C, 32 columns each

  // Passes: one over the list; where tiles were left out another one over those, with a
  // pass for the rows' true maxima in between where a sum has overflowed.  Every warp waits
  // for `pass_end`, so all agree on the tiles.  `done` counts the tiles of earlier passes:
  // stages and parities run on.
  bool ok = true;
  int done = 0, count = n_iter;
  const int coarse = 32 - __clz((n_iter - 1) / kHNoted);  // a bit of the note stands for 2^coarse tiles
  auto last_pass = [&]() {
    const int again = *static_cast<volatile int *>(&sh.again);
    return again == 0 ? 0 : again & kAgainFar ? 2 : 1;
  };
  auto list_position = [&](int i) { return i + n_iter / 2 < n_iter ? i + n_iter / 2 : i + n_iter / 2 - n_iter; };

  // wait for tile j's use of one of a pair of barriers (tile j uses number j & 1)
  auto wait_tile = [&](uint64_t (&bar)[2], int j, int code, int factor) {
    return warp_wait(&bar[j & 1], static_cast<uint32_t>(j >> 1) & 1u, abort_word, code, factor * prm.wait_budget_ns);
  };
  auto wait_stage = [&](int j) {
    return warp_wait(&sh.kv_full[j % kHStages], static_cast<uint32_t>(j / kHStages) & 1u, abort_word, kAbortKvFull,
                     prm.wait_budget_ns);
  };

  if (warp == kHSoftmaxWarps) {
    // =================== TMA producer and QK^T issuer ===================
    // QK^T(j) waits for P.V(j-2), which also frees that tile's stage: tile j+2's
    // loads go out behind it.  The whole warp fetches the tile indices and K scales
    // of 32 tiles at a time, one block ahead of their use; lane 0 leaves each stage's
    // index and scale in shared memory for the softmax warps.
    constexpr uint32_t idesc_qk = ptx::umma_idesc(2, 1, 1, H3S_Q_TILE, H3S_KV_TILE);
    const uint64_t k_desc0 = ptx::umma_desc_kmajor(ptx::smem_u32(smem + kHOffK), 1024, ptx::kSwizzle128);
    const float *k_scale = prm.k_scale + static_cast<int64_t>(head) * prm.kv_tiles;
    if (lane == 0) {
      ptx::prefetch_tensormap(&map_k);
      ptx::prefetch_tensormap(&map_v);
    }
    int my_tile = 0, next_tile = 0, block = -1;  // tile list entries 32*block .. +31, one per lane, and the 32 after
    float my_scale = 0.f, next_scale = 0.f;
    auto fetch_block = [&](int b) {
      const int mine = list_position(min(b * 32 + lane, n_iter - 1));
      next_tile = dense ? first_tile + mine : __ldg(route_row + mine);
      next_scale = __ldg(k_scale + next_tile);
    };
    int cursor = 0;               // where a later pass goes on in the note
    auto load = [&](int pass, int i) {  // tile i of the pass, into the stage of its running number
      if (i >= count) return;
      int t;
      float ks;
      if (pass == 0) {
        if ((i >> 5) != block) {
          block = i >> 5;
          my_tile = next_tile; my_scale = next_scale;
          fetch_block(block + 1);
        }
        t = __shfl_sync(0xffffffffu, my_tile, i & 31);
        ks = __shfl_sync(0xffffffffu, my_scale, i & 31);
      } else {
        for (;;) {  // the next noted tile; there is one, i < count
          const int bit = cursor >> coarse;
          const uint32_t w = sh.noted[bit >> 5] >> (bit & 31);
          if (w & 1u) break;
          cursor = (w != 0u ? bit + __ffs(w) - 1 : ((bit >> 5) + 1) << 5) << coarse;
        }
        const int at = list_position(cursor++);
        t = dense ? first_tile + at : __ldg(route_row + at);
        ks = __ldg(k_scale + t);
      }
      if (lane == 0 && done + i != prm.drop_kv_load) {
        const int s = (done + i) % kHStages;
        sh.tile_index[s] = t;
        sh.tile_scale[s] = ks;
        ptx::mbar_arrive_expect_tx(&sh.kv_full[s], kHKBytes + kHVBytes);
        ptx::tma_load_3d(smem + kHOffK + s * kHKBytes, &map_k, &sh.kv_full[s], 0, t * H3S_KV_TILE, head);
        ptx::tma_load_3d(smem + kHOffV + s * kHVBytes, &map_v, &sh.kv_full[s], t * H3S_KV_TILE * 2, 0, head);
      }
      __syncwarp();
    };
    for (int pass = 0; ok; ++pass) {
      cursor = 0;
      if (pass == 0) fetch_block(0);
      for (int i = 0; i < kHStages; ++i) load(pass, i);
      if (pass == 0) ok = warp_wait(&sh.q_ready, 0, abort_word, kAbortQFull, prm.wait_budget_ns);
      for (int i = 0; ok && i < count; ++i) {
        const int j = done + i;
        ok = wait_stage(j) && (i < 1 || wait_tile(sh.s_taken, j - 1, kAbortPEmpty, 3)) &&
             (i < 2 || wait_tile(sh.pv_done, j - 2, kAbortPvDone, 4));
        if (!ok) break;
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          const uint64_t k_desc = k_desc0 + static_cast<uint64_t>((j % kHStages) * (kHKBytes >> 4));
#pragma unroll
          for (int k = 0; k < H3S_HEAD_DIM / 32; ++k)
            ptx::umma_i8_ts(tmem_s + (j & 1) * 32, tmem_q + k * 8, k_desc + 2 * k, idesc_qk, k > 0);
          ptx::tc_commit(&sh.s_full[j & 1]);
        }
        __syncwarp();
        if (i >= 2) load(pass, i + 2);
      }
      // (what the loop has not waited for, so that every barrier is one use behind at most)
      const int last = done + count - 1;
      ok = ok && wait_tile(sh.s_taken, last, kAbortPEmpty, 3) && (count < 2 || wait_tile(sh.pv_done, last - 1, kAbortFinal, 4)) &&
           wait_tile(sh.pv_done, last, kAbortFinal, 4);
      done += count;
      ok = ok && warp_wait(&sh.pass_end, pass & 1u, abort_word, kAbortFinal, 4 * prm.wait_budget_ns);
      if (pass == last_pass()) break;
      if (pass == 0) count = noted_tiles(sh.noted, n_iter, coarse, lane);
    }
  } else if (warp == kHSoftmaxWarps + 1) {
    // =================== P.V issuer ===================
    constexpr uint32_t idesc_pv = ptx::umma_idesc(1, 0, 0, H3S_Q_TILE, H3S_HEAD_DIM);
    const uint64_t v_desc0 = ptx::umma_desc_kmajor(ptx::smem_u32(smem + kHOffV), 1024, ptx::kSwizzle128);
    for (int pass = 0; ok; ++pass) {
      for (int j = done; j < done + count; ++j) {
        if (!wait_tile(sh.p_full, j, kAbortPFull, 3) || !wait_stage(j)) { ok = false; break; }
        ptx::tc_fence_after();
        if (ptx::elect_one()) {
          const uint64_t v_desc = v_desc0 + static_cast<uint64_t>((j % kHStages) * (kHVBytes >> 4));
#pragma unroll
          for (int k = 0; k < H3S_KV_TILE / 16; ++k)
            ptx::umma_f16_ts(tmem_o, tmem_s + (j & 1) * 64 + k * 8, v_desc + 2 * k, idesc_pv, (j > 0 || k > 0) ? 1u : 0u);
          ptx::tc_commit(&sh.pv_done[j & 1]);
        }
        __syncwarp();
      }
      done += count;
      // Lists of one or two tiles: nothing in the next pass up to its own pass_end waits for this
      // warp, so that without its arrival here two passes could end before it looks, and the
      // parity it waits for would be that of a third.
      if (ok && lane == 0) ptx::mbar_arrive(&sh.pass_end);
      ok = ok && warp_wait(&sh.pass_end, pass & 1u, abort_word, kAbortFinal, 4 * prm.wait_budget_ns);
      if (pass == last_pass()) break;
      if (pass == 0) count = noted_tiles(sh.noted, n_iter, coarse, lane);
    }
  } else {
    // =================== softmax + epilogue (warps 0-7) ===================
    const int quarter = warp & 3, group = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    if (group == 0) {
      // this thread's Q row -> its TMEM lane
      uint32_t q[32];
      const int grow = tq * H3S_Q_TILE + row;
      const uint4 *src = reinterpret_cast<const uint4 *>(q8 + (static_cast<int64_t>(head) * prm.sequence + grow) * H3S_HEAD_DIM);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint4 w = grow < prm.sequence ? __ldg(src + i) : make_uint4(0u, 0u, 0u, 0u);
        q[4 * i] = w.x; q[4 * i + 1] = w.y; q[4 * i + 2] = w.z; q[4 * i + 3] = w.w;
      }
      H3S_TMEM_ST32(tmem_q + lane_addr, q);
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.q_ready);
    }
    const float q_scale = __ldg(prm.q_scale + head * prm.q_tiles + tq) * (0.08838834764831845f * 1.4426950408889634f);
    float m = 0.f, l = 0.f;

    // scores of tile j -> registers, and the factor that belongs to them
    auto take = [&](int j, uint32_t (&s)[H3S_KV_TILE], float &c) {
      if (!wait_tile(sh.s_full, j, kAbortSFull, 2)) return false;
      ptx::tc_fence_after();
      H3S_TMEM_LD64(tmem_s + lane_addr + group * 32, s);
      // index and K scale of this tile, left in shared memory by the producer
      // before the stage was handed to the tensor pipe (free only after P.V(j))
      const int n_valid = prm.sequence - sh.tile_index[j % kHStages] * H3S_KV_TILE;
      c = q_scale * sh.tile_scale[j % kHStages];
      ptx::tmem_wait_ld(s);
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.s_taken[group]);
      // Keys beyond the sequence (ragged last tile only): the integer whose biased
      // bits are those of -inf, so that P becomes 0; it is also below every score.
      if (n_valid < H3S_KV_TILE) {
#pragma unroll
        for (int i = 0; i < H3S_KV_TILE; ++i)
          if (i >= n_valid) s[i] = 0xff800000u - kIntBiasBits;
      }
      return true;
    };
    // P -> slot A or C: part of S(j), which is in registers
    auto put = [&](const uint32_t (&packed)[H3S_KV_TILE / 2]) { H3S_TMEM_ST32(tmem_s + lane_addr + group * 64, packed); };
    auto hand_over = [&]() {
      ptx::tmem_wait_st();
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.p_full[group]);
    };
    auto own_first = [&](int from) { return (from & 1) == group ? from : from + 1; };  // of this group's tiles
    // both threads of a row leave a value, then wait for everything else of the pass
    auto end_pass = [&](int pass, float value) {
      sh.row[pass & 1][group][row] = value;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.pass_end);
      return warp_wait(&sh.pass_end, pass & 1u, abort_word, kAbortFinal, 4 * prm.wait_budget_ns);
    };
    auto leave_first = [&](float value) {
      sh.first[group][row] = value;
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.first_max);
    };
    auto first_reference = [&]() { return ceilf(fmaxf(sh.first[0][row], sh.first[1][row])) + kHFirstBits; };
    uint32_t staged_uses = 0;
    auto meet = [&]() {  // all softmax warps
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&sh.staged);
      return warp_wait(&sh.staged, staged_uses++ & 1u, abort_word, kAbortFinal, 4 * prm.wait_budget_ns);
    };

    float largest = 0.f;  // sum over a tile that this thread has left out
    if (group == 1 && n_iter == 1) leave_first(-INFINITY);
    for (int j = group; j < n_iter; j += 2) {
      uint32_t s[H3S_KV_TILE];
      float c;
      if (!take(j, s, c)) { ok = false; break; }
      if (j < 2) {
        leave_first(c * static_cast<float>(max_score(s)));  // c > 0
        if (!warp_wait(&sh.first_max, 0, abort_word, kAbortSFull, 2 * prm.wait_budget_ns)) { ok = false; break; }
        m = first_reference();
        // the maxima bring the groups together; the second one waits, so that they are out of
        // step again (24 heads x 2304 tokens 45.1 -> 43.3 us, 7 x 10384 84.5 -> 83.6, long lists alike)
        if (j == 1 && !warp_wait(&sh.first_exp, 0, abort_word, kAbortSFull, 2 * prm.wait_budget_ns)) { ok = false; break; }
      }
      uint32_t packed[H3S_KV_TILE / 2];
      float sum = exp_sum<true, false>(s, c, -fmaf(c, kIntBias, m), packed);
      if (j == 0) {
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(&sh.first_exp);
      }
      put(packed);
      const bool out = !(sum <= kHSumLimit);
      if (__any_sync(0xffffffffu, out)) {  // these rows leave the tile out
        const bool far = __any_sync(0xffffffffu, sum == INFINITY || c > 1.f);  // no measure of the maximum
        ptx::tmem_wait_st();
        if (out) {
          largest = fmaxf(largest, sum);
          sum = 0.f;
#pragma unroll
          for (int i = 0; i < H3S_KV_TILE / 2; ++i) packed[i] = 0u;
        }
        put(packed);
        if (lane == 0) {
          atomicOr(&sh.noted[(j >> coarse) >> 5], 1u << ((j >> coarse) & 31));
          atomicOr(&sh.again, far ? kAgainNoted | kAgainFar : kAgainNoted);
        }
      }
      l += sum;
      hand_over();
    }
    done = n_iter;
    sh.row[1][group][row] = largest;
    ok = ok && end_pass(0, l);
    const int final_pass = ok ? last_pass() : 0;
    if (final_pass > 0) {
      count = noted_tiles(sh.noted, n_iter, coarse, lane);
      m = first_reference();  // (a group without a tile has none yet)
      float m_again = m;
      if (final_pass == 1) {
        const uint32_t bits = __float_as_uint(fmaxf(sh.row[1][0][row], sh.row[1][1][row]));
        if (bits != 0u) m_again = m + (static_cast<float>(static_cast<int>(bits >> 23) - 126) - kHAgainBits);
      } else {
        float top = -INFINITY;
        for (int j = own_first(done); j < done + count; j += 2) {
          uint32_t s[H3S_KV_TILE];
          float c;
          if (!take(j, s, c)) { ok = false; break; }
          top = fmaxf(top, c * static_cast<float>(max_score(s)));
          uint32_t none[H3S_KV_TILE / 2];  // O stays as it is
#pragma unroll
          for (int i = 0; i < H3S_KV_TILE / 2; ++i) none[i] = 0u;
          put(none);
          hand_over();
        }
        done += count;
        ok = ok && end_pass(1, top);
        top = fmaxf(sh.row[1][0][row], sh.row[1][1][row]);
        if (top > m + kHMostBits) m_again = ceilf(top) - kHAgainBits;
      }
      // every P.V so far (one barrier per group): O may be touched
      ok = ok && (done < 2 || wait_tile(sh.pv_done, done - 2, kAbortFinal, 4)) && wait_tile(sh.pv_done, done - 1, kAbortFinal, 4);
      const float factor = fast_exp2(m - m_again);  // a power of two
      l *= factor;
      if (ok && __any_sync(0xffffffffu, m_again != m)) {
        ptx::tc_fence_after();
#pragma unroll 1
        for (int cc = group * 2; cc < group * 2 + 2; ++cc) {
          uint32_t o[32];
          H3S_TMEM_LD32(tmem_o + lane_addr + cc * 32, o);
          ptx::tmem_wait_ld(o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
          H3S_TMEM_ST32(tmem_o + lane_addr + cc * 32, o);
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
      }
      ok = ok && meet();  // the first P.V of the next pass waits for one group only
      for (int j = own_first(done); ok && j < done + count; j += 2) {
        uint32_t s[H3S_KV_TILE];
        float c;
        if (!take(j, s, c)) { ok = false; break; }
        uint32_t packed[H3S_KV_TILE / 2];
        // the same sum as in the first pass, so the same tiles
        const bool out = !(exp_sum<false, false>(s, c, -fmaf(c, kIntBias, m), packed) <= kHSumLimit);
        const float sum = exp_sum<true, true>(s, c, -m_again, packed);
        if (out) {
          l += sum;
        } else {
#pragma unroll
          for (int i = 0; i < H3S_KV_TILE / 2; ++i) packed[i] = 0u;
        }
        put(packed);
        hand_over();
      }
      done += count;
      m = m_again;
      ok = ok && end_pass(final_pass, l);
    }
    if (ok) l = sh.row[final_pass & 1][0][row] + sh.row[final_pass & 1][1][row];

    // every P.V of the last pass (one barrier per group)
    if (ok && done > 1) ok = wait_tile(sh.pv_done, done - 2, kAbortFinal, 4);
    if (ok) ok = wait_tile(sh.pv_done, done - 1, kAbortFinal, 4);
    if (ok) {
      // Epilogue: O / l * v_scale -> OutT, staged through shared memory (the
      // stage ring is free: every TMA load has been consumed).  A warp converts its
      // 32 rows of one column half; the two warps of a row quarter then each write
      // 16 of the quarter's rows as full contiguous lines.
      ptx::tc_fence_after();
      // Partial sums of part p: [32 groups of 4 columns][128 rows] float4, so that a warp's rows are
      // neighbours; then 128 row sums and 128 reference points.
      constexpr int kPartFloats = H3S_Q_TILE * (H3S_HEAD_DIM + 2);
      const float *parts_base = prm.partial + static_cast<int64_t>(dense_row) * prm.parts * kPartFloats;
      float top = 0.f;  // largest reference point of the parts
      if (split) {
        float *mine = const_cast<float *>(parts_base) + static_cast<int64_t>(part) * kPartFloats;
#pragma unroll 1
        for (int cc = group * 2; cc < group * 2 + 2; ++cc) {
          uint32_t o[32];
          H3S_TMEM_LD32(tmem_o + lane_addr + cc * 32, o);
          ptx::tmem_wait_ld(o);
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            __stcg(reinterpret_cast<float4 *>(mine) + (cc * 8 + i / 4) * H3S_Q_TILE + row,
                   make_float4(__uint_as_float(o[i]), __uint_as_float(o[i + 1]), __uint_as_float(o[i + 2]),
                               __uint_as_float(o[i + 3])));
        }
        if (group == 0) {
          __stcg(mine + H3S_Q_TILE * H3S_HEAD_DIM + row, l);
          __stcg(mine + H3S_Q_TILE * (H3S_HEAD_DIM + 1) + row, m);
        }
        __threadfence();
        ok = meet();
        if (ok && warp == 0 && lane == 0) {
          __threadfence();
          sh.finish = atomicAdd(prm.arrived + dense_row, 1u) == static_cast<unsigned int>(prm.parts - 1);
          __threadfence();
        }
        ok = ok && meet();
        if (ok && sh.finish) {
          l = 0.f;
          top = -INFINITY;
          for (int p = 0; p < prm.parts; ++p)
            top = fmaxf(top, __ldcg(parts_base + p * kPartFloats + H3S_Q_TILE * (H3S_HEAD_DIM + 1) + row));
          for (int p = 0; p < prm.parts; ++p) {
            const float *at = parts_base + p * kPartFloats + H3S_Q_TILE * H3S_HEAD_DIM + row;
            l = fmaf(__ldcg(at), fast_exp2(__ldcg(at + H3S_Q_TILE) - top), l);
          }
        }
      }
      const bool finish = ok && sh.finish;
      const float inv_l = 1.0f / l;
      constexpr int kRowBytes = H3S_HEAD_DIM * static_cast<int>(sizeof(OutT));
      static_assert(H3S_Q_TILE * kRowBytes <= kHOffBar, "output tile must fit the stage ring");
      unsigned char *my_row = smem + row * kRowBytes;
#pragma unroll 1
      for (int cc = group * 2; finish && cc < group * 2 + 2; ++cc) {
        uint32_t o[32];
        if (!split) {
          H3S_TMEM_LD32(tmem_o + lane_addr + cc * 32, o);
          ptx::tmem_wait_ld(o);
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0u;
#pragma unroll 1
          for (int p = 0; p < prm.parts; ++p) {
            const float *at = parts_base + p * kPartFloats;
            // the reference points are integers: the factors are powers of two
            const float weight = fast_exp2(__ldcg(at + H3S_Q_TILE * (H3S_HEAD_DIM + 1) + row) - top);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const float4 x = __ldcg(reinterpret_cast<const float4 *>(at) + (cc * 8 + i / 4) * H3S_Q_TILE + row);
              o[i] = __float_as_uint(fmaf(x.x, weight, __uint_as_float(o[i])));
              o[i + 1] = __float_as_uint(fmaf(x.y, weight, __uint_as_float(o[i + 1])));
              o[i + 2] = __float_as_uint(fmaf(x.z, weight, __uint_as_float(o[i + 2])));
              o[i + 3] = __float_as_uint(fmaf(x.w, weight, __uint_as_float(o[i + 3])));
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e)
            v[e] = __uint_as_float(o[i + e]) * inv_l * sh.v_scale[cc * 32 + i + e];  // |o / l| <= 448: nothing overflows
          // 8 values = one (bf16/fp16) or two (fp32) 16-byte chunks; the chunk index is
          // XORed with the row so that the 32 rows of a warp do not collide on banks
          constexpr int kChunks8 = 8 * static_cast<int>(sizeof(OutT)) / 16;
          const int chunk0 = (cc * 32 + i) * static_cast<int>(sizeof(OutT)) / 16;
          __align__(16) OutT tmp[8];
          store_out8<OutT>(tmp, v);
#pragma unroll
          for (int k = 0; k < kChunks8; ++k)
            *reinterpret_cast<uint4 *>(my_row + (((chunk0 + k) ^ (row & 15)) << 4)) =
                reinterpret_cast<const uint4 *>(tmp)[k];
        }
      }
      ptx::tc_fence_before();
      // both halves of the rows are staged
      if (finish && meet()) store_rows<OutT>(prm, smem, head, tq, quarter * 32 + group * 16, 16, lane);
    }
  }

  // ---- teardown ----
  __syncthreads();
  const int code = sh.abort_word;
  if (code != 0) {
    // leave time for copies / MMAs still in flight before releasing TMEM and shared memory
    __nanosleep(200000);
    if (threadIdx.x == 0 && prm.status != nullptr) {
      if (atomicCAS(prm.status, 0, code) == 0) {
        prm.status[1] = blockIdx.x;
        prm.status[2] = head;
        prm.status[3] = tq;
      }
    }
  }
  if (warp == kHSoftmaxWarps + 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_o, kHTmemCols);
  }
  // head-sharded run: the producer and MMA warps have nothing left to do and share the copy
  if (code == 0 && prm.n_peer_out > 0 && sh.finish) scatter_to_peers<OutT>(prm, smem, head, tq, kHThreads);
}

// E4M3 codes -> FP16 values: 16 per thread
__global__ void __launch_bounds__(256) v_half_kernel(const uint4 *__restrict__ v8, uint4 *__restrict__ v16, int64_t chunks) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= chunks) return;
  const uint4 codes = __ldg(v8 + i);
  v16[2 * i] = e4m3x8_to_half(make_uint2(codes.x, codes.y));
  v16[2 * i + 1] = e4m3x8_to_half(make_uint2(codes.z, codes.w));
}

// Whether and how the dense rows' tile lists are cut.  Two CTAs run on each of 148 SMs; a
// slot gets `share` tiles on average.  A dense row much longer than that ends after
// everything else has: seven heads of 10384 tokens at 15 % (28 dense rows of 163 tiles
// beside 546 routed ones of 31, share 73) take 195 us for the whole layer uncut, 176 us in
// parts.  At the line itself, an eighth longer than the share, both are equal (three heads
// of 33272 tokens at 30 %: 520 against a share of 441, 523 and 521 us), and below it the
// order "long rows first" fills the slots, so that parts would only cost their traffic.  A
// quarter of the share keeps the last parts short; under 24 tiles a part's start and end
// (about 4 us) would show.
constexpr int kSlots = 2 * 148, kMinPartTiles = 24, kMaxParts = 16;

static int split_dense_rows(int heads, int q_tiles, int kv_tiles, int n_sparse, int route_len, int *part_tiles) {
  const int64_t n_dense = q_tiles - n_sparse;
  const int64_t total = heads * (n_dense * kv_tiles + static_cast<int64_t>(n_sparse) * route_len);
  *part_tiles = kv_tiles;
  if (n_dense == 0 || static_cast<int64_t>(kv_tiles) * kSlots * 7 <= total * 8) return 1;
  int tiles = static_cast<int>(total / (4 * kSlots));
  if (tiles < kMinPartTiles) tiles = kMinPartTiles;
  if (tiles < ceil_div(kv_tiles, kMaxParts)) tiles = ceil_div(kv_tiles, kMaxParts);
  const int parts = ceil_div(kv_tiles, tiles);
  *part_tiles = ceil_div(kv_tiles, parts);  // even parts; none is empty
  return ceil_div(kv_tiles, *part_tiles);
}

static size_t split_bytes(int64_t dense_rows, int parts, size_t *arrived_bytes) {
  *arrived_bytes = (static_cast<size_t>(dense_rows) * sizeof(unsigned int) + 255) & ~static_cast<size_t>(255);
  return *arrived_bytes + static_cast<size_t>(dense_rows) * parts * H3S_Q_TILE * (H3S_HEAD_DIM + 2) * sizeof(float);
}

template <typename OutT>
static int launch_attn_half(const CUtensorMap &mk, const CUtensorMap &mv, const int8_t *q8, const AttnParams &prm,
                            cudaStream_t stream) {
  H3S_CHECK_CUDA(cudaFuncSetAttribute(sparse_attn_half_kernel<OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kHSmemBytes)));
  const int n_sparse = prm.route != nullptr ? prm.q_stop - prm.q_start : 0;
  const int ctas = prm.heads * ((prm.q_tiles - n_sparse) * prm.parts + n_sparse);
  sparse_attn_half_kernel<OutT><<<ctas, kHThreads, kHSmemBytes, stream>>>(mk, mv, q8, prm);
  H3S_CHECK_CUDA(cudaGetLastError());
  return H3S_OK;
}

}  // namespace h3s

extern "C" int h3s_v_half(const uint8_t *v8t, void *v16t, int heads, int sequence, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(v8t != nullptr && v16t != nullptr, "v_half: NULL pointer");
  H3S_CHECK_ARG(heads > 0 && sequence > 0, "v_half: empty problem (heads=%d sequence=%d)", heads, sequence);
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(v8t) | reinterpret_cast<uintptr_t>(v16t)) & 15) == 0, "v_half: carriers must be 16-byte aligned");
  const int64_t chunks = static_cast<int64_t>(heads) * H3S_HEAD_DIM * (ceil_div(sequence, 128) * 128) / 16;
  v_half_kernel<<<static_cast<unsigned>((chunks + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const uint4 *>(v8t), static_cast<uint4 *>(v16t), chunks);
  H3S_CHECK_CUDA(cudaGetLastError());
  return H3S_OK;
}

extern "C" size_t h3s_sparse_attn_half_workspace_bytes(int heads, int sequence, int route_len, int q_start, int q_stop) {
  using namespace h3s;
  if (heads <= 0 || sequence <= 0) return 0;
  const int q_tiles = ceil_div(sequence, H3S_Q_TILE), kv_tiles = ceil_div(sequence, H3S_KV_TILE);
  const int n_sparse = route_len > 0 ? q_stop - q_start : 0;
  int part_tiles;
  const int parts = split_dense_rows(heads, q_tiles, kv_tiles, n_sparse, route_len, &part_tiles);
  size_t arrived_bytes;
  return parts > 1 ? split_bytes(static_cast<int64_t>(heads) * (q_tiles - n_sparse), parts, &arrived_bytes) : 0;
}

extern "C" int h3s_sparse_attn_half_fwd(const int8_t *q8, const int8_t *k8, const void *v16t, const float *q_scale,
                                        const float *k_scale, const float *v_scale, const int32_t *route,
                                        int route_len, int q_start, int q_stop, void *out, void *const *peer_out,
                                        int n_peer_out, int out_dtype, int64_t out_stride_h, int64_t out_stride_s,
                                        int heads, int sequence, int flags, void *workspace, size_t workspace_bytes,
                                        int32_t *status, h3s_stream_t stream) {
  using namespace h3s;
  AttnParams prm;
  int rc = fill_attn_params(&prm, q8, k8, v16t, q_scale, k_scale, v_scale, route, route_len, q_start, q_stop, out,
                            peer_out, n_peer_out, out_dtype, out_stride_h, out_stride_s, heads, sequence, flags, status,
                            "sparse_attn_half_fwd");
  if (rc) return rc;
  const uint64_t S = static_cast<uint64_t>(sequence);
  const uint64_t row_bytes = static_cast<uint64_t>(ceil_div(sequence, 128)) * 128 * 2;
  CUtensorMap mk, mv;
  rc = make_tensor_map_u8_3d(&mk, k8, H3S_HEAD_DIM, S, heads, H3S_HEAD_DIM, S * H3S_HEAD_DIM, H3S_HEAD_DIM,
                             H3S_KV_TILE, CU_TENSOR_MAP_SWIZZLE_128B, "sparse_attn_half_fwd K map");
  if (rc) return rc;
  rc = make_tensor_map_u8_3d(&mv, v16t, row_bytes, H3S_HEAD_DIM, heads, row_bytes, row_bytes * H3S_HEAD_DIM,
                             H3S_KV_TILE * 2, H3S_HEAD_DIM, CU_TENSOR_MAP_SWIZZLE_128B, "sparse_attn_half_fwd V map");
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  prm.parts = 1; prm.part_tiles = prm.kv_tiles; prm.partial = nullptr; prm.arrived = nullptr;
  if (workspace != nullptr) {
    const int n_sparse = route != nullptr ? q_stop - q_start : 0;
    int part_tiles;
    const int parts = split_dense_rows(heads, prm.q_tiles, prm.kv_tiles, n_sparse, n_sparse ? route_len : 0, &part_tiles);
    size_t arrived_bytes;
    const size_t need = split_bytes(static_cast<int64_t>(heads) * (prm.q_tiles - n_sparse), parts, &arrived_bytes);
    if (parts > 1) {
      H3S_CHECK_ARG(workspace_bytes >= need && (reinterpret_cast<uintptr_t>(workspace) & 15) == 0,
                    "sparse_attn_half_fwd: the workspace must be 16-byte aligned and hold %zu bytes, got %zu", need, workspace_bytes);
      prm.parts = parts; prm.part_tiles = part_tiles;
      prm.arrived = static_cast<unsigned int *>(workspace);
      prm.partial = reinterpret_cast<float *>(static_cast<unsigned char *>(workspace) + arrived_bytes);
      H3S_CHECK_CUDA(cudaMemsetAsync(workspace, 0, arrived_bytes, s));
    }
  }
  switch (out_dtype) {
    case H3S_F32: return launch_attn_half<float>(mk, mv, q8, prm, s);
    case H3S_BF16: return launch_attn_half<__nv_bfloat16>(mk, mv, q8, prm, s);
    default: return launch_attn_half<__half>(mk, mv, q8, prm, s);
  }
}
