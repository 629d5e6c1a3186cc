// Carrier quantisation kernels (HBM-bound): whole-sequence column statistics,
// per-block INT8 Q/K with tile means, FP8-E4M3 transposed V.
//
// Thread mapping shared by all three: 16 consecutive threads read one
// 128-channel row as 16-byte vectors (8 channels each), so a warp covers two
// full rows and every global load/store is a fully used 128/256/512-byte line.
#include <mutex>
#include <type_traits>

#include "attn_common.cuh"

namespace h3s {

// ---------------------------------------------------------------------------
// Column statistics: sum_s K[h,s,d] (FP64) and max_s |V[h,s,d]|.
// scratch layout: double k_sum[heads*128]; uint32 v_amax_bits[heads*128].
// ---------------------------------------------------------------------------

constexpr int kStatsThreads = 256;
constexpr int kStatsRowsPerBlock = 512;

// Rows [row_begin, row_end) of one head: column sums of K, or column maxima of V, added to the head's totals.  Where registers are plenty
// (80 here) the choice is left to run time: as two bodies the compiler made do with 52, and three heads of 33272 tokens took 20 us beside the
// Q quantiser instead of 15; a kernel of 64 registers spills with one body for both.
enum StatsOf { kStatsOfK, kStatsOfV, kStatsOfEither };
template <typename T, StatsOf kOf, int kAhead = 8>
__device__ __forceinline__ void column_stats_rows(const T *__restrict__ src, int64_t stride_s, int row_begin, int row_end, bool v_now,
                                                  double (&red)[kStatsThreads / 16][H3S_HEAD_DIM], double *__restrict__ k_sum,
                                                  unsigned int *__restrict__ v_amax_bits) {
  const bool is_v = kOf == kStatsOfEither ? v_now : kOf == kStatsOfV;
  const int slot = threadIdx.x >> 4;
  const int c0 = (threadIdx.x & 15) * 8;
  double acc[8];
  float amax[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { acc[i] = 0.0; amax[i] = 0.f; }
  const T *base = src + c0;
  // kAhead rows are requested before the first is used (rows past the end count as zeros), eight for one:
  // 24 heads x 33272 tokens 117 -> 85 us, 3 heads 32 -> 22 us
  constexpr int kStep = kStatsThreads / 16;
  for (int row = row_begin + slot; row < row_end; row += kStep * kAhead) {
    typename Elem<T>::Raw raw[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      raw[u] = Elem<T>::load_raw_if(base + (row + u * kStep) * stride_s, row + u * kStep < row_end);
    if (is_v) {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        float x[8];
        Elem<T>::unpack(raw[u], x);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax[i] = fmaxf(amax[i], fabsf(x[i]));
      }
    } else {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        float x[8];
        Elem<T>::unpack(raw[u], x);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += static_cast<double>(x[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[slot][c0 + i] = is_v ? static_cast<double>(amax[i]) : acc[i];
  __syncthreads();
  if (threadIdx.x < H3S_HEAD_DIM) {
    const int d = threadIdx.x;
    if (is_v) {
      double m = 0.0;
#pragma unroll
      for (int s = 0; s < kStatsThreads / 16; ++s) m = fmax(m, red[s][d]);
      // non-negative floats order like their bit patterns
      atomicMax(&v_amax_bits[d], __float_as_uint(static_cast<float>(m)));
    } else {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < kStatsThreads / 16; ++i) s += red[i][d];
      atomicAdd(&k_sum[d], s);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kStatsThreads)
column_stats_kernel(const T *__restrict__ k, int64_t k_stride_h, int64_t k_stride_s,
                    const T *__restrict__ v, int64_t v_stride_h, int64_t v_stride_s,
                    int sequence, double *__restrict__ k_sum,
                    unsigned int *__restrict__ v_amax_bits) {
  __shared__ double red[kStatsThreads / 16][H3S_HEAD_DIM];
  let_next_start();
  wait_for_previous();
  const int head = blockIdx.y;
  const bool is_v = blockIdx.z == 1;
  const T *src = is_v ? v : k;
  if (src == nullptr) return;
  const int row_begin = blockIdx.x * kStatsRowsPerBlock;
  column_stats_rows<T, kStatsOfEither>(src + head * (is_v ? v_stride_h : k_stride_h), is_v ? v_stride_s : k_stride_s, row_begin,
                    min(row_begin + kStatsRowsPerBlock, sequence), is_v, red, k_sum + head * H3S_HEAD_DIM, v_amax_bits + head * H3S_HEAD_DIM);
}

template <typename T>
__device__ __forceinline__ float finalize_mean(double sum, int sequence) {
  return Elem<T>::round_trip(static_cast<float>(sum / static_cast<double>(sequence)));
}
__device__ __forceinline__ float finalize_scale(unsigned int amax_bits, float v_bound) {
  return fmaxf(__fdiv_rn(__uint_as_float(amax_bits), v_bound), 1.0e-20f);
}

template <typename T>
__global__ void column_stats_finalize_kernel(const double *__restrict__ k_sum,
                                             const unsigned int *__restrict__ v_amax_bits,
                                             int total, int sequence, float v_bound,
                                             float *__restrict__ k_mean,
                                             float *__restrict__ v_scale) {
  let_next_start();
  wait_for_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  if (k_mean != nullptr) k_mean[i] = finalize_mean<T>(load_written(k_sum + i), sequence);
  if (v_scale != nullptr) v_scale[i] = finalize_scale(load_written(v_amax_bits + i), v_bound);
}

// ---------------------------------------------------------------------------
// Per-block INT8 quantisation with optional tile means.
// One CTA = one (block, head); the whole block lives in registers, as loaded
// (64 values per thread, 32 registers for 16-bit inputs), between the amax
// reduction and the store, so it is read from memory exactly once.
// ---------------------------------------------------------------------------

template <int BLOCK>
struct QkShared {
  float warp_amax[BLOCK / 16];
  double red[BLOCK / 8][H3S_HEAD_DIM];
};

// One block of BLOCK rows by 2 * BLOCK threads, of which this is the t-th.  `x` is the block's first row, `out` the carrier's.  `sync` lets
// these threads meet; `minus_mean(m)` gives this thread's eight channels of the mean, negated (x - mu == x + (-mu)), and is called when the
// block's loads have been issued.
template <typename T, int BLOCK, bool kHasMean, typename Sync, typename Mean>
__device__ __forceinline__ void quant_qk_block(const T *__restrict__ x, int64_t stride_s, int valid_rows, int8_t *__restrict__ out,
                                               float *__restrict__ scale_out, void *__restrict__ summary, int summary_dtype,
                                               int64_t summary_at, int t, QkShared<BLOCK> &sh, Sync sync, Mean minus_mean) {
  constexpr int kThreads = BLOCK * 2;
  constexpr int kSlots = kThreads / 16;  // rows per pass
  constexpr int kPasses = BLOCK / kSlots;  // == 8
  const int slot = t >> 4;
  const int c0 = (t & 15) * 8;
  typename Elem<T>::Raw raw[kPasses];
  float2 col[4];  // this thread's rows (at most 8) summed in fp32, widened once
#pragma unroll
  for (int i = 0; i < 4; ++i) col[i] = make_float2(0.f, 0.f);
  float amax = 0.f;
  const T *base = x + c0;
#pragma unroll
  for (int p = 0; p < kPasses; ++p) {
    const int r = p * kSlots + slot;
    raw[p] = Elem<T>::load_raw_if(base + r * stride_s, r < valid_rows);
  }
  float2 minus_mu[4];
  minus_mean(minus_mu);
#pragma unroll
  for (int p = 0; p < kPasses; ++p) {
    const int r = p * kSlots + slot;
    if (r < valid_rows) {
      float v[8];
      Elem<T>::unpack(raw[p], v);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 pair = make_float2(v[2 * i], v[2 * i + 1]);
        col[i] = add2(col[i], pair);
        const float2 x = kHasMean ? add2(pair, minus_mu[i]) : pair;
        amax = fmaxf(amax, fmaxf(fabsf(x.x), fabsf(x.y)));
      }
    }
  }
  amax = warp_max(amax);
  if ((t & 31) == 0) sh.warp_amax[t >> 5] = amax;
  if (summary != nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sh.red[slot][c0 + 2 * i] = static_cast<double>(col[i].x);
      sh.red[slot][c0 + 2 * i + 1] = static_cast<double>(col[i].y);
    }
  }
  sync();
  amax = sh.warp_amax[0];
#pragma unroll
  for (int w = 1; w < kThreads / 32; ++w) amax = fmaxf(amax, sh.warp_amax[w]);
  const float scale = __fadd_rn(__fdiv_rn(amax, 127.0f), 1.0e-7f);
  const SharedDivisor by_scale = make_divisor(scale);

  if (t == 0 && scale_out != nullptr) *scale_out = scale;

  int8_t *dst = out + c0;
  // code = trunc(v/scale +- 0.5): the half carries the quotient's sign bit, the four
  // codes of a word are gathered with byte permutes.  The divisor's exactness is
  // tested once, around the whole loop (see divide<>).
  auto emit = [&](auto exact_tag) {
    constexpr bool kExact = decltype(exact_tag)::value;
#pragma unroll
    for (int p = 0; p < kPasses; ++p) {
      const int r = p * kSlots + slot;
      if (out != nullptr && r < valid_rows) {
        float v[8];
        Elem<T>::unpack(raw[p], v);
        uint32_t code[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 pair = make_float2(v[2 * i], v[2 * i + 1]);
          round_codes(divide2<kExact>(by_scale, kHasMean ? add2(pair, minus_mu[i]) : pair), code[2 * i], code[2 * i + 1]);
        }
        uint32_t packed[2];
#pragma unroll
        for (int w = 0; w < 2; ++w)
          packed[w] = __byte_perm(__byte_perm(code[4 * w], code[4 * w + 1], 0x0040),
                                  __byte_perm(code[4 * w + 2], code[4 * w + 3], 0x0040), 0x5410);
        *reinterpret_cast<uint2 *>(dst + static_cast<int64_t>(r) * H3S_HEAD_DIM) = make_uint2(packed[0], packed[1]);
      }
    }
  };
  if (by_scale.exact) emit(std::true_type{}); else emit(std::false_type{});

  if (summary != nullptr && t < H3S_HEAD_DIM) {
    const int d = t;
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < kSlots; ++i) s += sh.red[i][d];
    const double m = valid_rows == BLOCK ? s * (1.0 / BLOCK) : s / static_cast<double>(valid_rows);  // a power of two divides exactly
    const int64_t at = summary_at + d;
    switch (summary_dtype) {
      case H3S_F64: static_cast<double *>(summary)[at] = m; break;
      case H3S_F32: static_cast<float *>(summary)[at] = static_cast<float>(m); break;
      case H3S_BF16:
        static_cast<__nv_bfloat16 *>(summary)[at] = __float2bfloat16_rn(static_cast<float>(m));
        break;
      default:
        static_cast<__half *>(summary)[at] = __float2half_rn(static_cast<float>(m));
        break;
    }
  }
}

template <typename T, int BLOCK, bool kHasMean>
__global__ void __launch_bounds__(BLOCK * 2, (sizeof(T) == 2 ? 1024 : 512) / (BLOCK * 2))
quant_qk_blocks_kernel(const T *__restrict__ x, int64_t stride_h, int64_t stride_s,
                       const float *__restrict__ mean, int8_t *__restrict__ out,
                       float *__restrict__ scale_out, void *__restrict__ summary,
                       int summary_dtype, int rows, int row_start, int sequence_total,
                       int blocks_total) {
  __shared__ QkShared<BLOCK> sh;
  let_next_start();
  wait_for_previous();
  const int head = blockIdx.y;
  const int first_row = blockIdx.x * BLOCK;  // within this chunk
  const int64_t block = static_cast<int64_t>(head) * blocks_total + row_start / BLOCK + blockIdx.x;
  // Here the mean is complete, and asked for before the rows.  us, behind the rows / before them: fp32 24 heads x 1000 tokens 4.9 / 4.6, 3 x
  // 33272 13.3 / 13.1, bf16 3 x 33272 9.5 / 9.2, 24 x 33272 66.9 / 66.7.
  float2 minus_mu[4];
  if (kHasMean) {
    const float *mu = mean + head * H3S_HEAD_DIM + (threadIdx.x & 15) * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) minus_mu[i] = make_float2(-load_written(mu + 2 * i), -load_written(mu + 2 * i + 1));
  }
  auto minus_mean = [&](float2 (&m)[4]) {
    if (!kHasMean) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) m[i] = minus_mu[i];
  };
  quant_qk_block<T, BLOCK, kHasMean>(
      x + head * stride_h + first_row * stride_s, stride_s, min(BLOCK, rows - first_row),
      out == nullptr ? nullptr : out + (static_cast<int64_t>(head) * sequence_total + row_start + first_row) * H3S_HEAD_DIM,
      scale_out == nullptr ? nullptr : scale_out + block, summary, summary_dtype, block * H3S_HEAD_DIM, threadIdx.x, sh,
      []() { __syncthreads(); }, minus_mean);
}

// ---------------------------------------------------------------------------
// FP8-E4M3 V carrier, transposed to (heads, 128, pad128(S)).
// One CTA = 128 sequence rows of one head, staged through shared memory so
// that both the row-major reads and the channel-major writes are full lines.
// All eight rows of a thread are requested before the first is used, and the FP16 copy
// is written as whole lines of 256 bytes (two 16-byte pieces a thread with a gap between
// them cost twice the L2 writes): 24 heads x 33272 tokens 133 -> 88 us.
// ---------------------------------------------------------------------------

constexpr int kVTile = 128;
constexpr int kVThreads = 256;

// Shared tile: 128 channel rows of 128 bytes; the 16-byte chunk index of
// channel row d is XORed with (d>>3)&7 so the transposing 4-byte stores of
// the 16 lanes that share a sequence position fall in different banks.
__device__ __forceinline__ int v_tile_offset(int d, int s) {
  const int chunk = (s >> 4) ^ ((d >> 3) & 7);
  return d * kVTile + chunk * 16 + (s & 15);
}

// One tile of 128 sequence rows by 256 threads.  `v` is its first row, `out` and `out_half` the tile's first column of the head's carrier;
// `scales(s)` gives this thread's eight channels' scales and is called when the tile's loads have been issued.
template <typename T, typename Scales>
__device__ __forceinline__ void quant_v_tile(const T *__restrict__ v, int64_t stride_s, int valid_rows, uint8_t *__restrict__ out,
                                             uint16_t *__restrict__ out_half, int padded_total, float v_bound,
                                             uint8_t (&tile)[H3S_HEAD_DIM * kVTile], Scales scales) {
  const int slot = threadIdx.x >> 4;
  const int c0 = (threadIdx.x & 15) * 8;
  const T *base = v + c0;
  constexpr int kPasses = kVTile / (kVThreads / 16 * 4);
  typename Elem<T>::Raw raw[kPasses][4];
#pragma unroll
  for (int p = 0; p < kPasses; ++p) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = (p * (kVThreads / 16) + slot) * 4 + j;  // four consecutive rows
      raw[p][j] = Elem<T>::load_raw_if(base + r * stride_s, r < valid_rows);  // 0 / scale is the padding's code
    }
  }
  float2 minus_sc[4], rc[4];
  bool all_exact = true;
  const bool clamp = v_bound < 448.0f;
  {
    float scale[8];
    scales(scale);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const SharedDivisor a = make_divisor(fmaxf(scale[2 * i], 1.0e-20f)), b = make_divisor(fmaxf(scale[2 * i + 1], 1.0e-20f));
      minus_sc[i] = make_float2(-a.b, -b.b);
      rc[i] = make_float2(a.r, b.r);
      all_exact = all_exact && a.exact && b.exact;
    }
  }
  // the divisors' exactness is tested once, around the whole loop (see divide<>)
  auto fill = [&](auto exact_tag) {
  constexpr bool kExact = decltype(exact_tag)::value;
#pragma unroll
  for (int p = 0; p < kPasses; ++p) {
    const int r0 = (p * (kVThreads / 16) + slot) * 4;
    // four consecutive rows of 8 channels -> per channel one word of four codes
    // (two 2-wide conversions and one byte permute)
    float q[4][8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x[8];
      Elem<T>::unpack(raw[p][j], x);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 pair = make_float2(x[2 * i], x[2 * i + 1]);
        float2 y;
        if (kExact) {  // shared-divisor division, see SharedDivisor
          const float2 q0 = mul2(pair, rc[i]);
          y = fma2(fma2(minus_sc[i], q0, pair), rc[i], q0);
        } else {
          y = make_float2(__fdiv_rn(pair.x, -minus_sc[i].x), __fdiv_rn(pair.y, -minus_sc[i].y));
        }
        // the conversion saturates at +-448 by itself; a tighter bound is applied here
        if (clamp) y = make_float2(fminf(fmaxf(y.x, -v_bound), v_bound), fminf(fmaxf(y.y, -v_bound), v_bound));
        q[j][2 * i] = y.x;
        q[j][2 * i + 1] = y.y;
      }
    }
    uint32_t word[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint16_t lo, hi;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(q[1][i]), "f"(q[0][i]));
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(q[3][i]), "f"(q[2][i]));
      word[i] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<uint32_t *>(&tile[v_tile_offset(c0 + i, r0)]) = word[i];
  }
  };
  if (all_exact) fill(std::true_type{}); else fill(std::false_type{});
  __syncthreads();
#pragma unroll
  for (int p = 0; p < H3S_HEAD_DIM / (kVThreads / 8); ++p) {
    const int d = p * (kVThreads / 8) + (threadIdx.x >> 3);
    const int chunk = threadIdx.x & 7;
    const uint4 data = *reinterpret_cast<const uint4 *>(&tile[v_tile_offset(d, chunk * 16)]);
    const int64_t at = static_cast<int64_t>(d) * padded_total + chunk * 16;
    *reinterpret_cast<uint4 *>(out + at) = data;
  }
  if (out_half != nullptr) {  // the copy the attention kernel multiplies with FP16 probabilities
#pragma unroll
    for (int p = 0; p < H3S_HEAD_DIM / (kVThreads / 16); ++p) {
      const int d = p * (kVThreads / 16) + slot, s = (threadIdx.x & 15) * 8;
      const uint2 data = *reinterpret_cast<const uint2 *>(&tile[v_tile_offset(d, s)]);
      *reinterpret_cast<uint4 *>(out_half + static_cast<int64_t>(d) * padded_total + s) = e4m3x8_to_half(data);
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kVThreads)
quant_v_fp8_kernel(const T *__restrict__ v, int64_t stride_h, int64_t stride_s,
                   const float *__restrict__ v_scale, uint8_t *__restrict__ out, uint16_t *__restrict__ out_half,
                   int rows, int row_start, int padded_total, float v_bound) {
  __shared__ __align__(16) uint8_t tile[H3S_HEAD_DIM * kVTile];
  let_next_start();
  wait_for_previous();
  const int head = blockIdx.y;
  const int first_row = blockIdx.x * kVTile;
  const int64_t at = static_cast<int64_t>(head) * H3S_HEAD_DIM * padded_total + row_start + first_row;
  quant_v_tile(v + head * stride_h + first_row * stride_s, stride_s, max(0, min(kVTile, rows - first_row)), out + at,
               out_half == nullptr ? nullptr : out_half + at, padded_total, v_bound, tile, [&](float (&scale)[8]) {
#pragma unroll
                 for (int i = 0; i < 8; ++i) scale[i] = load_written(v_scale + head * H3S_HEAD_DIM + (threadIdx.x & 15) * 8 + i);
               });
}

// ---------------------------------------------------------------------------
// Carriers of a layer in one launch: statistics of K and V, and the carriers of a head as soon as its statistics are complete.  Where
// layers are short, the chain of kernels for statistics, their end, Q, K and V is bound by latency, of the host and of the kernels: each fills
// the chip for a few microseconds and waits for the last block of the one before.  Here blocks take jobs in order, by a counter, and only K and
// V of a head wait for that head's statistics.  us, the chain on two streams / this with the clearing before it: 1 head x 1200 tokens 19.5 /
// 9.2, 4 x 2304 fp32 20.5 / 12.8, 24 x 2304 32.3 / 27.1, 7 x 10384 37.9 / 33.8, 24 x 9872 90.1 / 85.0.  Long layers 24 x 33272 269 / 263 by
// themselves, but it is the slower one behind an attention kernel, which leaves a lower SM clock: a job's bookkeeping is half as many
// instructions again as its work.  Sixty-four registers, four blocks an SM: with three and no spills 24 x 76112 692 for 650.  Measured and not
// kept: four steps of 128 rows to a job (24 x 76112 3 % faster, all short layers slower), a head's means and scales made by its last
// statistics job (4 x 2304 15.9 for 13.8), K and V right behind their head's statistics, with streaming hints (re-reads still miss L2).
// ---------------------------------------------------------------------------

constexpr int kCarrierThreads = 256, kCarrierRows = 128;  // rows of a step: one Q block, two K blocks or a tile of V
enum CarrierKind { kCarrierKStats, kCarrierVStats, kCarrierQ, kCarrierK, kCarrierV };

struct CarrierParams {
  const void *q, *k, *v;
  int64_t q_stride_h, q_stride_s, k_stride_h, k_stride_s, v_stride_h, v_stride_s;
  int8_t *q8, *k8;
  uint8_t *v8;
  uint16_t *v16;
  float *q_scale, *k_scale, *v_scale, *k_mean;
  void *q_summary, *k_summary;
  int summary_dtype;
  int heads, sequence, padded, steps;
  float v_bound;
  double *k_sum;                    // (heads, 128), and
  unsigned int *v_amax_bits;        // (heads, 128): totals, cleared before the launch with the counters below, or complete
  unsigned int *next, *stats_done;  // the next job; per head: statistics jobs that are through
  int32_t *status, *status_mirror;
  unsigned long long wait_budget_ns;
  int missing;                                   // self-test of the wait: statistics jobs of a head that it expects and nobody does
  int stats_rows;                                // of a statistics job
  int k_stats, v_stats, q_jobs, k_jobs, v_jobs;  // jobs of a head
};

struct CarrierJob {
  int kind, head, index;
};

// Jobs in the order in which they are taken: head by head the statistics and Q, which needs none, then head by head K and V.  What a job
// waits for comes before it, so whoever has the first job that is not through can go on, however many blocks run at a time.
__host__ __device__ inline CarrierJob carrier_job(const CarrierParams &p, int t) {
  const int early = p.k_stats + p.v_stats + p.q_jobs, late = p.k_jobs + p.v_jobs;
  if (t < p.heads * early) {
    const int head = t / early;
    t -= head * early;
    if (t < p.k_stats) return {kCarrierKStats, head, t};
    t -= p.k_stats;
    return t < p.v_stats ? CarrierJob{kCarrierVStats, head, t} : CarrierJob{kCarrierQ, head, t - p.v_stats};
  }
  t -= p.heads * early;
  const int head = t / late;
  t -= head * late;
  return t < p.k_jobs ? CarrierJob{kCarrierK, head, t} : CarrierJob{kCarrierV, head, t - p.k_jobs};
}

union CarrierShared {
  double red[kStatsThreads / 16][H3S_HEAD_DIM];
  QkShared<H3S_Q_TILE> q;
  QkShared<H3S_KV_TILE> k[2];
  uint8_t tile[H3S_HEAD_DIM * kVTile];
};
static_assert(kStatsThreads == kCarrierThreads && kVThreads == kCarrierThreads && kVTile == kCarrierRows, "carrier jobs");

// Until the count has reached `target`: what was written before the arrivals is visible to this thread then
__device__ __forceinline__ bool wait_for_count(const unsigned int *count, unsigned int target, unsigned long long budget_ns) {
  if (ptx::load_acquire(count) >= target) return true;
  const unsigned long long start = ptx::global_timer_ns();
  while (ptx::load_acquire(count) < target)
    if (ptx::global_timer_ns() - start > budget_ns) return false;
  return true;
}

template <typename T, bool kSmooth>
__global__ void __launch_bounds__(kCarrierThreads, sizeof(T) == 2 ? 4 : 2)
layer_carriers_kernel(const __grid_constant__ CarrierParams p) {
  __shared__ __align__(16) CarrierShared sh;
  __shared__ __align__(16) float head_values[H3S_HEAD_DIM];
  __shared__ int jobs[2];
  __shared__ bool late;  // the first thread's alone: its wait has run out
  let_next_start();
  wait_for_previous();
  const int total = p.heads * (p.k_stats + p.v_stats + p.q_jobs + p.k_jobs + p.v_jobs);
  const int t = threadIdx.x, c0 = (t & 15) * 8;
  int next = t == 0 ? static_cast<int>(atomicAdd(p.next, 1u)) : 0;
  if (t == 0) late = false;
  for (int turn = 0;; turn ^= 1) {
    if (t == 0) jobs[turn] = next;
    __syncthreads();  // and the job before this one has left shared memory
    const int number = jobs[turn];
    if (number >= total) break;
    if (t == 0) next = static_cast<int>(atomicAdd(p.next, 1u));  // asked for ahead of its use
    const CarrierJob job = carrier_job(p, number);
    const int head = job.head;
    if (job.kind <= kCarrierVStats) {
      constexpr int kAhead = sizeof(T) == 4 ? 4 : 8;  // as the registers allow
      const int begin = job.index * p.stats_rows, end = min(begin + p.stats_rows, p.sequence);
      if (job.kind == kCarrierKStats)
        column_stats_rows<T, kStatsOfK, kAhead>(static_cast<const T *>(p.k) + head * p.k_stride_h, p.k_stride_s, begin, end, false, sh.red,
                                                p.k_sum + head * H3S_HEAD_DIM, nullptr);
      else
        column_stats_rows<T, kStatsOfV, kAhead>(static_cast<const T *>(p.v) + head * p.v_stride_h, p.v_stride_s, begin, end, true, sh.red,
                                                nullptr, p.v_amax_bits + head * H3S_HEAD_DIM);
      __syncthreads();
      if (t == 0) {
        __threadfence();
        ptx::add_release(p.stats_done + head, 1u);
      }
      continue;
    }
    const int step = job.index, row = step * kCarrierRows;
    // The head's K mean or V scale, when its statistics are in; every thread calls it.  After a wait that has run out the block goes through
    // its jobs without another one: nobody else takes them, and what reads the carriers next is to find values, if wrong ones.
    auto wait_for_head = [&](bool is_v) {
      if (t == 0 && !late && !wait_for_count(p.stats_done + head, p.k_stats + p.v_stats + p.missing, p.wait_budget_ns)) {
        late = true;
        report_status(p.status, p.status_mirror, kAbortStatistics, number, head, step);
      }
      __syncthreads();
      if (t < H3S_HEAD_DIM) {
        const int at = head * H3S_HEAD_DIM + t;
        const float value = is_v ? finalize_scale(__ldcg(p.v_amax_bits + at), p.v_bound) : finalize_mean<T>(__ldcg(p.k_sum + at), p.sequence);
        head_values[t] = value;
        if (step == 0) (is_v ? p.v_scale : p.k_mean)[at] = value;
      }
      __syncthreads();
    };
    if (job.kind == kCarrierQ) {
      const int64_t block = static_cast<int64_t>(head) * p.steps + step;
      quant_qk_block<T, H3S_Q_TILE, false>(
          static_cast<const T *>(p.q) + head * p.q_stride_h + row * p.q_stride_s, p.q_stride_s, min(kCarrierRows, p.sequence - row),
          p.q8 + (static_cast<int64_t>(head) * p.sequence + row) * H3S_HEAD_DIM, p.q_scale + block, p.q_summary, p.summary_dtype,
          block * H3S_HEAD_DIM, t, sh.q, []() { __syncthreads(); }, [](float2 (&)[4]) {});
    } else if (job.kind == kCarrierK) {
      const int half = t >> 7, blocks = (p.sequence + H3S_KV_TILE - 1) / H3S_KV_TILE;
      const int half_row = row + half * H3S_KV_TILE;
      const int64_t block = static_cast<int64_t>(head) * blocks + 2 * step + half;
      const bool some = half_row < p.sequence;  // the last step's second block may be past the end: it is gone through, nothing is stored
      quant_qk_block<T, H3S_KV_TILE, kSmooth>(
          static_cast<const T *>(p.k) + head * p.k_stride_h + half_row * p.k_stride_s, p.k_stride_s, min(H3S_KV_TILE, p.sequence - half_row),
          some ? p.k8 + (static_cast<int64_t>(head) * p.sequence + half_row) * H3S_HEAD_DIM : nullptr, some ? p.k_scale + block : nullptr,
          some ? p.k_summary : nullptr, p.summary_dtype, block * H3S_HEAD_DIM, t & 127, sh.k[half], []() { __syncthreads(); },
          [&](float2 (&minus_mu)[4]) {
            if (!kSmooth) return;
            wait_for_head(false);
#pragma unroll
            for (int i = 0; i < 4; ++i) minus_mu[i] = make_float2(-head_values[c0 + 2 * i], -head_values[c0 + 2 * i + 1]);
          });
    } else {
      const int64_t at = static_cast<int64_t>(head) * H3S_HEAD_DIM * p.padded + row;
      quant_v_tile(static_cast<const T *>(p.v) + head * p.v_stride_h + row * p.v_stride_s, p.v_stride_s, min(kVTile, p.sequence - row),
                   p.v8 + at, p.v16 == nullptr ? nullptr : p.v16 + at, p.padded, p.v_bound, sh.tile, [&](float (&scale)[8]) {
                     wait_for_head(true);
#pragma unroll
                     for (int i = 0; i < 8; ++i) scale[i] = head_values[c0 + i];
                   });
    }
  }
}

// ---------------------------------------------------------------------------
// Second phase of the projection in one launch: K without its mean and V by its scale, from bf16 staging and complete totals.  For short
// sequences, which are bound by latency: every block makes its head's means or scales itself, from totals that it asks for before its rows, so
// that no kernel stands between the last projection tile and this one, and no second stream.  Long sequences go the other way, figures at
// h3s_project_qkv_norms; of the 19 us that they would lose 5 are the 64-bit divisions of every block.
// ---------------------------------------------------------------------------

template <bool kSmooth>
__global__ void __launch_bounds__(kCarrierThreads, 4)
staged_carriers_kernel(const __grid_constant__ CarrierParams p) {
  using T = __nv_bfloat16;
  __shared__ __align__(16) CarrierShared sh;
  __shared__ __align__(16) float head_values[H3S_HEAD_DIM];
  let_next_start();
  wait_for_previous();
  const int t = threadIdx.x, c0 = (t & 15) * 8;
  constexpr int kKinds = kSmooth ? 2 : 1;
  const int place = blockIdx.x / kKinds, head = place / p.steps;
  const int step = place - head * p.steps, row = step * kCarrierRows;
  const bool is_v = !kSmooth || blockIdx.x % kKinds != 0;
  const int at_value = head * H3S_HEAD_DIM + (t & (H3S_HEAD_DIM - 1));
  // asked for before the rows
  const double k_total = is_v ? 0.0 : load_written(p.k_sum + at_value);
  const unsigned int v_top = is_v ? load_written(p.v_amax_bits + at_value) : 0u;
  auto make_values = [&]() {
    if (t < H3S_HEAD_DIM) {
      const float value = is_v ? finalize_scale(v_top, p.v_bound) : finalize_mean<T>(k_total, p.sequence);
      head_values[t] = value;
      if (step == 0) (is_v ? p.v_scale : p.k_mean)[at_value] = value;
    }
    __syncthreads();
  };
  if (kSmooth && !is_v) {
    const int half = t >> 7, blocks = (p.sequence + H3S_KV_TILE - 1) / H3S_KV_TILE;
    const int half_row = row + half * H3S_KV_TILE;
    const bool some = half_row < p.sequence;  // the last step's second block may be past the end: it is gone through, nothing is stored
    quant_qk_block<T, H3S_KV_TILE, true>(
        static_cast<const T *>(p.k) + head * p.k_stride_h + half_row * p.k_stride_s, p.k_stride_s, min(H3S_KV_TILE, p.sequence - half_row),
        some ? p.k8 + (static_cast<int64_t>(head) * p.sequence + half_row) * H3S_HEAD_DIM : nullptr,
        some ? p.k_scale + static_cast<int64_t>(head) * blocks + 2 * step + half : nullptr, nullptr, H3S_F32, 0, t & 127, sh.k[half],
        []() { __syncthreads(); }, [&](float2 (&minus_mu)[4]) {
          make_values();
#pragma unroll
          for (int i = 0; i < 4; ++i) minus_mu[i] = make_float2(-head_values[c0 + 2 * i], -head_values[c0 + 2 * i + 1]);
        });
  } else {
    const int64_t at = static_cast<int64_t>(head) * H3S_HEAD_DIM * p.padded + row;
    quant_v_tile(static_cast<const T *>(p.v) + head * p.v_stride_h + row * p.v_stride_s, p.v_stride_s, min(kVTile, p.sequence - row),
                 p.v8 + at, p.v16 == nullptr ? nullptr : p.v16 + at, p.padded, p.v_bound, sh.tile, [&](float (&scale)[8]) {
                   make_values();
#pragma unroll
                   for (int i = 0; i < 8; ++i) scale[i] = head_values[c0 + i];
                 });
  }
}

__global__ void __launch_bounds__(256) clear_words_kernel(unsigned int *words, int n, unsigned int *more, int m) {
  let_next_start();
  wait_for_previous();
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n + m; i += gridDim.x * 256) (i < n ? words[i] : more[i - n]) = 0u;
}

// ---------------------------------------------------------------------------
// Per-row FP8-E4M3 quantisation of a bf16 matrix (activations of the FP8 MLP).
// Kept in registers between the amax reduction and the store.  Rows of up to 4096
// channels: one warp each, no barrier, all loads of the row in flight (4096 x 3072: 23 -> 13 us);
// longer rows: one CTA each.
// ---------------------------------------------------------------------------

// E4M3 codes of 8 consecutive channels
template <bool kExact>
__device__ __forceinline__ uint2 row_codes8(const SharedDivisor &by_scale, const float (&v)[8]) {
  uint32_t word[2];
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    uint16_t lo, hi;
    const float2 a = divide2<kExact>(by_scale, make_float2(v[4 * w], v[4 * w + 1]));
    const float2 b = divide2<kExact>(by_scale, make_float2(v[4 * w + 2], v[4 * w + 3]));
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(lo) : "f"(a.y), "f"(a.x));
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(hi) : "f"(b.y), "f"(b.x));
    word[w] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
  }
  return make_uint2(word[0], word[1]);
}

constexpr int kRowWarps = 4;  // rows (warps) per CTA

template <int kChunks>  // 16-byte loads per lane
__global__ void __launch_bounds__(kRowWarps * 32)
quant_rows_fp8_warp_kernel(const __nv_bfloat16 *__restrict__ x, int64_t stride_row, int rows, int channels,
                           uint8_t *__restrict__ out, float *__restrict__ row_scale) {
  let_next_start();
  wait_for_previous();
  const int row = blockIdx.x * kRowWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const __nv_bfloat16 *src = x + row * stride_row;
  Elem<__nv_bfloat16>::Raw raw[kChunks];
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int c0 = (i * 32 + lane) * 8;
    raw[i] = c0 < channels ? Elem<__nv_bfloat16>::load_raw(src + c0) : Elem<__nv_bfloat16>::zero_raw();
  }
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    float v[8];
    Elem<__nv_bfloat16>::unpack(raw[i], v);
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
  }
  amax = warp_max(amax);
  const float scale = fmaxf(__fdiv_rn(amax, 448.0f), 1.0e-20f);
  if (lane == 0) row_scale[row] = scale;
  const SharedDivisor by_scale = make_divisor(scale);
  uint8_t *dst = out + static_cast<int64_t>(row) * channels;
  auto emit = [&](auto exact_tag) {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      const int c0 = (i * 32 + lane) * 8;
      float v[8];
      Elem<__nv_bfloat16>::unpack(raw[i], v);
      if (c0 < channels) *reinterpret_cast<uint2 *>(dst + c0) = row_codes8<decltype(exact_tag)::value>(by_scale, v);
    }
  };
  if (by_scale.exact) emit(std::true_type{}); else emit(std::false_type{});
}

constexpr int kRowQuantThreads = 256;
constexpr int kRowQuantMaxChunks = 8;  // 16-byte loads per thread: rows of up to 16384 channels

__global__ void __launch_bounds__(kRowQuantThreads)
quant_rows_fp8_kernel(const __nv_bfloat16 *__restrict__ x, int64_t stride_row, int rows, int channels,
                      uint8_t *__restrict__ out, float *__restrict__ row_scale) {
  __shared__ float warp_amax[kRowQuantThreads / 32];
  let_next_start();
  wait_for_previous();
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16 *src = x + row * stride_row;
    Elem<__nv_bfloat16>::Raw raw[kRowQuantMaxChunks];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < kRowQuantMaxChunks; ++i) {
      const int c0 = (i * kRowQuantThreads + threadIdx.x) * 8;
      raw[i] = c0 < channels ? Elem<__nv_bfloat16>::load_raw(src + c0) : Elem<__nv_bfloat16>::zero_raw();
      float v[8];
      Elem<__nv_bfloat16>::unpack(raw[i], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
    }
    amax = warp_max(amax);
    __syncthreads();  // the previous row's readers are done
    if ((threadIdx.x & 31) == 0) warp_amax[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = warp_amax[0];
#pragma unroll
    for (int w = 1; w < kRowQuantThreads / 32; ++w) amax = fmaxf(amax, warp_amax[w]);
    const float scale = fmaxf(__fdiv_rn(amax, 448.0f), 1.0e-20f);
    if (threadIdx.x == 0) row_scale[row] = scale;
    const SharedDivisor by_scale = make_divisor(scale);
    auto emit = [&](auto exact_tag) {
      constexpr bool kExact = decltype(exact_tag)::value;
#pragma unroll
      for (int i = 0; i < kRowQuantMaxChunks; ++i) {
        const int c0 = (i * kRowQuantThreads + threadIdx.x) * 8;
        if (c0 < channels) {
          float v[8];
          Elem<__nv_bfloat16>::unpack(raw[i], v);
          *reinterpret_cast<uint2 *>(out + static_cast<int64_t>(row) * channels + c0) = row_codes8<kExact>(by_scale, v);
        }
      }
    };
    if (by_scale.exact) emit(std::true_type{}); else emit(std::false_type{});
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

static int check_view(const void *p, int dtype, int64_t stride_h, int64_t stride_s, const char *what) {
  const int vec = dtype == H3S_F32 ? 4 : 8;  // elements per 16 bytes
  H3S_CHECK_ARG(dtype == H3S_F32 || dtype == H3S_BF16 || dtype == H3S_F16,
                "%s: unsupported dtype %d", what, dtype);
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(p) & 15) == 0, "%s: pointer must be 16-byte aligned", what);
  H3S_CHECK_ARG(stride_h % vec == 0 && stride_s % vec == 0 && stride_s >= H3S_HEAD_DIM,
                "%s: strides (%lld,%lld) must be multiples of %d elements with row stride >= 128",
                what, static_cast<long long>(stride_h), static_cast<long long>(stride_s), vec);
  return H3S_OK;
}

template <typename T>
static int launch_column_stats(const void *k, int64_t ksh, int64_t kss, const void *v, int64_t vsh,
                               int64_t vss, int heads, int sequence, float v_bound, float *k_mean,
                               float *v_scale, void *scratch, cudaStream_t stream) {
  double *k_sum = static_cast<double *>(scratch);
  unsigned int *v_bits = reinterpret_cast<unsigned int *>(k_sum + heads * H3S_HEAD_DIM);
  H3S_CHECK_CUDA(cudaMemsetAsync(scratch, 0, h3s_column_stats_scratch_bytes(heads), stream));
  dim3 grid(ceil_div(sequence, kStatsRowsPerBlock), heads, 2);
  H3S_CHECK_CUDA(launch_next(column_stats_kernel<T>, grid, kStatsThreads, 0, stream, static_cast<const T *>(k), ksh, kss,
                             static_cast<const T *>(v), vsh, vss, sequence, k_sum, v_bits));
  const int total = heads * H3S_HEAD_DIM;
  H3S_CHECK_CUDA(launch_next(column_stats_finalize_kernel<T>, ceil_div(total, 256), 256, 0, stream, k_sum, v_bits, total, sequence,
                             v_bound, k == nullptr ? nullptr : k_mean, v == nullptr ? nullptr : v_scale));
  return H3S_OK;
}

template <typename T>
static int launch_quant_qk(const void *x, int64_t sh, int64_t ss, const float *mean, int8_t *out,
                           float *scale, void *summary, int summary_dtype, int heads, int rows,
                           int row_start, int sequence_total, int block, cudaStream_t stream) {
  const int blocks = ceil_div(rows, block);
  const int blocks_total = ceil_div(sequence_total, block);
  dim3 grid(blocks, heads);
#define H3S_LAUNCH_QK(BLOCK, HAS_MEAN)                                                               \
  H3S_CHECK_CUDA(launch_next(quant_qk_blocks_kernel<T, BLOCK, HAS_MEAN>, grid, BLOCK * 2, 0, stream,                     \
                             static_cast<const T *>(x), sh, ss, mean, out, scale, summary, summary_dtype, rows, row_start, \
                             sequence_total, blocks_total))
  if (block == H3S_Q_TILE) {
    if (mean != nullptr) H3S_LAUNCH_QK(H3S_Q_TILE, true); else H3S_LAUNCH_QK(H3S_Q_TILE, false);
  } else {
    if (mean != nullptr) H3S_LAUNCH_QK(H3S_KV_TILE, true); else H3S_LAUNCH_QK(H3S_KV_TILE, false);
  }
#undef H3S_LAUNCH_QK
  return H3S_OK;
}

template <typename T>
static int launch_quant_v(const void *v, int64_t sh, int64_t ss, const float *v_scale, uint8_t *out,
                          uint16_t *out_half, int heads, int rows, int row_start, int sequence_total, float v_bound,
                          cudaStream_t stream) {
  const int padded_total = ceil_div(sequence_total, 128) * 128;
  // the final chunk also writes the zero padding up to the carrier's end
  const bool last = row_start + rows == sequence_total;
  const int covered = last ? padded_total - row_start : rows;
  dim3 grid(ceil_div(covered, kVTile), heads);
  H3S_CHECK_CUDA(launch_next(quant_v_fp8_kernel<T>, grid, kVThreads, 0, stream, static_cast<const T *>(v), sh, ss, v_scale, out,
                             out_half, rows, row_start, padded_total, v_bound));
  return H3S_OK;
}

// Rows of a statistics job: as many as leave enough jobs for all SMs at once, since everything but Q waits for the last of them.  us,
// both kernels, jobs of 128 / 256 / 512 / 1024 rows: 4 heads x 2304 tokens, fp32 13 / 16 / 22 / 32, 7 x 10384 37 / 35 / 38 / 46, 24 x 2304
// 30 / 29 / 31 / 36, 8 x 20000 71 / 66 / 64 / 69, 24 x 33272 315 / 289 / 279 / 276.
static int carrier_stats_rows(int heads, int sequence, bool smooth_k) {
  constexpr int64_t kEnough = 380;
  int rows = 1024;
  while (rows > 64 && static_cast<int64_t>(heads) * ceil_div(sequence, rows) * (smooth_k ? 2 : 1) < kEnough) rows /= 2;
  return rows;
}

template <typename T>
static int launch_layer_carriers(const CarrierParams &p, bool smooth_k, cudaStream_t stream) {
  constexpr int kResident = kSmCount * (sizeof(T) == 2 ? 4 : 2);
  const int jobs = p.heads * (p.k_stats + p.v_stats + p.q_jobs + p.k_jobs + p.v_jobs);
  const int grid = jobs < kResident ? jobs : kResident;
  if (smooth_k) H3S_CHECK_CUDA(launch_next(layer_carriers_kernel<T, true>, grid, kCarrierThreads, 0, stream, p));
  else H3S_CHECK_CUDA(launch_next(layer_carriers_kernel<T, false>, grid, kCarrierThreads, 0, stream, p));
  return H3S_OK;
}

int staged_carriers(const h3s_layer_carriers *c, const void *k_stage, const void *v_stage, int heads, int sequence, bool smooth_k,
                    float v_bound, cudaStream_t stream) {
  H3S_CHECK_ARG(v_bound > 0.f, "project_qkv: v_bound must be positive");
  H3S_CHECK_ARG(c->v8 && c->v_scale && v_stage && (!smooth_k || (c->k8 && c->k_scale && c->k_mean && k_stage)), "project_qkv: NULL carrier");
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(c->k8) | reinterpret_cast<uintptr_t>(c->scratch)) & 7) == 0 &&
                ((reinterpret_cast<uintptr_t>(c->v8) | reinterpret_cast<uintptr_t>(c->v16)) & 15) == 0, "project_qkv: misaligned buffers");
  CarrierParams p = {};
  p.k = k_stage; p.v = v_stage;
  p.k_stride_h = p.v_stride_h = static_cast<int64_t>(sequence) * H3S_HEAD_DIM;
  p.k_stride_s = p.v_stride_s = H3S_HEAD_DIM;
  if (smooth_k) {
    int rc = check_view(k_stage, H3S_BF16, p.k_stride_h, p.k_stride_s, "project_qkv k_stage");
    if (rc) return rc;
  }
  { int rc = check_view(v_stage, H3S_BF16, p.v_stride_h, p.v_stride_s, "project_qkv v_stage"); if (rc) return rc; }
  p.k8 = c->k8; p.v8 = c->v8; p.v16 = static_cast<uint16_t *>(c->v16);
  p.k_scale = c->k_scale; p.v_scale = c->v_scale; p.k_mean = c->k_mean;
  p.heads = heads; p.sequence = sequence; p.padded = ceil_div(sequence, kVTile) * kVTile; p.v_bound = v_bound;
  p.k_sum = static_cast<double *>(c->scratch);
  p.v_amax_bits = reinterpret_cast<unsigned int *>(p.k_sum + heads * H3S_HEAD_DIM);
  p.steps = ceil_div(sequence, kCarrierRows);
  const int grid = heads * p.steps * (smooth_k ? 2 : 1);
  if (smooth_k) H3S_CHECK_CUDA(launch_next(staged_carriers_kernel<true>, grid, kCarrierThreads, 0, stream, p));
  else H3S_CHECK_CUDA(launch_next(staged_carriers_kernel<false>, grid, kCarrierThreads, 0, stream, p));
  return H3S_OK;
}

// ---------------------------------------------------------------------------
// Scratch that lives inside the library image, for hosts that cannot hand
// h3s_column_stats a scratch buffer of their own (see h3s_column_stats_static).
// Every device that loads this library carries one copy (96 KiB) until the
// process exits.  In host code the name below is only a stand-in for the
// symbol; the device address comes from cudaGetSymbolAddress, once per device.
// ---------------------------------------------------------------------------

constexpr int kStaticStatsMaxHeads = 64;
constexpr size_t kStaticStatsBytes =
    static_cast<size_t>(kStaticStatsMaxHeads) * H3S_HEAD_DIM * (sizeof(double) + sizeof(unsigned int));
static __device__ __align__(256) unsigned char g_static_stats_scratch[kStaticStatsBytes];

constexpr int kStaticStatsMaxDevices = 64;
static void *g_static_stats_addr[kStaticStatsMaxDevices] = {nullptr};
static std::mutex g_static_stats_mutex;

// Device address of the built-in scratch on the CURRENT device (looked up on
// the first call for that device, cached afterwards).
static int static_stats_scratch(void **out) {
  int device = 0;
  H3S_CHECK_CUDA(cudaGetDevice(&device));
  H3S_CHECK_ARG(device >= 0 && device < kStaticStatsMaxDevices,
                "column_stats_static: device ordinal %d is beyond the %d this library tracks", device,
                kStaticStatsMaxDevices);
  std::lock_guard<std::mutex> lock(g_static_stats_mutex);
  if (g_static_stats_addr[device] == nullptr) {
    void *ptr = nullptr;
    H3S_CHECK_CUDA(cudaGetSymbolAddress(&ptr, g_static_stats_scratch));
    H3S_CHECK_ARG(ptr != nullptr, "column_stats_static: the built-in scratch has no device address");
    g_static_stats_addr[device] = ptr;
  }
  *out = g_static_stats_addr[device];
  return H3S_OK;
}

}  // namespace h3s

extern "C" {

size_t h3s_column_stats_scratch_bytes(int heads) {
  return static_cast<size_t>(heads) * H3S_HEAD_DIM * (sizeof(double) + sizeof(unsigned int));
}

int h3s_column_stats(const void *k, int64_t k_stride_h, int64_t k_stride_s, const void *v,
                     int64_t v_stride_h, int64_t v_stride_s, int dtype, int heads, int sequence,
                     float v_bound, float *k_mean, float *v_scale, void *scratch,
                     h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(heads > 0 && sequence > 0, "column_stats: empty problem (heads=%d sequence=%d)", heads, sequence);
  H3S_CHECK_ARG(k != nullptr || v != nullptr, "column_stats: both inputs are NULL");
  H3S_CHECK_ARG(scratch != nullptr && (reinterpret_cast<uintptr_t>(scratch) & 7) == 0,
                "column_stats: scratch must be non-NULL and 8-byte aligned");
  H3S_CHECK_ARG(k == nullptr || k_mean != nullptr, "column_stats: k given without k_mean");
  H3S_CHECK_ARG(v == nullptr || (v_scale != nullptr && v_bound > 0.f), "column_stats: v given without v_scale/bound");
  if (k != nullptr) { int rc = check_view(k, dtype, k_stride_h, k_stride_s, "column_stats k"); if (rc) return rc; }
  if (v != nullptr) { int rc = check_view(v, dtype, v_stride_h, v_stride_s, "column_stats v"); if (rc) return rc; }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case H3S_F32: return launch_column_stats<float>(k, k_stride_h, k_stride_s, v, v_stride_h, v_stride_s, heads, sequence, v_bound, k_mean, v_scale, scratch, s);
    case H3S_BF16: return launch_column_stats<__nv_bfloat16>(k, k_stride_h, k_stride_s, v, v_stride_h, v_stride_s, heads, sequence, v_bound, k_mean, v_scale, scratch, s);
    default: return launch_column_stats<__half>(k, k_stride_h, k_stride_s, v, v_stride_h, v_stride_s, heads, sequence, v_bound, k_mean, v_scale, scratch, s);
  }
}

size_t h3s_prepare_layer_counter_bytes(int heads) { return (static_cast<size_t>(heads) + 1) * sizeof(unsigned int); }

int h3s_prepare_layer(const h3s_layer_carriers *c, const void *q, const void *k, const void *v, const int64_t *strides, int dtype,
                      int heads, int sequence, int smooth_k, float v_bound, void *counters, int32_t *status,
                      int32_t *host_mirror, h3s_stream_t stream) {
  return h3s_prepare_layer_flags(c, q, k, v, strides, dtype, heads, sequence, smooth_k, v_bound, 0, counters, status, host_mirror, stream);
}

int h3s_prepare_layer_flags(const h3s_layer_carriers *c, const void *q, const void *k, const void *v, const int64_t *strides, int dtype,
                            int heads, int sequence, int smooth_k, float v_bound, int flags, void *counters, int32_t *status,
                            int32_t *host_mirror, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(c != nullptr && strides != nullptr && counters != nullptr, "prepare_layer: NULL argument");
  H3S_CHECK_ARG(q != nullptr && k != nullptr && v != nullptr, "prepare_layer: NULL input");
  H3S_CHECK_ARG(heads > 0 && sequence > 0 && v_bound > 0.f, "prepare_layer: empty problem (heads=%d sequence=%d)", heads, sequence);
  H3S_CHECK_ARG(c->q8 && c->q_scale && c->k8 && c->k_scale && c->v8 && c->v_scale && c->scratch && (!smooth_k || c->k_mean), "prepare_layer: NULL output");
  H3S_CHECK_ARG((c->q_summary != nullptr) == (c->k_summary != nullptr) &&
                (c->q_summary == nullptr || (c->summary_dtype >= H3S_F32 && c->summary_dtype <= H3S_F64)), "prepare_layer: bad tile means");
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(c->q8) | reinterpret_cast<uintptr_t>(c->k8) | reinterpret_cast<uintptr_t>(c->scratch)) & 7) == 0 &&
                ((reinterpret_cast<uintptr_t>(c->v8) | reinterpret_cast<uintptr_t>(c->v16)) & 15) == 0, "prepare_layer: misaligned buffers");
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(counters) & 3) == 0, "prepare_layer: misaligned counters");
  { int rc = check_view(q, dtype, strides[0], strides[1], "prepare_layer q"); if (rc) return rc; }
  { int rc = check_view(k, dtype, strides[2], strides[3], "prepare_layer k"); if (rc) return rc; }
  { int rc = check_view(v, dtype, strides[4], strides[5], "prepare_layer v"); if (rc) return rc; }
  CarrierParams p;
  p.q = q; p.k = k; p.v = v;
  p.q_stride_h = strides[0]; p.q_stride_s = strides[1]; p.k_stride_h = strides[2]; p.k_stride_s = strides[3];
  p.v_stride_h = strides[4]; p.v_stride_s = strides[5];
  p.q8 = c->q8; p.k8 = c->k8; p.v8 = c->v8; p.v16 = static_cast<uint16_t *>(c->v16);
  p.q_scale = c->q_scale; p.k_scale = c->k_scale; p.v_scale = c->v_scale; p.k_mean = c->k_mean;
  p.q_summary = c->q_summary; p.k_summary = c->k_summary; p.summary_dtype = c->summary_dtype;
  p.heads = heads; p.sequence = sequence; p.padded = ceil_div(sequence, kVTile) * kVTile; p.v_bound = v_bound;
  p.k_sum = static_cast<double *>(c->scratch);
  p.v_amax_bits = reinterpret_cast<unsigned int *>(p.k_sum + heads * H3S_HEAD_DIM);
  p.next = static_cast<unsigned int *>(counters); p.stats_done = p.next + 1;
  p.status = status; p.status_mirror = host_mirror; p.wait_budget_ns = wait_budget_ns();
  p.missing = (flags & H3S_PREPARE_TEST_MISSING_STATISTICS) != 0;
  p.steps = ceil_div(sequence, kCarrierRows);
  p.q_jobs = p.k_jobs = p.v_jobs = p.steps;
  p.stats_rows = carrier_stats_rows(heads, sequence, smooth_k != 0);
  p.v_stats = ceil_div(sequence, p.stats_rows);
  p.k_stats = smooth_k ? p.v_stats : 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int words = static_cast<int>(h3s_column_stats_scratch_bytes(heads) / sizeof(unsigned int)), clears = ceil_div(words + heads + 1, 1024);
  H3S_CHECK_CUDA(launch_next(clear_words_kernel, clears < 64 ? clears : 64, 256, 0, s, reinterpret_cast<unsigned int *>(c->scratch), words,
                             p.next, heads + 1));
  switch (dtype) {
    case H3S_F32: return launch_layer_carriers<float>(p, smooth_k != 0, s);
    case H3S_BF16: return launch_layer_carriers<__nv_bfloat16>(p, smooth_k != 0, s);
    default: return launch_layer_carriers<__half>(p, smooth_k != 0, s);
  }
}

int h3s_quant_rows_fp8(const void *x_bf16, int64_t x_stride_row, int rows, int channels, uint8_t *out,
                       float *row_scale, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(x_bf16 != nullptr && out != nullptr && row_scale != nullptr, "quant_rows_fp8: NULL pointer");
  H3S_CHECK_ARG(rows > 0 && channels > 0 && channels % 8 == 0 && channels <= kRowQuantThreads * 8 * kRowQuantMaxChunks,
                "quant_rows_fp8: channels %d must be a multiple of 8 and at most %d", channels,
                kRowQuantThreads * 8 * kRowQuantMaxChunks);
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(x_bf16) & 15) == 0 && x_stride_row % 8 == 0 && x_stride_row >= channels,
                "quant_rows_fp8: input must be 16-byte aligned with a row stride that is a multiple of 8");
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(out) & 7) == 0, "quant_rows_fp8: output must be 8-byte aligned");
  const __nv_bfloat16 *bf16 = static_cast<const __nv_bfloat16 *>(x_bf16);
#define H3S_LAUNCH_ROWS(CHUNKS)                                                                                  \
  H3S_CHECK_CUDA(launch_next(quant_rows_fp8_warp_kernel<CHUNKS>, ceil_div(rows, kRowWarps), kRowWarps * 32, 0, \
                             static_cast<cudaStream_t>(stream), bf16, x_stride_row, rows, channels, out, row_scale))
  if (channels <= 4096) {
    if (channels <= 1024) H3S_LAUNCH_ROWS(4); else if (channels <= 2048) H3S_LAUNCH_ROWS(8);
    else if (channels <= 3072) H3S_LAUNCH_ROWS(12); else H3S_LAUNCH_ROWS(16);
    return H3S_OK;
  }
#undef H3S_LAUNCH_ROWS
  const int grid = rows < 148 * 8 ? rows : 148 * 8;
  H3S_CHECK_CUDA(launch_next(quant_rows_fp8_kernel, grid, kRowQuantThreads, 0, static_cast<cudaStream_t>(stream), bf16, x_stride_row,
                             rows, channels, out, row_scale));
  return H3S_OK;
}

int h3s_column_stats_finalize(const void *stats, int dtype, int heads, int sequence, float v_bound,
                              float *k_mean, float *v_scale, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(stats != nullptr && (reinterpret_cast<uintptr_t>(stats) & 7) == 0, "column_stats_finalize: stats must be non-NULL and 8-byte aligned");
  H3S_CHECK_ARG(heads > 0 && sequence > 0, "column_stats_finalize: empty problem");
  H3S_CHECK_ARG(k_mean != nullptr || v_scale != nullptr, "column_stats_finalize: nothing to produce");
  H3S_CHECK_ARG(v_scale == nullptr || v_bound > 0.f, "column_stats_finalize: v_bound must be positive");
  H3S_CHECK_ARG(dtype == H3S_F32 || dtype == H3S_BF16 || dtype == H3S_F16, "column_stats_finalize: unsupported dtype %d", dtype);
  const double *k_sum = static_cast<const double *>(stats);
  const unsigned int *v_bits = reinterpret_cast<const unsigned int *>(k_sum + heads * H3S_HEAD_DIM);
  const int total = heads * H3S_HEAD_DIM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case H3S_F32: H3S_CHECK_CUDA(launch_next(column_stats_finalize_kernel<float>, ceil_div(total, 256), 256, 0, s, k_sum, v_bits, total, sequence, v_bound, k_mean, v_scale)); break;
    case H3S_BF16: H3S_CHECK_CUDA(launch_next(column_stats_finalize_kernel<__nv_bfloat16>, ceil_div(total, 256), 256, 0, s, k_sum, v_bits, total, sequence, v_bound, k_mean, v_scale)); break;
    default: H3S_CHECK_CUDA(launch_next(column_stats_finalize_kernel<__half>, ceil_div(total, 256), 256, 0, s, k_sum, v_bits, total, sequence, v_bound, k_mean, v_scale)); break;
  }
  return H3S_OK;
}

int h3s_quant_qk_blocks(const void *x, int dtype, int64_t x_stride_h, int64_t x_stride_s,
                        const float *mean, int8_t *out, float *scale, void *summary,
                        int summary_dtype, int heads, int rows, int row_start, int sequence_total,
                        int block, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(block == H3S_Q_TILE || block == H3S_KV_TILE, "quant_qk_blocks: block must be 128 or 64, got %d", block);
  H3S_CHECK_ARG(heads > 0 && rows > 0 && sequence_total > 0, "quant_qk_blocks: empty problem");
  H3S_CHECK_ARG(row_start >= 0 && row_start % block == 0, "quant_qk_blocks: row_start %d is not a multiple of the block %d", row_start, block);
  H3S_CHECK_ARG(row_start + rows <= sequence_total, "quant_qk_blocks: chunk [%d,%d) exceeds sequence %d", row_start, row_start + rows, sequence_total);
  H3S_CHECK_ARG(rows % block == 0 || row_start + rows == sequence_total,
                "quant_qk_blocks: only the final chunk may contain a partial tile");
  H3S_CHECK_ARG(x != nullptr, "quant_qk_blocks: NULL input");
  H3S_CHECK_ARG((out != nullptr) == (scale != nullptr), "quant_qk_blocks: out and scale must be given together");
  H3S_CHECK_ARG(out != nullptr || summary != nullptr, "quant_qk_blocks: nothing to produce");
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(out) & 7) == 0, "quant_qk_blocks: out must be 8-byte aligned");
  H3S_CHECK_ARG(summary == nullptr || (summary_dtype >= H3S_F32 && summary_dtype <= H3S_F64),
                "quant_qk_blocks: bad summary dtype %d", summary_dtype);
  { int rc = check_view(x, dtype, x_stride_h, x_stride_s, "quant_qk_blocks x"); if (rc) return rc; }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case H3S_F32: return launch_quant_qk<float>(x, x_stride_h, x_stride_s, mean, out, scale, summary, summary_dtype, heads, rows, row_start, sequence_total, block, s);
    case H3S_BF16: return launch_quant_qk<__nv_bfloat16>(x, x_stride_h, x_stride_s, mean, out, scale, summary, summary_dtype, heads, rows, row_start, sequence_total, block, s);
    default: return launch_quant_qk<__half>(x, x_stride_h, x_stride_s, mean, out, scale, summary, summary_dtype, heads, rows, row_start, sequence_total, block, s);
  }
}

int h3s_quant_v_fp8(const void *v, int dtype, int64_t v_stride_h, int64_t v_stride_s,
                    const float *v_scale, uint8_t *out, int heads, int rows, int row_start,
                    int sequence_total, float v_bound, h3s_stream_t stream) {
  return h3s_quant_v_fp8_half(v, dtype, v_stride_h, v_stride_s, v_scale, out, nullptr, heads, rows, row_start,
                              sequence_total, v_bound, stream);
}

int h3s_quant_v_fp8_half(const void *v, int dtype, int64_t v_stride_h, int64_t v_stride_s, const float *v_scale,
                         uint8_t *out, void *out_half, int heads, int rows, int row_start, int sequence_total,
                         float v_bound, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(heads > 0 && rows > 0 && sequence_total > 0, "quant_v_fp8: empty problem");
  H3S_CHECK_ARG(row_start >= 0 && row_start % 128 == 0, "quant_v_fp8: row_start %d must be 128 aligned", row_start);
  H3S_CHECK_ARG(row_start + rows <= sequence_total, "quant_v_fp8: chunk exceeds sequence");
  H3S_CHECK_ARG(rows % 128 == 0 || row_start + rows == sequence_total,
                "quant_v_fp8: only the final chunk may contain a partial tile");
  H3S_CHECK_ARG(v != nullptr && v_scale != nullptr && out != nullptr, "quant_v_fp8: NULL pointer");
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(out_half)) & 15) == 0, "quant_v_fp8: outputs must be 16-byte aligned");
  uint16_t *half = static_cast<uint16_t *>(out_half);
  H3S_CHECK_ARG(v_bound > 0.f, "quant_v_fp8: v_bound must be positive");
  { int rc = check_view(v, dtype, v_stride_h, v_stride_s, "quant_v_fp8 v"); if (rc) return rc; }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case H3S_F32: return launch_quant_v<float>(v, v_stride_h, v_stride_s, v_scale, out, half, heads, rows, row_start, sequence_total, v_bound, s);
    case H3S_BF16: return launch_quant_v<__nv_bfloat16>(v, v_stride_h, v_stride_s, v_scale, out, half, heads, rows, row_start, sequence_total, v_bound, s);
    default: return launch_quant_v<__half>(v, v_stride_h, v_stride_s, v_scale, out, half, heads, rows, row_start, sequence_total, v_bound, s);
  }
}


int h3s_column_stats_static(const void *k, int64_t k_stride_h, int64_t k_stride_s, const void *v,
                            int64_t v_stride_h, int64_t v_stride_s, int dtype, int heads, int sequence,
                            float v_bound, float *k_mean, float *v_scale, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(heads > 0 && sequence > 0, "column_stats_static: empty problem (heads=%d sequence=%d)", heads, sequence);
  H3S_CHECK_ARG(heads <= kStaticStatsMaxHeads,
                "column_stats_static: %d heads exceed the %d the built-in scratch holds; use h3s_column_stats "
                "with a caller-provided scratch buffer instead", heads, kStaticStatsMaxHeads);
  H3S_CHECK_ARG(k != nullptr || v != nullptr, "column_stats_static: both inputs are NULL");
  H3S_CHECK_ARG(k == nullptr || k_mean != nullptr, "column_stats_static: k given without k_mean");
  H3S_CHECK_ARG(v == nullptr || (v_scale != nullptr && v_bound > 0.f), "column_stats_static: v given without v_scale/bound");
  if (k != nullptr) { int rc = check_view(k, dtype, k_stride_h, k_stride_s, "column_stats_static k"); if (rc) return rc; }
  if (v != nullptr) { int rc = check_view(v, dtype, v_stride_h, v_stride_s, "column_stats_static v"); if (rc) return rc; }
  void *scratch = nullptr;
  { int rc = static_stats_scratch(&scratch); if (rc) return rc; }
  // launch_column_stats clears the part of the scratch it uses (a memset on the
  // stream, not an allocation) before the accumulating kernel runs
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case H3S_F32: return launch_column_stats<float>(k, k_stride_h, k_stride_s, v, v_stride_h, v_stride_s, heads, sequence, v_bound, k_mean, v_scale, scratch, s);
    case H3S_BF16: return launch_column_stats<__nv_bfloat16>(k, k_stride_h, k_stride_s, v, v_stride_h, v_stride_s, heads, sequence, v_bound, k_mean, v_scale, scratch, s);
    default: return launch_column_stats<__half>(k, k_stride_h, k_stride_s, v, v_stride_h, v_stride_s, heads, sequence, v_bound, k_mean, v_scale, scratch, s);
  }
}

}  // extern "C"
