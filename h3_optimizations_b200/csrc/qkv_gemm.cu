// Chunked ConvRot INT8 QKV projection for sm_100a.
//
//   convrot_quant_rows : x (rows, hidden) bf16 -> Hadamard-256 on every
//                        256-channel group (fast Walsh-Hadamard in registers
//                        across one pass through shared memory), per-row INT8
//                        (scale = amax/127).  HBM-bound, one warp per row.
//   qkv_gemm_chunk     : persistent warp-specialised tcgen05 GEMM
//                        acc[rows, n] = x_i8 . w_i8^T (kind::i8, int32 in TMEM),
//                        256x256 tiles on a pair of SMs (cta_group::2), K step 128
//                        bytes (SWIZZLE_128B), TMA ring, two TMEM accumulators so
//                        the epilogue of one tile overlaps the MMAs of the next.
//                        The epilogue
//                        de-quantises (acc * (x_scale[row] * w_scale[col])), rounds
//                        to bf16 and scatters into head-major (3*H, rows, 128)
//                        staging that the carrier kernels consume.
//   qkv_gemm_chunk_carriers : the same GEMM whose epilogue emits the carriers
//                        themselves: INT8 Q blocks with scale and tile mean
//                        (a 128-row Q block of one head is one accumulator
//                        tile half), INT8 K half-blocks when K is not smoothed;
//                        K (when smoothed) and V, which need whole-sequence
//                        statistics, are staged as bf16 while their column sums
//                        / maxima are accumulated for the short second phase.
#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "ptx.cuh"
#include "tma.cuh"

namespace h3s {

// ---------------------------------------------------------------------------
// ConvRot prologue
// ---------------------------------------------------------------------------

constexpr int kRotGroup = 256;

// The stages of a Walsh-Hadamard transform behind the first, on pairs of neighbouring values; a - b as the exactly rounded a + (-1) * b
template <int kPairs>
__device__ __forceinline__ void fwht_pairs(float2 (&v)[kPairs]) {
#pragma unroll
  for (int stride = 1; stride < kPairs; stride <<= 1) {
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      if ((i & stride) == 0) {
        const float2 a = v[i], b = v[i + stride];
        v[i] = add2(a, b);
        v[i + stride] = fma2(b, make_float2(-1.f, -1.f), a);
      }
    }
  }
}

// The larger magnitude, with some sign; a NaN stays one
__device__ __forceinline__ float larger_magnitude(float a, float b) {
  float d;
  asm("max.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// One warp per row.  The three low index bits are transformed as loaded (8 channels a lane);
// the row then crosses shared memory once, so that a lane holds the 32 values that share
// their low bits and the five remaining stages are additions of its own registers.  With
// those stages as warp shuffles (40 per 8 channels) and a row spread over all warps of a CTA
// (two barriers a row), 4096 rows of 3072 channels took 24.5 us and 21.4 so.  Instructions bound it then, two for each that
// the transform needs: with packed additions, the integer taken from the low bits of a shifted quotient, and NaN looked for once a
// row instead of a clamp for each code, 15.1 -> 13.0 us behind one another (2.9 TB/s; 2304 rows 9.0 -> 8.0, 900 rows 8.1 -> 7.1).
// What is left is sixteen warps an SM, as many as shared memory has rows for, that wait for their loads.
// Shared memory of a warp: [32 upper indices][8 * groups + 4 floats]; the padding puts
// the 16-byte stores of eight lanes into different banks.
constexpr int kRotWarps = 4;  // rows (warps) per CTA, at most

__host__ __device__ constexpr int rot_stride(int groups) { return 8 * groups + 4; }

template <int kAhead>  // 16-byte loads of a lane in flight
__global__ void __launch_bounds__(kRotWarps * 32)
convrot_quant_rows_kernel(const __nv_bfloat16 *__restrict__ x, int64_t x_stride, int rows, int hidden,
                          int8_t *__restrict__ out, float *__restrict__ scale_out, uint32_t *__restrict__ clear, int words) {
  extern __shared__ __align__(16) float rot_smem[];
  let_next_start();
  wait_for_previous();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) clear[i] = 0u;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = hidden / kRotGroup, stride = rot_stride(groups);
  float *mine = rot_smem + warp * 32 * stride;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;  // warps of a CTA do not meet
  const __nv_bfloat16 *src = x + row * x_stride + lane * 8;
  for (int g0 = 0; g0 < groups; g0 += kAhead) {
    Elem<__nv_bfloat16>::Raw raw[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      raw[i] = g0 + i < groups ? Elem<__nv_bfloat16>::load_raw(src + (g0 + i) * kRotGroup) : Elem<__nv_bfloat16>::zero_raw();
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (g0 + i < groups) {
        float x[8];
        Elem<__nv_bfloat16>::unpack(raw[i], x);
        float2 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = make_float2(__fadd_rn(x[2 * k], x[2 * k + 1]), __fsub_rn(x[2 * k], x[2 * k + 1]));
        fwht_pairs(v);
        float4 *dst = reinterpret_cast<float4 *>(mine + lane * stride + (g0 + i) * 8);
        dst[0] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
        dst[1] = make_float4(v[2].x, v[2].y, v[3].x, v[3].y);
      }
    }
  }
  __syncwarp();
  float amax = 0.f;
  for (int c = lane; c < 8 * groups; c += 32) {  // (group, low bits)
    float2 v[16];  // two upper indices at a time
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float a = mine[(2 * i) * stride + c], b = mine[(2 * i + 1) * stride + c];
      v[i] = make_float2(__fadd_rn(a, b), __fsub_rn(a, b));
    }
    fwht_pairs(v);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      v[i] = mul2(v[i], make_float2(0.0625f, 0.0625f));  // 1/sqrt(256), exact
      amax = larger_magnitude(larger_magnitude(amax, v[i].x), v[i].y);
      mine[(2 * i) * stride + c] = v[i].x;
      mine[(2 * i + 1) * stride + c] = v[i].y;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = larger_magnitude(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  amax = fabsf(amax);
  __syncwarp();
  const bool some_nan = amax != amax;
  if (some_nan) {  // it counts as nothing
    amax = 0.f;
    for (int c = lane; c < 8 * groups; c += 32)
      for (int l = 0; l < 32; ++l) amax = fmaxf(amax, fabsf(mine[l * stride + c]));
    amax = warp_max(amax);
  }
  const float scale = amax > 0.f ? __fdiv_rn(amax, 127.0f) : 1.0f;
  if (lane == 0) scale_out[row] = scale;
  const SharedDivisor by_scale = make_divisor(scale);  // exact v/scale without a divide per element
  int8_t *dst = out + static_cast<int64_t>(row) * hidden + lane * 8;
  auto emit = [&](auto exact_tag) {
    constexpr bool kExact = decltype(exact_tag)::value;
#pragma unroll 2
    for (int g = 0; g < groups; ++g) {
      const float4 *at = reinterpret_cast<const float4 *>(mine + lane * stride + g * 8);
      const float4 lo = at[0], hi = at[1];
      const float2 v[4] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y), make_float2(hi.z, hi.w)};
      uint32_t code[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 q = divide2<kExact>(by_scale, v[i]);
        if (kExact) {  // |q| <= 127.0001: the nearest integer is in the low bits of q + 1.5 * 2^23
          const float2 shifted = add2(q, make_float2(12582912.0f, 12582912.0f));
          code[2 * i] = __float_as_uint(shifted.x);
          code[2 * i + 1] = __float_as_uint(shifted.y);
        } else {
          code[2 * i] = static_cast<uint32_t>(max(-127, min(127, __float2int_rn(q.x))));
          code[2 * i + 1] = static_cast<uint32_t>(max(-127, min(127, __float2int_rn(q.y))));
        }
      }
      uint32_t packed[2];
#pragma unroll
      for (int w = 0; w < 2; ++w)
        packed[w] = __byte_perm(__byte_perm(code[4 * w], code[4 * w + 1], 0x0040),
                                __byte_perm(code[4 * w + 2], code[4 * w + 3], 0x0040), 0x5410);
      *reinterpret_cast<uint2 *>(dst + g * kRotGroup) = make_uint2(packed[0], packed[1]);
    }
  };
  if (by_scale.exact && !some_nan) emit(std::true_type{}); else emit(std::false_type{});
}

// ---------------------------------------------------------------------------
// INT8 GEMM
// ---------------------------------------------------------------------------

// One tile is 256 x 256, computed by a cluster of two CTAs on neighbouring SMs: each CTA
// holds the accumulators of its own 128 rows x 256 columns, loads its 128 rows of A and
// HALF of B's 256 rows, and the first CTA issues the MMAs of both (cta_group::2).  A
// 128x256 tile per SM pulled 48 KB through L2 for every 512 cycles of MMA work, 96 bytes
// a clock and SM, which is more than L2 delivers to all SMs at once; the pair needs 64,
// and the smaller stages leave room for one more.  MLP of 33272 x 3072 x 12288: 3.59 ->
// 3.02 ms (with the GELU below), of 1000 tokens 147 -> 119 us; attention block of 33272
// tokens 6.09 -> 5.90 ms; 2.74 ms, 108 us and 5.5 ms with the epilogues and quantisers as they
// are now.  A single row tile wastes half a pair, but what such a call waits for is the
// weights, which are read once either way.
constexpr int kGemmM = 128, kGemmN = 256, kGemmK = 128;  // per CTA; K in bytes == int8 elements
constexpr int kGemmPairM = 2 * kGemmM;
// Row pairs visited before the next column of tiles: 4096 rows of A (12 to 50 MB) and the
// weights stay in L2 while every column passes over them.
constexpr int kGemmGroupM = 16;
// A warp may only touch the TMEM lanes 32*(warp%4)...  Staging and dense: warps 0-3 epilogue of
// the tile's first 128 columns, 4 TMA, 5 MMA, 6-7 idle, 8-11 epilogue of the second 128.
// Carriers: warps 0-15 epilogue (four per lane quarter, two per 128 columns, each thread half a row), 16 TMA,
// 17 MMA: with eight warps, one row a thread, 168 registers and half the warps to hide latencies behind,
// the projection of 33272 rows with norm and rotation took 1.63 ms, 1.52 with sixteen.
template <int kMode>
struct GemmWarps {
  static constexpr bool kMany = kMode == 1;  // kModeCarriers
  static constexpr int kEpilogue = kMany ? 16 : 8;
  static constexpr int kLoad = kMany ? 16 : 4, kIssue = kLoad + 1;
  static constexpr int kThreads = kMany ? 18 * 32 : 384;
  static __device__ __forceinline__ bool epilogue(int warp) { return kMany ? warp < 16 : warp < 4 || warp >= 8; }
};
constexpr uint32_t kGemmABytes = kGemmM * kGemmK;  // 16384
constexpr uint32_t kGemmBBytes = kGemmN / 2 * kGemmK;  // 16384: this CTA's half
constexpr uint32_t kGemmTmemCols = 512;

// A sum as an unevaluated triple of floats: `sum`, what rounding has taken from it, and what rounding has taken from
// that.  Of n floats it is off by about n^2 * 2^-72 of the largest intermediate sum, where a 64-bit sum is off by
// n * 2^-53; sums beyond the range of a float become infinite or NaN.  Against totals kept as pairs of floats (46 bits) the
// projection of 33272 x 3072 with norm and table takes 1.07 ms for 1.06; in 64 bits it was 1.14 for 1.03 without them.
struct TripleSum {
  float sum, lost, rest;
};

// What the eight warps of one 128-column half of a tile tell each other in the carrier
// epilogue: the sums of squares of a row's two shares of channels, then per-warp largest
// magnitudes and per-channel partial sums (maxima for V) of the rows 0-63 and 64-127 of the tile.
struct EpilogueExchange {
  TripleSum squares[2][kGemmM];      // [channel share][row]
  float amax[2][8];                  // [row half][warp]
  float column[2][8][H3S_HEAD_DIM];  // [row half][warp][channel]
};
constexpr uint32_t kEpilogueTileBytes = kGemmM * H3S_HEAD_DIM * 2;  // one half tile as bf16: 32 KB

// Shared-memory layout.  The carrier epilogue stages each half tile as bf16 so
// that it can be re-read column-wise (quantisation, statistics and every global
// store then run on contiguous lines); it pays for the two 32 KB staging tiles
// with stages of the operand ring.
// Epilogue of the GEMM kernel
enum GemmMode {
  kModeStaging = 0,   // INT8 x INT8 -> bf16 head-major staging (h3s_qkv_gemm_chunk[_norm_rope])
  kModeCarriers = 1,  // INT8 x INT8 -> carriers (h3s_qkv_gemm_chunk_carriers)
  kModeDense = 2,     // any operand kind -> scaled, biased, activated bf16 row-major matrix (h3s_dense_gemm)
};

static_assert(kModeCarriers == 1, "GemmWarps");

template <int kMode>
struct GemmLayout {
  static constexpr bool kCarriers = kMode != kModeStaging;  // both stage half tiles for coalesced stores
  static constexpr int kStages = kMode == kModeStaging ? 6 : kMode == kModeDense ? 5 : 4;
  static constexpr uint32_t kOffB = kStages * kGemmABytes;
  static constexpr uint32_t kOffTile = kOffB + kStages * kGemmBBytes;
  static constexpr uint32_t kOffExchange = kOffTile + (kCarriers ? 2 * kEpilogueTileBytes : 0);
  static constexpr uint32_t kOffNorm = kOffExchange + (kMode == kModeCarriers ? 2 * sizeof(EpilogueExchange) : 0);  // weights of Q, of K
  static constexpr uint32_t kOffScale = kOffNorm + (kMode == kModeCarriers ? 2 * H3S_HEAD_DIM * sizeof(float) : 0);  // a warp's 64 column scales
  static constexpr uint32_t kOffBar = kOffScale + (kMode == kModeCarriers ? 16 * 64 * sizeof(float) : 0);
  static constexpr uint32_t kBytes = kOffBar + 256 + 1024;
  static_assert(sizeof(uint64_t) * (2 * 6 + 16) + 8 <= 256, "barriers");
  static_assert(kBytes <= 227 * 1024, "GEMM shared memory exceeds the per-CTA limit");
};
constexpr int kGemmMaxStages = 6;

enum GemmAbort { kGemmAbortFull = 21, kGemmAbortEmpty, kGemmAbortAccFull, kGemmAbortAccEmpty, kGemmAbortTile, kGemmAbortExchange, kGemmAbortSquares };

struct GemmShared {
  uint64_t full[kGemmMaxStages];   // first CTA's: the stage's four loads, two by each CTA
  uint64_t empty[kGemmMaxStages];  // both CTAs': the pair's MMAs have read the stage
  uint64_t acc_full[2];            // both CTAs'
  uint64_t acc_empty[2];           // first CTA's: the epilogue warps of both
  uint64_t tile_ready[2];      // per tile half: its warps have staged their rows
  uint64_t exchange_ready[2];  // per tile half: its warps have written their EpilogueExchange
  uint64_t squares_ready[2][4];  // per tile half and lane quarter: its two warps have written their sums of squares
  uint32_t tmem_base;
  int abort_word;
};

struct GemmParams {
  const float *x_scale;   // (rows)
  const float *w_scale;   // (n_out)
  __nv_bfloat16 *out;     // (n_out/128, out_rows_stride/128.., 128): head-major staging
  int64_t out_stride_head;  // elements between consecutive 128-column groups
  int32_t *status;
  int rows, n_out, hidden;
  int m_pairs, n_tiles;  // pairs of 128-row tiles, tiles of tile_n columns
  // Column tiles are visited in the order of the weight rows, [Q | K | V]: the tiles that are
  // dearer in the epilogue (norm, rotation, quantisation) are dealt out first, the cheap
  // V tiles even out what is left.  Alternating between the kinds, as suits a kernel that is
  // bound by its MMAs, left some pairs of SMs with seven dear tiles and others with four
  // (4096 rows with norm and rotation, together with the spills below: 174 -> 159 us).
  // optional per-head RMS norm (+ split-half rotation) of the Q and K groups
  const float *q_norm;    // (128) or null: no norm, no rotation
  const float *k_norm;    // (128)
  int norm_dtype;         // carriers: type of both, which the epilogue reads from shared memory; else fp32
  const void *rope;       // (rows, 48, 2, 2) view with the strides below, or null
  int64_t rope_stride_seq, rope_stride_dim, rope_stride_rot, rope_stride_pair;
  int rope_dtype;         // H3S_F32 or H3S_BF16
  int heads;
  float epsilon;
  unsigned long long wait_budget_ns;  // bound of every mbarrier wait
  // carrier epilogue (h3s_qkv_gemm_chunk_carriers); all tensors cover the whole sequence
  int8_t *q8, *k8;                 // (heads, sequence_total, 128); k8 null: K is staged
  float *q_scale, *k_scale;        // (heads, ceil(S/128)), (heads, ceil(S/64))
  void *q_summary, *k_summary;     // (heads, blocks, 128) tile means, summary_dtype
  __nv_bfloat16 *k_stage, *v_stage;  // (heads, sequence_total, 128)
  double *k_sum;                   // (heads, 128) running column sums of K, or null
  unsigned int *v_amax_bits;       // (heads, 128) running column maxima of |V| as float bits
  int summary_dtype, sequence_total, row_start;
  // dense epilogue (h3s_dense_gemm): out[m, n] = act(acc * row_scale[m] * col_scale[n] + bias[n]) as bf16
  int operand_kind;                // H3S_GEMM_I8 / BF16 / F16 / E4M3
  const float *row_scale;          // (rows) or null
  const float *col_scale;          // (n_out) or null
  const float *bias;               // (n_out) or null
  int activation;                  // H3S_ACT_NONE / H3S_ACT_GELU_TANH
  int tile_n;                      // columns of a tile: kGemmN or less, a multiple of 32
  bool vector_columns;             // col_scale and bias, where given, are 16-byte aligned
  __nv_bfloat16 *dense_out;        // (rows, ldc)
  int64_t ldc;
};

// 0.5 x (1 + tanh(u)), u = sqrt(2/pi) (x + 0.044715 x^3), the formula of torch's approximate='tanh', as
// x / (1 + exp(-2u)): nothing cancels for negative x, where 1 + tanh(u) loses all but a few bits.  Two values at a time:
// everything but the exponentials and the reciprocals is packed (MLP of 33272 x 3072 x 12288, under the power cap, 2605 -> 2595 us).
// 28 of 8.4 million bf16 results differ from the unpacked form's, errors against 64 bits are the same to seven digits.
__device__ __forceinline__ float2 gelu_tanh2(float2 x) {
  constexpr float kLinear = -2.0f * 0.7978845608028654f * 1.4426950408889634f, kCubic = kLinear * 0.044715f;
  const float2 t = mul2(x, fma2(mul2(x, x), make_float2(kCubic, kCubic), make_float2(kLinear, kLinear)));
  float2 e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
  e = add2(e, make_float2(1.0f, 1.0f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(e.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(e.y));
  return mul2(x, r);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 t = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&t);
}

// 32 accumulators of one row -> 16 bf16 pairs.  What is applied is fixed at compile time:
// tests inside the element loop cut it into one dependent chain per element (fc1 of the
// MLP with GELU, 4096 x 3072 x 12288: 157 -> 127 us).  `col` is a multiple of 32; columns
// past n_out (a multiple of 8) repeat the last four, nothing of them is stored.
template <bool kScale, bool kBias, bool kGelu>
__device__ __forceinline__ void dense_row32(const uint32_t (&acc)[32], float row_scale, const float *__restrict__ col_scale,
                                            const float *__restrict__ bias, int col, int n_out, uint32_t (&y)[16]) {
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    const int at = min(col + i, n_out - 4);
    float4 cs = make_float4(1.0f, 1.0f, 1.0f, 1.0f), shift = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kScale) cs = __ldg(reinterpret_cast<const float4 *>(col_scale + at));
    if (kBias) shift = __ldg(reinterpret_cast<const float4 *>(bias + at));
    const float c[4] = {cs.x, cs.y, cs.z, cs.w}, b[4] = {shift.x, shift.y, shift.z, shift.w};
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      float2 value = mul2(make_float2(__uint_as_float(acc[i + e]), __uint_as_float(acc[i + e + 1])),
                          mul2(make_float2(row_scale, row_scale), make_float2(c[e], c[e + 1])));
      if (kBias) value = add2(value, make_float2(b[e], b[e + 1]));
      if (kGelu) value = gelu_tanh2(value);
      y[(i + e) >> 1] = pack_bf16x2(value.x, value.y);
    }
  }
}

// Four consecutive floats of a per-column vector; n_out is a multiple of 8, so a group of
// four lies inside or outside as a whole
__device__ __forceinline__ float4 column4(const float *base, int col, int n_out, float otherwise) {
  if (base == nullptr || col >= n_out) return make_float4(otherwise, otherwise, otherwise, otherwise);
  return make_float4(__ldg(base + col), __ldg(base + col + 1), __ldg(base + col + 2), __ldg(base + col + 3));
}

__device__ __forceinline__ float rope_load(const void *base, int64_t index, int dtype) {
  return dtype == H3S_F32 ? load_written(static_cast<const float *>(base) + index)
                          : __bfloat162float(load_written(static_cast<const __nv_bfloat16 *>(base) + index));
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ void store_summary(void *base, int dtype, int64_t at, double value) {
  switch (dtype) {
    case H3S_F64: static_cast<double *>(base)[at] = value; break;
    case H3S_F32: static_cast<float *>(base)[at] = static_cast<float>(value); break;
    case H3S_BF16: static_cast<__nv_bfloat16 *>(base)[at] = __float2bfloat16_rn(static_cast<float>(value)); break;
    default: static_cast<__half *>(base)[at] = __float2half_rn(static_cast<float>(value)); break;
  }
}

// INT8 codes of eight consecutive channels held as four bf16 pairs:
// code = trunc(v/scale +- 0.5) with the correctly rounded quotient (the arithmetic
// of quant_qk_blocks_kernel), written as one 8-byte store.
template <bool kExact>
__device__ __forceinline__ void quantise8(const uint4 &raw, const SharedDivisor &by_scale, int8_t *dst) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t code[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) round_codes(divide2<kExact>(by_scale, bf16_pair(w[i])), code[2 * i], code[2 * i + 1]);
  uint32_t packed[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
    packed[k] = __byte_perm(__byte_perm(code[4 * k], code[4 * k + 1], 0x0040),
                            __byte_perm(code[4 * k + 2], code[4 * k + 3], 0x0040), 0x5410);
  *reinterpret_cast<uint2 *>(dst) = make_uint2(packed[0], packed[1]);
}

// One row of one Q or K head after the GEMM, held as 64 bf16 pairs (every
// intermediate of the reference epilogue is rounded to bf16, so the packed
// form loses nothing): RMS norm over the 128 channels with the per-channel
// weight, then the split-half rotation of channels [0,48) against [48,96).
// Same order of operations and roundings as the reference
// (attention/sparse/fused_qkv.py:218-289); the sum of squares is accumulated
// in FP64 so that it does not depend on the order of the additions.  The staging
// epilogue does this, a row to a thread; the carrier epilogue deals a row to two (HalfRow).
//
// The table is read 16 bytes at a time where it is stored as the model produces it; the
// form is decided once per row, so that the loads of a batch are all in flight together
// and the first batch travels while the norm is computed.  With the decision inside the
// element loop, and one chain of dependent FP64 additions, a 4096-row chunk of the QKV
// projection took 197 us for 155, when the carrier epilogue had this form.
enum RopeForm { kRopeNone, kRopeBf16, kRopeF32, kRopeStrided };

__device__ __forceinline__ void rotate_pair(uint32_t &first, uint32_t &second, const float (&f)[2][4]) {
  const float2 a = bf16_pair(first), b = bf16_pair(second);
  const float2 out_first = add2(mul2(make_float2(f[0][0], f[1][0]), a), mul2(make_float2(f[0][1], f[1][1]), b));
  const float2 out_second = add2(mul2(make_float2(f[0][2], f[1][2]), a), mul2(make_float2(f[0][3], f[1][3]), b));
  first = pack_bf16x2(out_first.x, out_first.y);
  second = pack_bf16x2(out_second.x, out_second.y);
}

__device__ __forceinline__ void norm_row(uint32_t (&y)[H3S_HEAD_DIM / 2], const float *__restrict__ norm_weight,
                                         float epsilon) {
  double part[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < H3S_HEAD_DIM / 2; ++i) {
    const double lo = static_cast<double>(bf16_lo(y[i])), hi = static_cast<double>(bf16_hi(y[i]));
    part[(2 * i) & 3] = fma(lo, lo, part[(2 * i) & 3]);
    part[(2 * i + 1) & 3] = fma(hi, hi, part[(2 * i + 1) & 3]);
  }
  const double sum = (part[0] + part[1]) + (part[2] + part[3]);
  const float mean = __fadd_rn(__fmul_rn(static_cast<float>(sum), 1.0f / H3S_HEAD_DIM), epsilon);
  const float inverse_rms = __frsqrt_rn(mean);
#pragma unroll
  for (int i = 0; i < H3S_HEAD_DIM / 2; ++i) {
    const float2 w = __ldg(reinterpret_cast<const float2 *>(norm_weight) + i);
    const float2 normed = mul2(mul2(bf16_pair(y[i]), make_float2(inverse_rms, inverse_rms)), w);
    y[i] = pack_bf16x2(normed.x, normed.y);
  }
}

// channels 2i, 2i+1 against 2i+48, 2i+49 for i in [0, 24), the eight factors of a pair in 16 (bf16) or 32 bytes
template <int kForm>
__device__ __forceinline__ void norm_rope_packed(uint32_t (&y)[H3S_HEAD_DIM / 2], const float *__restrict__ norm_weight,
                                                 float epsilon, const uint4 *__restrict__ table) {
  constexpr int kWords = kForm == kRopeBf16 ? 1 : 2;  // 16-byte words per i
  constexpr int kBatch = kForm == kRopeBf16 ? 6 : 3;  // of i: 48 registers in flight beside the row's 64
  uint4 ahead[kBatch * kWords];
#pragma unroll
  for (int k = 0; k < kBatch * kWords; ++k) ahead[k] = __ldg(table + k);
  norm_row(y, norm_weight, epsilon);
#pragma unroll
  for (int b = 0; b < 24 / kBatch; ++b) {
    uint4 now[kBatch * kWords];
#pragma unroll
    for (int k = 0; k < kBatch * kWords; ++k) {
      now[k] = ahead[k];
      if (b + 1 < 24 / kBatch) ahead[k] = __ldg(table + (b + 1) * kBatch * kWords + k);
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      float f[2][4];  // [channel][f00, f01, f10, f11]
      if (kForm == kRopeBf16) {
        const uint4 w = now[k];
        f[0][0] = bf16_lo(w.x); f[0][1] = bf16_hi(w.x); f[0][2] = bf16_lo(w.y); f[0][3] = bf16_hi(w.y);
        f[1][0] = bf16_lo(w.z); f[1][1] = bf16_hi(w.z); f[1][2] = bf16_lo(w.w); f[1][3] = bf16_hi(w.w);
      } else {
        const uint4 u = now[k * kWords], w = now[k * kWords + kWords - 1];
        f[0][0] = __uint_as_float(u.x); f[0][1] = __uint_as_float(u.y); f[0][2] = __uint_as_float(u.z); f[0][3] = __uint_as_float(u.w);
        f[1][0] = __uint_as_float(w.x); f[1][1] = __uint_as_float(w.y); f[1][2] = __uint_as_float(w.z); f[1][3] = __uint_as_float(w.w);
      }
      const int i = b * kBatch + k;
      rotate_pair(y[i], y[i + 24], f);
    }
  }
}

// Tables of any strides.  A call of its own with the row in local memory: unrolled in place,
// its addresses took registers from the common forms, which then spilled 336 bytes a thread.
// kPairs channel pairs from `pair0` on, and as many behind them that they are rotated against.
template <int kPairs>
__device__ __noinline__ void rotate_strided(uint32_t *row, int pair0, const void *rope_row, int rope_dtype, int64_t stride_dim,
                                            int64_t stride_rot, int64_t stride_pair) {
#pragma unroll 1
  for (int i = 0; i < kPairs; ++i) {
    float f[2][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int64_t at = (2 * (pair0 + i) + e) * stride_dim;
      f[e][0] = rope_load(rope_row, at, rope_dtype);
      f[e][1] = rope_load(rope_row, at + stride_pair, rope_dtype);
      f[e][2] = rope_load(rope_row, at + stride_rot, rope_dtype);
      f[e][3] = rope_load(rope_row, at + stride_rot + stride_pair, rope_dtype);
    }
    rotate_pair(row[i], row[i + kPairs], f);
  }
}

__device__ __forceinline__ void norm_rope_row(uint32_t (&y)[H3S_HEAD_DIM / 2], const float *__restrict__ norm_weight,
                                              float epsilon, const void *rope_row, int rope_dtype,
                                              int64_t stride_dim, int64_t stride_rot, int64_t stride_pair) {
  const bool packed = stride_pair == 1 && stride_rot == 2 && stride_dim == 4 &&
                      (reinterpret_cast<uintptr_t>(rope_row) & 15) == 0;
  const RopeForm form = rope_row == nullptr ? kRopeNone
                        : !packed           ? kRopeStrided
                        : rope_dtype == H3S_BF16 ? kRopeBf16 : kRopeF32;
  if (form == kRopeBf16) return norm_rope_packed<kRopeBf16>(y, norm_weight, epsilon, static_cast<const uint4 *>(rope_row));
  if (form == kRopeF32) return norm_rope_packed<kRopeF32>(y, norm_weight, epsilon, static_cast<const uint4 *>(rope_row));
  norm_row(y, norm_weight, epsilon);
  if (form == kRopeNone) return;
  uint32_t row[H3S_HEAD_DIM / 2];
#pragma unroll
  for (int i = 0; i < H3S_HEAD_DIM / 2; ++i) row[i] = y[i];
  rotate_strided<24>(row, 0, rope_row, rope_dtype, stride_dim, stride_rot, stride_pair);
#pragma unroll
  for (int i = 0; i < H3S_HEAD_DIM / 2; ++i) y[i] = row[i];
}

// Half of such a row, as the carrier epilogue deals it to a thread: the channels
// 24*share + [0, 24) and 48 + 24*share + [0, 24), which are rotated against each other, and
// 96 + 16*share + [0, 16).
struct HalfRow {
  uint32_t first[12], second[12], rest[8];
};

// sum + x = the result + error, exactly (Knuth's two-sum)
__device__ __forceinline__ float two_sum(float a, float b, float &error) {
  const float s = __fadd_rn(a, b), back = __fsub_rn(s, a);
  error = __fadd_rn(__fsub_rn(a, __fsub_rn(s, back)), __fsub_rn(b, back));
  return s;
}

__device__ __forceinline__ void add_to(TripleSum &a, float x) {
  float e, f;
  a.sum = two_sum(a.sum, x, e);
  a.lost = two_sum(a.lost, e, f);
  a.rest = __fadd_rn(a.rest, f);
}

__device__ __forceinline__ TripleSum add_sums(const TripleSum &a, const TripleSum &b) {  // the same in either order
  float e, f, g;
  const float sum = two_sum(a.sum, b.sum, e);
  const float lost = two_sum(two_sum(a.lost, b.lost, f), e, g);
  return {sum, lost, __fadd_rn(__fadd_rn(a.rest, b.rest), __fadd_rn(f, g))};
}

// The nearest float: sum + lost = t + r exactly, and r + rest is rounded to odd, which keeps the last
// rounding from falling on the wrong side of a tie (Boldo and Melquiond)
__device__ __forceinline__ float nearest(const TripleSum &a) {
  float r, q;
  const float t = two_sum(a.sum, a.lost, r);
  const float d = two_sum(r, a.rest, q);
  int bits = __float_as_int(d);
  if (q != 0.f && (bits & 1) == 0) bits += (q > 0.f) == (d > 0.f) ? 1 : -1;
  return __fadd_rn(t, __int_as_float(bits));
}

__device__ __forceinline__ double wide(const TripleSum &a) {
  return static_cast<double>(a.sum) + (static_cast<double>(a.lost) + static_cast<double>(a.rest));
}

// `parts` partial sums `stride` floats apart, for totals that leave the range of a float
__device__ __noinline__ double wide_total(const float *partial, int parts, int stride) {
  double sum = 0.0;
#pragma unroll 1
  for (int i = 0; i < parts; ++i) sum += static_cast<double>(partial[i * stride]);
  return sum;
}

__device__ __forceinline__ TripleSum split_wide(double sum) {
  const float hi = static_cast<float>(sum);
  if (!(hi < INFINITY)) return {hi, 0.f, 0.f};
  const float lo = static_cast<float>(sum - static_cast<double>(hi));
  return {hi, lo, static_cast<float>(sum - static_cast<double>(hi) - static_cast<double>(lo))};
}

// Half rows whose squares leave the range in which every step below is exact.  Sums that are too small for that
// are handed on times -2^160.
constexpr double kTinySquares = 0x1p160;

__device__ __noinline__ TripleSum square_sum_wide(const uint32_t *row, bool tiny) {
  double sum = 0.0;
#pragma unroll 1
  for (int i = 0; i < 32; ++i) {
    const double lo = static_cast<double>(bf16_lo(row[i])), hi = static_cast<double>(bf16_hi(row[i]));
    sum = fma(lo, lo, sum);
    sum = fma(hi, hi, sum);
  }
  const TripleSum split = split_wide(tiny ? sum * kTinySquares : sum);
  return tiny ? TripleSum{-split.sum, -split.lost, -split.rest} : split;
}

__device__ __noinline__ float add_tiny_squares(const TripleSum &a, const TripleSum &b) {
  const double x = a.sum < 0.f ? wide(a) / -kTinySquares : wide(a), y = b.sum < 0.f ? wide(b) / -kTinySquares : wide(b);
  return static_cast<float>(x + y);
}

// The sum of squares of half a row, as good as in 64 bits (it keeps at least 56) and without its unit, which took 2000 to
// 6000 cycles a tile here and 30000 for a CTA's first.  The square of a bf16 value is exact in fp32.  The accumulator begins at a
// power of two that no square exceeds, so that acc + p - acc loses exactly what rounding took from p (Dekker's
// fast two-sum, which wants the larger operand first).  With base = 2^b the accumulator stays below 2^(b+5) and a loss
// below 2^(b-20); the losses have an accumulator of their own that begins at 2^(b-14), and what that one loses, at most
// 2^(b-38) at a time, is added up beside it.  With plain sums of the losses a row with one outlier kept 42 bits; the
// projection of 33272 x 3072 with norm and table took 1.06 ms then, 1.10 now, 1.52 in 64 bits.
__device__ __forceinline__ TripleSum half_row_squares(const HalfRow &y) {
  __nv_bfloat162 top = __floats2bfloat162_rn(0.f, 0.f);
  auto magnitude = [&](uint32_t w) {
    w &= 0x7fff7fffu;
    top = __hmax2_nan(top, *reinterpret_cast<const __nv_bfloat162 *>(&w));
  };
#pragma unroll
  for (int i = 0; i < 12; ++i) { magnitude(y.first[i]); magnitude(y.second[i]); }
#pragma unroll
  for (int i = 0; i < 8; ++i) magnitude(y.rest[i]);
  const uint32_t bits = *reinterpret_cast<const uint32_t *>(&top);
  const float lo_top = bf16_lo(bits), hi_top = bf16_hi(bits);
  const float most = fmaxf(lo_top, hi_top);
  const bool tiny = most < 1e-12f && most > 0.f && lo_top < 1e-12f && hi_top < 1e-12f;  // (a NaN is not)
  if (!(lo_top < 1e17f && hi_top < 1e17f) || tiny) {
    uint32_t row[32];
#pragma unroll
    for (int i = 0; i < 12; ++i) { row[i] = y.first[i]; row[12 + i] = y.second[i]; }
#pragma unroll
    for (int i = 0; i < 8; ++i) row[24 + i] = y.rest[i];
    return square_sum_wide(row, tiny);
  }
  // the next power of two above the largest square
  const float base = __uint_as_float((__float_as_uint(__fmul_rn(most, most)) & 0x7f800000u) + 0x00800000u);
  const float lost_base = __fmul_rn(base, 0x1p-14f);
  const float2 minus = make_float2(-1.f, -1.f);
  float2 acc[2] = {make_float2(base, base), make_float2(base, base)};
  float2 lost[2] = {make_float2(lost_base, lost_base), make_float2(lost_base, lost_base)};
  float2 rest[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  auto square = [&](uint32_t w, int i) {
    float2 &a = acc[i & 1], &l = lost[i & 1], &r = rest[i & 1];
    const float2 v = bf16_pair(w);
    const float2 next = fma2(v, v, a);
    const float2 loss = fma2(v, v, fma2(next, minus, a));  // v * v - (next - a)
    const float2 after = add2(l, loss);
    r = add2(r, add2(loss, fma2(after, minus, l)));  // loss - (after - l)
    a = next;
    l = after;
  };
#pragma unroll
  for (int i = 0; i < 12; ++i) { square(y.first[i], i); square(y.second[i], i + 1); }
#pragma unroll
  for (int i = 0; i < 8; ++i) square(y.rest[i], i);
  auto sum = [&](float a, float l, float r) { return TripleSum{__fsub_rn(a, base), __fsub_rn(l, lost_base), r}; };  // exact
  return add_sums(add_sums(sum(acc[0].x, lost[0].x, rest[0].x), sum(acc[0].y, lost[0].y, rest[0].y)),
                  add_sums(sum(acc[1].x, lost[1].x, rest[1].x), sum(acc[1].y, lost[1].y, rest[1].y)));
}

__device__ __forceinline__ uint32_t norm_pair(uint32_t y, float2 inverse_rms, const float *__restrict__ weight) {
  const float2 normed = mul2(mul2(bf16_pair(y), inverse_rms), *reinterpret_cast<const float2 *>(weight));
  return pack_bf16x2(normed.x, normed.y);
}

__device__ __forceinline__ void norm_half_row(HalfRow &y, float squares, const float *__restrict__ norm_weight,
                                              float epsilon, int share) {
  const float mean = __fadd_rn(__fmul_rn(squares, 1.0f / H3S_HEAD_DIM), epsilon);
  const float inverse_rms = __frsqrt_rn(mean);
  const float2 inverse = make_float2(inverse_rms, inverse_rms);
#pragma unroll
  for (int i = 0; i < 12; ++i) y.first[i] = norm_pair(y.first[i], inverse, norm_weight + 24 * share + 2 * i);
#pragma unroll
  for (int i = 0; i < 12; ++i) y.second[i] = norm_pair(y.second[i], inverse, norm_weight + 48 + 24 * share + 2 * i);
#pragma unroll
  for (int i = 0; i < 8; ++i) y.rest[i] = norm_pair(y.rest[i], inverse, norm_weight + 96 + 16 * share + 2 * i);
}

// The factors of one channel pair: 16 (bf16) or 32 bytes
__device__ __forceinline__ void rotate_bf16(uint32_t &first, uint32_t &second, const uint4 &w) {
  const float f[2][4] = {{bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y)},
                         {bf16_lo(w.z), bf16_hi(w.z), bf16_lo(w.w), bf16_hi(w.w)}};
  rotate_pair(first, second, f);
}
// 32 bytes of a row's table: whole sectors where it is aligned to them, as 16-byte loads of 32 different
// rows visit each one twice
__device__ __forceinline__ void load_sector(uint4 (&to)[2], const uint4 *from, bool sectors) {
  if (!sectors) {
    to[0] = __ldg(from);
    to[1] = __ldg(from + 1);
    return;
  }
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(to[0].x), "=r"(to[0].y), "=r"(to[0].z), "=r"(to[0].w), "=r"(to[1].x), "=r"(to[1].y), "=r"(to[1].z), "=r"(to[1].w)
               : "l"(from));
}
__device__ __forceinline__ void rotate_f32(uint32_t &first, uint32_t &second, const uint4 &u, const uint4 &w) {
  const float f[2][4] = {{__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w)},
                         {__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w)}};
  rotate_pair(first, second, f);
}

// Tile `tile` of the persistent order: row pair and column tile
__device__ __forceinline__ void tile_position(const GemmParams &prm, int tile, int &pair, int &tn) {
  const int per_group = kGemmGroupM * prm.n_tiles;
  const int group = tile / per_group, within = tile - group * per_group;
  const int first = group * kGemmGroupM;
  const int height = min(kGemmGroupM, prm.m_pairs - first);
  const int column = within / height;
  pair = first + within - column * height;
  tn = column;
}

template <int kMode>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GemmWarps<kMode>::kThreads, 1)
qkv_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const GemmParams prm) {
  extern __shared__ unsigned char smem_dyn[];
  // Offset arithmetic, so that the compiler still sees shared memory: with a pointer rounded up the epilogues' accesses were
  // generic ones (us, in turn: MLP of 33130 x 1024 x 4096 571 / 558, of 33272 x 3072 x 12288 2598 / 2586, block of 33272 tokens alike)
  unsigned char *smem = smem_dyn + ((1024u - (ptx::smem_u32(smem_dyn) & 1023u)) & 1023u);
  using L = GemmLayout<kMode>;
  using W = GemmWarps<kMode>;
  constexpr bool kCarriers = kMode == kModeCarriers;
  GemmShared &sh = *reinterpret_cast<GemmShared *>(smem + L::kOffBar);
  volatile int *abort_word = &sh.abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_steps = prm.hidden / kGemmK;
  const int total_tiles = prm.m_pairs * prm.n_tiles;
  const int rank = ptx::cluster_rank();  // 0: issues the pair's MMAs
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int tile_n = kMode == kModeDense ? prm.tile_n : kGemmN;

  let_next_start();
  if (threadIdx.x == 0) {
    for (int i = 0; i < L::kStages; ++i) {
      ptx::mbar_init(&sh.full[i], 1);
      ptx::mbar_init(&sh.empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&sh.acc_full[i], 1);
      ptx::mbar_init(&sh.acc_empty[i], 2 * W::kEpilogue);
      ptx::mbar_init(&sh.tile_ready[i], W::kEpilogue / 2);
      ptx::mbar_init(&sh.exchange_ready[i], W::kEpilogue / 2);
      for (int quarter = 0; quarter < 4; ++quarter) ptx::mbar_init(&sh.squares_ready[i][quarter], 2);
    }
    sh.abort_word = 0;
    ptx::fence_mbar_init();
  }
  if (warp == W::kIssue) {
    ptx::tmem_alloc_pair(&sh.tmem_base, kGemmTmemCols);
    ptx::tmem_relinquish_pair();
  }
  wait_for_previous();
  float *norm_weights = reinterpret_cast<float *>(smem + L::kOffNorm);
  if (kCarriers && prm.q_norm != nullptr) {
    for (int i = threadIdx.x; i < 2 * H3S_HEAD_DIM; i += W::kThreads) {
      const void *from = i < H3S_HEAD_DIM ? prm.q_norm : prm.k_norm;
      norm_weights[i] = rope_load(from, i % H3S_HEAD_DIM, prm.norm_dtype);
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::cluster_sync();  // both CTAs' barriers are initialised
  ptx::tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;

  if (warp == W::kLoad) {
    // One thread, its state kept from step to step: at 128 bytes of K a step the MMAs take 512 cycles, and
    // what this thread and the issuing one do for a step is a chain of dependent instructions.
    if (ptx::elect_one()) {
      ptx::prefetch_tensormap(&map_a);
      ptx::prefetch_tensormap(&map_b);
      // all four loads of the pair count on the first CTA's barrier
      const uint32_t full0 = ptx::cluster_address(&sh.full[0], 0);
      int stage = 0;
      uint32_t it = 0, previous = 1;  // steps so far, parity of the ring's previous use
      bool ok = true;
      for (int tile = first_tile; ok && tile < total_tiles; tile += tile_step) {
        int pair, tn;
        tile_position(prm, tile, pair, tn);
        const int row0 = pair * kGemmPairM + rank * kGemmM, col0 = tn * tile_n + rank * (tile_n / 2);
        for (int k = 0; k < prm.hidden; k += kGemmK) {
          if (!ptx::mbar_wait(&sh.empty[stage], previous, abort_word, kGemmAbortEmpty, prm.wait_budget_ns)) { ok = false; break; }
          const uint32_t full = full0 + stage * sizeof(uint64_t);
          if (rank == 0) ptx::mbar_arrive_expect_tx(&sh.full[stage], 2 * kGemmABytes + tile_n * kGemmK);
          ptx::tma_load_2d_pair(smem + stage * kGemmABytes, &map_a, full, k, row0);
          ptx::tma_load_2d_pair(smem + L::kOffB + stage * kGemmBBytes, &map_b, full, k, col0);
          ++it;
          if (++stage == L::kStages) { stage = 0; previous ^= 1u; }
        }
      }
      // the other CTA's last arrivals on `empty` have landed before this CTA may exit
      for (uint32_t i = it > L::kStages ? it - L::kStages : 0; ok && i < it; ++i)
        ok = ptx::mbar_wait(&sh.empty[i % L::kStages], (i / L::kStages) & 1u, abort_word, kGemmAbortEmpty, prm.wait_budget_ns);
    }
  } else if (warp == W::kIssue) {
    if (rank == 0 && ptx::elect_one()) {
      // every kind consumes 32 bytes of K per instruction: four instructions per 128-byte stage
      const int kind = kMode == kModeDense ? prm.operand_kind : H3S_GEMM_I8;
      const uint64_t a_desc0 = ptx::umma_desc_kmajor(ptx::smem_u32(smem), 1024, ptx::kSwizzle128);
      const uint64_t b_desc0 = ptx::umma_desc_kmajor(ptx::smem_u32(smem + L::kOffB), 1024, ptx::kSwizzle128);
      auto issue = [&](uint32_t idesc, auto mma) {
        int stage = 0;
        uint32_t round = 0, local = 0;
        for (int tile = first_tile; tile < total_tiles; tile += tile_step, ++local) {
          const int a = local & 1;
          const uint32_t acc_use = local >> 1, acc = tmem_base + a * kGemmN;
          if (!ptx::mbar_wait(&sh.acc_empty[a], (acc_use & 1u) ^ 1u, abort_word, kGemmAbortAccEmpty, prm.wait_budget_ns)) return;
          ptx::tc_fence_after();
          for (int ks = 0; ks < k_steps; ++ks) {
            if (!ptx::mbar_wait(&sh.full[stage], round, abort_word, kGemmAbortFull, prm.wait_budget_ns)) return;
            ptx::tc_fence_after();
            const uint64_t a_desc = a_desc0 + static_cast<uint64_t>(stage * (kGemmABytes >> 4));
            const uint64_t b_desc = b_desc0 + static_cast<uint64_t>(stage * (kGemmBBytes >> 4));
#pragma unroll
            for (int k = 0; k < kGemmK / 32; ++k) mma(acc, a_desc + 2 * k, b_desc + 2 * k, idesc, (ks > 0 || k > 0) ? 1u : 0u);
            ptx::tc_commit_pair(&sh.empty[stage]);
            if (++stage == L::kStages) { stage = 0; round ^= 1u; }
          }
          ptx::tc_commit_pair(&sh.acc_full[a]);
        }
      };
      auto i8 = [](uint32_t d, uint64_t x, uint64_t y, uint32_t i, uint32_t accumulate) { ptx::umma_i8_pair(d, x, y, i, accumulate); };
      auto f8 = [](uint32_t d, uint64_t x, uint64_t y, uint32_t i, uint32_t accumulate) { ptx::umma_f8_pair(d, x, y, i, accumulate); };
      auto f16 = [](uint32_t d, uint64_t x, uint64_t y, uint32_t i, uint32_t accumulate) { ptx::umma_f16_pair(d, x, y, i, accumulate); };
      if (kind == H3S_GEMM_I8) issue(ptx::umma_idesc(2, 1, 1, kGemmPairM, tile_n), i8);
      else if (kind == H3S_GEMM_E4M3) issue(ptx::umma_idesc(1, 0, 0, kGemmPairM, tile_n), f8);
      else if (kind == H3S_GEMM_BF16) issue(ptx::umma_idesc(1, 1, 1, kGemmPairM, tile_n), f16);
      else issue(ptx::umma_idesc(1, 0, 0, kGemmPairM, tile_n), f16);
    }
  } else if (W::epilogue(warp)) {
    // epilogue: warp group <-> 128-column half of the tile, thread <-> accumulator row (carriers: half a row)
    const int quarter = warp & 3;
    const int gi = W::kMany ? (warp >> 2) & 1 : warp >= 8 ? 1 : 0;
    const int share = warp >> 3;  // carriers: which half of the channels
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    uint32_t local = 0;
    const uint32_t acc_empty[2] = {ptx::cluster_address(&sh.acc_empty[0], 0), ptx::cluster_address(&sh.acc_empty[1], 0)};
    uint32_t exchanges = 0;  // uses of this half's exchange buffer and barrier so far
    uint32_t squared = 0;    // ... and of the sums of squares
    bool ok = true;
    for (int tile = first_tile; ok && tile < total_tiles; tile += tile_step, ++local) {
      int pair, tn;
      tile_position(prm, tile, pair, tn);
      const int tm = 2 * pair + rank;  // this CTA's 128 rows; may lie past the last row
      const int a = local & 1;
      const uint32_t acc_use = local >> 1;
      const int row = tm * kGemmM + quarter * 32 + lane;
      const bool row_ok = row < prm.rows;
      const int group_col0 = tn * tile_n + gi * H3S_HEAD_DIM;
      // scales come while the MMAs are still at it
      const float xs = prm.x_scale == nullptr ? 1.0f : (row_ok ? load_written(prm.x_scale + row) : 0.f);
      float *my_scales = reinterpret_cast<float *>(smem + L::kOffScale) + warp * 64;
      if (kCarriers) {  // without a group nothing is stored
        const int i = 2 * lane, channel = i < 24 ? 24 * share + i : i < 48 ? 24 + 24 * share + i : 48 + 16 * share + i;
        reinterpret_cast<float2 *>(my_scales)[lane] = load_written(reinterpret_cast<const float2 *>(prm.w_scale + (group_col0 < prm.n_out ? group_col0 : 0) + channel));
        __syncwarp();
      }
      {
        const bool got = ptx::mbar_wait(&sh.acc_full[a], acc_use & 1u, abort_word, kGemmAbortAccFull, prm.wait_budget_ns);
        if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
      }
      ptx::tc_fence_after();
      {
        const int group = group_col0 >> 7;  // 128-column group == (kind, head)
        const int columns_end = min(prm.n_out, (tn + 1) * tile_n);  // of the tile
        const bool group_ok = group_col0 < columns_end && tm * kGemmM < prm.rows;
        const bool normed = prm.q_norm != nullptr && group < 2 * prm.heads;
        if (kMode == kModeDense) {
          // ---- dense epilogue: scaled, biased, activated bf16 rows, staged for coalesced stores ----
          unsigned char *tile = smem + L::kOffTile + gi * kEpilogueTileBytes;
          const int local_row = quarter * 32 + lane;
          const float rs = xs;  // row_scale[row], 1 without row scales
          const bool integer = prm.operand_kind == H3S_GEMM_I8;
          uint4 *my_row = reinterpret_cast<uint4 *>(tile + local_row * (H3S_HEAD_DIM * 2));
          const bool gelu = prm.activation == H3S_ACT_GELU_TANH;
          const int blocks = min(H3S_HEAD_DIM, tile_n - gi * H3S_HEAD_DIM) / 32;  // of 32 columns; none or less: nothing of this half
          auto convert = [&](auto scale_tag, auto bias_tag, auto gelu_tag) {
#pragma unroll 1
            for (int cc = 0; cc < blocks; ++cc) {
              uint32_t acc[32], y[16];
              H3S_TMEM_LD32(tmem_base + lane_addr + a * kGemmN + gi * H3S_HEAD_DIM + cc * 32, acc);
              ptx::tmem_wait_ld(acc);
              dense_row32<decltype(scale_tag)::value, decltype(bias_tag)::value, decltype(gelu_tag)::value>(
                  acc, rs, prm.col_scale, prm.bias, group_col0 + cc * 32, prm.n_out, y);
#pragma unroll
              for (int c4 = 0; c4 < 4; ++c4)
                my_row[(cc * 4 + c4) ^ (local_row & 15)] = make_uint4(y[4 * c4], y[4 * c4 + 1], y[4 * c4 + 2], y[4 * c4 + 3]);
            }
          };
          using Yes = std::true_type;
          using No = std::false_type;
          if (!integer && prm.vector_columns) {
            if (prm.col_scale != nullptr) {
              if (prm.bias != nullptr) { if (gelu) convert(Yes{}, Yes{}, Yes{}); else convert(Yes{}, Yes{}, No{}); }
              else { if (gelu) convert(Yes{}, No{}, Yes{}); else convert(Yes{}, No{}, No{}); }
            } else {
              if (prm.bias != nullptr) { if (gelu) convert(No{}, Yes{}, Yes{}); else convert(No{}, Yes{}, No{}); }
              else { if (gelu) convert(No{}, No{}, Yes{}); else convert(No{}, No{}, No{}); }
            }
          } else {
#pragma unroll 1
          for (int cc = 0; cc < blocks; ++cc) {
            uint32_t acc[32];
            H3S_TMEM_LD32(tmem_base + lane_addr + a * kGemmN + gi * H3S_HEAD_DIM + cc * 32, acc);
            ptx::tmem_wait_ld(acc);
            uint32_t y[16];
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const int col = group_col0 + cc * 32 + i;
              const float4 cs4 = column4(prm.col_scale, col, prm.n_out, 1.0f), bias4 = column4(prm.bias, col, prm.n_out, 0.f);
              const float cs[4] = {cs4.x, cs4.y, cs4.z, cs4.w}, bias[4] = {bias4.x, bias4.y, bias4.z, bias4.w};
              float v[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float value = integer ? static_cast<float>(static_cast<int>(acc[i + e])) : __uint_as_float(acc[i + e]);
                value = __fmul_rn(value, __fmul_rn(rs, cs[e]));
                if (prm.bias != nullptr) value = __fadd_rn(value, bias[e]);
                if (gelu) value = gelu_tanh2(make_float2(value, value)).x;
                v[e] = value;
              }
              y[i >> 1] = pack_bf16x2(v[0], v[1]);
              y[(i >> 1) + 1] = pack_bf16x2(v[2], v[3]);
            }
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4)
              my_row[(cc * 4 + c4) ^ (local_row & 15)] = make_uint4(y[4 * c4], y[4 * c4 + 1], y[4 * c4 + 2], y[4 * c4 + 3]);
          }
          }
          // the accumulator has been read: the MMA warp may refill it
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive_cluster(acc_empty[a]);
          if (!group_ok) continue;  // the same for the four warps of this half
          if (lane == 0) ptx::mbar_arrive(&sh.tile_ready[gi]);
          {
            const bool got = ptx::mbar_wait(&sh.tile_ready[gi], exchanges & 1u, abort_word, kGemmAbortTile,
                                            prm.wait_budget_ns);
            if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
          }
          // 16 threads per row, 16 bytes each: a warp writes two rows of 256 contiguous bytes
          const int g = quarter * 32 + lane, slot = g >> 4, c = g & 15;
          uint4 raw[16];
#pragma unroll
          for (int p = 0; p < 16; ++p) {
            const int r = p * 8 + slot;
            raw[p] = *reinterpret_cast<const uint4 *>(tile + r * (H3S_HEAD_DIM * 2) + ((c ^ (r & 15)) << 4));
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sh.exchange_ready[gi]);
          {
            const bool got = ptx::mbar_wait(&sh.exchange_ready[gi], exchanges & 1u, abort_word, kGemmAbortExchange,
                                            prm.wait_budget_ns);
            if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
            ++exchanges;
          }
          const int valid = min(kGemmM, prm.rows - tm * kGemmM);
          const int col = group_col0 + c * 8;
          if (col < columns_end) {  // a multiple of 8: a 16-byte chunk is inside or outside as a whole
            __nv_bfloat16 *dst = prm.dense_out + static_cast<int64_t>(tm) * kGemmM * prm.ldc + col;
#pragma unroll
            for (int p = 0; p < 16; ++p) {
              const int r = p * 8 + slot;
              if (r < valid) *reinterpret_cast<uint4 *>(dst + static_cast<int64_t>(r) * prm.ldc) = raw[p];
            }
          }
          continue;  // acc_empty was signalled above
        }
        if (kCarriers) {
          // ---- carriers straight from the accumulators ----
          // Phase A, two threads per row: de-quantise the row of this head to bf16
          // (+ norm and rotation) and stage it in shared memory, 16-byte chunk c of
          // row r at chunk position c ^ (r & 15) so that neither these row-wise
          // writes nor the column-wise reads of phase B collide on banks.
          unsigned char *tile = smem + L::kOffTile + gi * kEpilogueTileBytes;
          EpilogueExchange &ex = reinterpret_cast<EpilogueExchange *>(smem + L::kOffExchange)[gi];
          const int local_row = quarter * 32 + lane;
          {
            HalfRow y;
            const float2 xs2 = make_float2(xs, xs);
            const uint32_t columns = tmem_base + lane_addr + a * kGemmN + gi * H3S_HEAD_DIM;
            auto dequantise = [&](uint32_t lo, uint32_t hi, int i) {  // the i-th and the next of this share's channels
              const float2 ws = *reinterpret_cast<const float2 *>(my_scales + i);
              const float2 value = mul2(make_float2(static_cast<float>(static_cast<int>(lo)),
                                                    static_cast<float>(static_cast<int>(hi))), mul2(xs2, ws));
              return pack_bf16x2(value.x, value.y);
            };
            auto read24 = [&](uint32_t (&to)[12], int channel, int first) {
              uint32_t acc[16], more[8];
              H3S_TMEM_LD16(columns + channel, acc);
              H3S_TMEM_LD8(columns + channel + 16, more);
              ptx::tmem_wait_ld(acc);
              ptx::tmem_wait_ld(more);
#pragma unroll
              for (int i = 0; i < 8; ++i) to[i] = dequantise(acc[2 * i], acc[2 * i + 1], first + 2 * i);
#pragma unroll
              for (int i = 0; i < 4; ++i) to[8 + i] = dequantise(more[2 * i], more[2 * i + 1], first + 16 + 2 * i);
            };
            read24(y.first, 24 * share, 0);
            read24(y.second, 48 + 24 * share, 24);
            {
              uint32_t acc[16];
              H3S_TMEM_LD16(columns + 96 + 16 * share, acc);
              ptx::tmem_wait_ld(acc);
#pragma unroll
              for (int i = 0; i < 8; ++i) y.rest[i] = dequantise(acc[2 * i], acc[2 * i + 1], 48 + 2 * i);
            }
            // the accumulator is in registers: the MMA warp may refill it
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive_cluster(acc_empty[a]);
            if (!group_ok) continue;  // the same for the eight warps of this half
            if (normed) {
              const TripleSum mine = half_row_squares(y);
              ex.squares[share][local_row] = mine;
              __syncwarp();
              if (lane == 0) ptx::mbar_arrive(&sh.squares_ready[gi][quarter]);
              const void *rope_row = nullptr;
              if (prm.rope != nullptr && row_ok) {
                const int64_t offset = static_cast<int64_t>(row) * prm.rope_stride_seq;
                rope_row = prm.rope_dtype == H3S_F32
                               ? static_cast<const void *>(static_cast<const float *>(prm.rope) + offset)
                               : static_cast<const void *>(static_cast<const __nv_bfloat16 *>(prm.rope) + offset);
              }
              const bool packed = prm.rope_stride_pair == 1 && prm.rope_stride_rot == 2 && prm.rope_stride_dim == 4 &&
                                  (reinterpret_cast<uintptr_t>(rope_row) & 15) == 0;
              const bool sectors = (reinterpret_cast<uintptr_t>(rope_row) & 31) == 0;
              const RopeForm form = rope_row == nullptr ? kRopeNone
                                    : !packed           ? kRopeStrided
                                    : prm.rope_dtype == H3S_BF16 ? kRopeBf16 : kRopeF32;
              // the first factors travel while the norm is computed
              uint4 ahead[2][2];
              if (form == kRopeBf16) {
#pragma unroll
                for (int k = 0; k < 2; ++k) load_sector(ahead[k], static_cast<const uint4 *>(rope_row) + 12 * share + 2 * k, sectors);
              }
              const bool got = ptx::mbar_wait(&sh.squares_ready[gi][quarter], squared & 1u, abort_word, kGemmAbortSquares,
                                              prm.wait_budget_ns);
              if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
              ++squared;
              const TripleSum theirs = ex.squares[1 - share][local_row];
              float squares;
              if (mine.sum < 0.f || theirs.sum < 0.f) {
                squares = add_tiny_squares(mine, theirs);
              } else {
                const TripleSum both = add_sums(mine, theirs);
                squares = both.sum < INFINITY ? nearest(both) : both.sum;  // infinite: nothing is left to correct
              }
              norm_half_row(y, squares, norm_weights + (group < prm.heads ? 0 : H3S_HEAD_DIM), prm.epsilon, share);
              if (form == kRopeBf16) {
                const uint4 *table = static_cast<const uint4 *>(rope_row) + 12 * share;
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                  const uint4 now[2] = {ahead[k & 1][0], ahead[k & 1][1]};
                  if (k + 2 < 6) load_sector(ahead[k & 1], table + 2 * (k + 2), sectors);
                  rotate_bf16(y.first[2 * k], y.second[2 * k], now[0]);
                  rotate_bf16(y.first[2 * k + 1], y.second[2 * k + 1], now[1]);
                }
              } else if (form == kRopeF32) {
                const uint4 *table = static_cast<const uint4 *>(rope_row) + 24 * share;
#pragma unroll
                for (int b = 0; b < 12; b += 4) {
                  uint4 now[4][2];
#pragma unroll
                  for (int k = 0; k < 4; ++k) load_sector(now[k], table + 2 * (b + k), sectors);
#pragma unroll
                  for (int k = 0; k < 4; ++k) rotate_f32(y.first[b + k], y.second[b + k], now[k][0], now[k][1]);
                }
              } else if (form == kRopeStrided) {
                uint32_t pairs[24];
#pragma unroll
                for (int k = 0; k < 12; ++k) { pairs[k] = y.first[k]; pairs[12 + k] = y.second[k]; }
                rotate_strided<12>(pairs, 12 * share, rope_row, prm.rope_dtype, prm.rope_stride_dim, prm.rope_stride_rot,
                                   prm.rope_stride_pair);
#pragma unroll
                for (int k = 0; k < 12; ++k) { y.first[k] = pairs[k]; y.second[k] = pairs[12 + k]; }
              }
            }
            uint4 *my_row = reinterpret_cast<uint4 *>(tile + local_row * (H3S_HEAD_DIM * 2));
            auto stage = [&](int chunk, const uint32_t *w) {  // rows past the chunk count as zeros
              my_row[chunk ^ (local_row & 15)] = row_ok ? make_uint4(w[0], w[1], w[2], w[3]) : make_uint4(0u, 0u, 0u, 0u);
            };
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              stage(3 * share + c, y.first + 4 * c);
              stage(6 + 3 * share + c, y.second + 4 * c);
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) stage(12 + 2 * share + c, y.rest + 4 * c);
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sh.tile_ready[gi]);
          {
            const bool got = ptx::mbar_wait(&sh.tile_ready[gi], exchanges & 1u, abort_word, kGemmAbortTile,
                                            prm.wait_budget_ns);
            if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
          }
          // Phase B, 16 threads per row, 8 channels each: thread (slot, c) holds rows
          // slot, slot+16, ... slot+112 of channels 8c..8c+7.
          const int kind = group / prm.heads, head = group - kind * prm.heads;
          const int t = share * 128 + quarter * 32 + lane;  // thread within this half's 256
          const int slot = t >> 4, c = t & 15;
          const int half_warp = share * 4 + quarter;
          const bool quantise_here = kind == 0 || (kind == 1 && prm.k8 != nullptr);
          uint4 raw[8];
#pragma unroll
          for (int p = 0; p < 8; ++p) {
            const int r = p * 16 + slot;
            raw[p] = *reinterpret_cast<const uint4 *>(tile + r * (H3S_HEAD_DIM * 2) + ((c ^ (r & 15)) << 4));
          }
          {
            // partial statistics of rows 0-63 (passes 0-3) and 64-127 (passes 4-7)
            float part[2][8];
            __nv_bfloat162 top[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              top[h] = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
              for (int i = 0; i < 8; ++i) part[h][i] = 0.f;
#pragma unroll
              for (int p = 4 * h; p < 4 * h + 4; ++p) {
                const uint32_t w[4] = {raw[p].x, raw[p].y, raw[p].z, raw[p].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  if (kind == 2) {
                    part[h][2 * i] = fmaxf(part[h][2 * i], fabsf(bf16_lo(w[i])));
                    part[h][2 * i + 1] = fmaxf(part[h][2 * i + 1], fabsf(bf16_hi(w[i])));
                  } else {
                    const float2 sum = add2(make_float2(part[h][2 * i], part[h][2 * i + 1]), bf16_pair(w[i]));
                    part[h][2 * i] = sum.x;
                    part[h][2 * i + 1] = sum.y;
                    if (quantise_here) {  // magnitudes two at a time: clear both sign bits, packed bf16 maximum
                      const uint32_t magnitude = w[i] & 0x7fff7fffu;
                      top[h] = __hmax2(top[h], *reinterpret_cast<const __nv_bfloat162 *>(&magnitude));
                    }
                  }
                }
              }
              if (quantise_here) {
                const uint32_t bits = *reinterpret_cast<const uint32_t *>(&top[h]);
                const float amax = warp_max(fmaxf(bf16_lo(bits), bf16_hi(bits)));
                if (lane == 0) ex.amax[h][half_warp] = amax;
              }
            }
            // the warp's two slots together: one of them leaves the first half's values, one the second's
            float *column = ex.column[lane >> 4][half_warp] + c * 8;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float mine = lane < 16 ? part[0][i] : part[1][i];
              const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? part[1][i] : part[0][i], 16);
              column[i] = kind == 2 ? fmaxf(mine, other) : mine + other;
            }
          }
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(&sh.exchange_ready[gi]);
          {
            const bool got = ptx::mbar_wait(&sh.exchange_ready[gi], exchanges & 1u, abort_word, kGemmAbortExchange,
                                            prm.wait_budget_ns);
            if (!__all_sync(0xffffffffu, got)) { ok = false; break; }
            ++exchanges;
          }
          // every thread of this half now holds its share of the tile in registers: the
          // staging tile may be overwritten, the exchange block is read below
          const int tile_row0 = prm.row_start + tm * kGemmM;  // first row of this tile within the sequence
          const int valid = min(kGemmM, prm.rows - tm * kGemmM);
          const int valid_half[2] = {min(H3S_KV_TILE, valid), max(0, valid - H3S_KV_TILE)};
          float amax_half[2] = {0.f, 0.f};
          if (quantise_here) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
              for (int w = 0; w < 8; ++w) amax_half[h] = fmaxf(amax_half[h], ex.amax[h][w]);
            }
          }
          // channel g of this head: totals over the partial sums from `first` on, eight to a row half
          const int g = t & (H3S_HEAD_DIM - 1);
          auto total = [&](int first, auto parts) {
            const float *partial = &ex.column[0][0][g] + first * H3S_HEAD_DIM;
            TripleSum sum = {partial[0], 0.f, 0.f};
#pragma unroll
            for (int w = 1; w < decltype(parts)::value; ++w) add_to(sum, partial[w * H3S_HEAD_DIM]);
            return sum;
          };
          // every step towards such a sum was a finite float, and its mean is a normal one
          auto in_range = [](const TripleSum &sum) {
            return fabsf(sum.sum) < 1e30f && (fabsf(sum.sum) > 1e-20f || (sum.sum == 0.f && sum.lost == 0.f));
          };
          auto total64 = [&](const TripleSum &sum, int first, int parts) {
            return in_range(sum) ? wide(sum) : wide_total(&ex.column[0][0][g] + first * H3S_HEAD_DIM, parts, H3S_HEAD_DIM);
          };
          // the mean over `rows` rows; a power of two divides exactly
          auto store_mean = [&](void *base, int64_t at, int first, auto parts, int rows, int whole) {
            const TripleSum sum = total(first, parts);
            if (rows == whole && prm.summary_dtype == H3S_F32 && in_range(sum))
              static_cast<float *>(base)[at] = __fmul_rn(nearest(sum), 1.0f / static_cast<float>(whole));
            else
              store_summary(base, prm.summary_dtype, at, total64(sum, first, decltype(parts)::value) / rows);
            return sum;
          };
          using Sixteen = std::integral_constant<int, 16>;
          using Eight = std::integral_constant<int, 8>;
          if (kind == 0) {
            const int blocks_total = (prm.sequence_total + H3S_Q_TILE - 1) / H3S_Q_TILE;
            const int block = tile_row0 / H3S_Q_TILE;
            const float scale = __fadd_rn(__fdiv_rn(fmaxf(amax_half[0], amax_half[1]), 127.0f), 1.0e-7f);
            if (t == 0) prm.q_scale[head * blocks_total + block] = scale;
            if (share == 0)
              store_mean(prm.q_summary, (static_cast<int64_t>(head) * blocks_total + block) * H3S_HEAD_DIM + g, 0, Sixteen{},
                         valid, H3S_Q_TILE);
            int8_t *dst = prm.q8 + (static_cast<int64_t>(head) * prm.sequence_total + tile_row0) * H3S_HEAD_DIM + c * 8;
            const SharedDivisor by_scale = make_divisor(scale);
            auto emit = [&](auto exact) {
#pragma unroll
              for (int p = 0; p < 8; ++p) {
                const int r = p * 16 + slot;
                if (r < valid) quantise8<decltype(exact)::value>(raw[p], by_scale, dst + static_cast<int64_t>(r) * H3S_HEAD_DIM);
              }
            };
            if (by_scale.exact) emit(std::true_type{}); else emit(std::false_type{});
          } else if (kind == 1) {
            const int blocks_total = (prm.sequence_total + H3S_KV_TILE - 1) / H3S_KV_TILE;
            const int block0 = tile_row0 / H3S_KV_TILE;
            if (valid_half[share] > 0) {
              const TripleSum sum = store_mean(prm.k_summary, (static_cast<int64_t>(head) * blocks_total + block0 + share) * H3S_HEAD_DIM + g,
                                               8 * share, Eight{}, valid_half[share], H3S_KV_TILE);
              if (prm.k_sum != nullptr) atomicAdd(prm.k_sum + head * H3S_HEAD_DIM + g, total64(sum, 8 * share, 8));
            }
            if (prm.k8 != nullptr) {
              int8_t *dst = prm.k8 + (static_cast<int64_t>(head) * prm.sequence_total + tile_row0) * H3S_HEAD_DIM + c * 8;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const float scale = __fadd_rn(__fdiv_rn(amax_half[h], 127.0f), 1.0e-7f);
                if (t == 0 && valid_half[h] > 0) prm.k_scale[head * blocks_total + block0 + h] = scale;
                const SharedDivisor by_scale = make_divisor(scale);
                auto emit = [&](auto exact) {
#pragma unroll
                  for (int p = 4 * h; p < 4 * h + 4; ++p) {
                    const int r = p * 16 + slot;
                    if (r < valid) quantise8<decltype(exact)::value>(raw[p], by_scale, dst + static_cast<int64_t>(r) * H3S_HEAD_DIM);
                  }
                };
                if (by_scale.exact) emit(std::true_type{}); else emit(std::false_type{});
              }
            } else {
              __nv_bfloat16 *dst = prm.k_stage + (static_cast<int64_t>(head) * prm.sequence_total + tile_row0) * H3S_HEAD_DIM + c * 8;
#pragma unroll
              for (int p = 0; p < 8; ++p) {
                const int r = p * 16 + slot;
                if (r < valid) *reinterpret_cast<uint4 *>(dst + static_cast<int64_t>(r) * H3S_HEAD_DIM) = raw[p];
              }
            }
          } else {
            float peak = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w) peak = fmaxf(peak, ex.column[share][w][g]);
            // non-negative floats order like their bit patterns
            atomicMax(prm.v_amax_bits + head * H3S_HEAD_DIM + g, __float_as_uint(peak));
            __nv_bfloat16 *dst = prm.v_stage + (static_cast<int64_t>(head) * prm.sequence_total + tile_row0) * H3S_HEAD_DIM + c * 8;
#pragma unroll
            for (int p = 0; p < 8; ++p) {
              const int r = p * 16 + slot;
              if (r < valid) *reinterpret_cast<uint4 *>(dst + static_cast<int64_t>(r) * H3S_HEAD_DIM) = raw[p];
            }
          }
          continue;  // acc_empty was signalled above
        }
        if (!normed) {
#pragma unroll 1
          for (int cc = 0; cc < H3S_HEAD_DIM / 32; ++cc) {
            uint32_t acc[32];
            H3S_TMEM_LD32(tmem_base + lane_addr + a * kGemmN + gi * H3S_HEAD_DIM + cc * 32, acc);
            ptx::tmem_wait_ld(acc);
            const int col0 = group_col0 + cc * 32;
            if (row_ok && group_ok) {
              __nv_bfloat16 *dst = prm.out + group * prm.out_stride_head + static_cast<int64_t>(row) * H3S_HEAD_DIM + cc * 32;
#pragma unroll
              for (int i = 0; i < 32; i += 8) {
                uint4 w;
                uint32_t *wp = reinterpret_cast<uint32_t *>(&w);
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                  // acc * (row_scale * column_scale), the product of the scales first (fused_qkv.py:222,424)
                  const float y0 = __fmul_rn(static_cast<float>(static_cast<int>(acc[i + e])), __fmul_rn(xs, __ldg(prm.w_scale + col0 + i + e)));
                  const float y1 = __fmul_rn(static_cast<float>(static_cast<int>(acc[i + e + 1])), __fmul_rn(xs, __ldg(prm.w_scale + col0 + i + e + 1)));
                  const __nv_bfloat162 t = __floats2bfloat162_rn(y0, y1);
                  wp[e >> 1] = *reinterpret_cast<const uint32_t *>(&t);
                }
                *reinterpret_cast<uint4 *>(dst + i) = w;
              }
            }
          }
        } else {
          // Q or K head: the whole 128-channel row of this thread is needed at once
          uint32_t y[H3S_HEAD_DIM / 2];
#pragma unroll
          for (int cc = 0; cc < H3S_HEAD_DIM / 32; ++cc) {
            uint32_t acc[32];
            H3S_TMEM_LD32(tmem_base + lane_addr + a * kGemmN + gi * H3S_HEAD_DIM + cc * 32, acc);
            ptx::tmem_wait_ld(acc);
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const float2 ws = __ldg(reinterpret_cast<const float2 *>(prm.w_scale + group_col0 + cc * 32 + i));
              y[cc * 16 + (i >> 1)] =
                  pack_bf16x2(__fmul_rn(static_cast<float>(static_cast<int>(acc[i])), __fmul_rn(xs, ws.x)),
                              __fmul_rn(static_cast<float>(static_cast<int>(acc[i + 1])), __fmul_rn(xs, ws.y)));
            }
          }
          if (row_ok && group_ok) {
            const void *rope_row = nullptr;
            if (prm.rope != nullptr) {
              const int64_t offset = static_cast<int64_t>(row) * prm.rope_stride_seq;
              rope_row = prm.rope_dtype == H3S_F32
                             ? static_cast<const void *>(static_cast<const float *>(prm.rope) + offset)
                             : static_cast<const void *>(static_cast<const __nv_bfloat16 *>(prm.rope) + offset);
            }
            norm_rope_row(y, group < prm.heads ? prm.q_norm : prm.k_norm, prm.epsilon, rope_row, prm.rope_dtype,
                          prm.rope_stride_dim, prm.rope_stride_rot, prm.rope_stride_pair);
            __nv_bfloat16 *dst = prm.out + group * prm.out_stride_head + static_cast<int64_t>(row) * H3S_HEAD_DIM;
#pragma unroll
            for (int i = 0; i < H3S_HEAD_DIM / 2; i += 4)
              *reinterpret_cast<uint4 *>(dst + 2 * i) = make_uint4(y[i], y[i + 1], y[i + 2], y[i + 3]);
          }
        }
      }
      ptx::tc_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive_cluster(acc_empty[a]);
    }
  }

  __syncthreads();
  const int code = sh.abort_word;
  if (code != 0) {
    __nanosleep(200000);
    if (threadIdx.x == 0 && prm.status != nullptr) {
      if (atomicCAS(prm.status, 0, code) == 0) prm.status[1] = blockIdx.x;
    }
  }
  ptx::cluster_sync();  // neither CTA leaves while the other may still signal its barriers or its TMEM is written
  if (warp == W::kIssue) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc_pair(tmem_base, kGemmTmemCols);
  }
}

inline int make_tensor_map_u8_2d(CUtensorMap *map, const void *base, uint64_t dim0, uint64_t dim1,
                                 uint64_t stride1_bytes, uint32_t box0, uint32_t box1, const char *what) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return fail(H3S_ECUDA, "%s: cuTensorMapEncodeTiled is unavailable", what);
  const cuuint64_t dims[2] = {dim0, dim1};
  const cuuint64_t strides[1] = {stride1_bytes};
  const cuuint32_t box[2] = {box0, box1};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult rc = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, elem,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS)
    return fail(H3S_ECUDA, "%s: cuTensorMapEncodeTiled failed with CUresult %d", what, static_cast<int>(rc));
  return H3S_OK;
}

int convrot_quant_rows(const void *x, int64_t x_stride_row, int rows, int hidden, int8_t *x_i8, float *x_scale, uint32_t *clear, int words,
                       cudaStream_t stream) {
  H3S_CHECK_ARG(x != nullptr && x_i8 != nullptr && x_scale != nullptr, "convrot_quant_rows: NULL pointer");
  H3S_CHECK_ARG(rows > 0 && hidden > 0 && hidden % kRotGroup == 0 && hidden / kRotGroup <= 32,
                "convrot_quant_rows: hidden %d must be a multiple of 256 and at most 8192", hidden);
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15) == 0 && x_stride_row % 8 == 0 && x_stride_row >= hidden,
                "convrot_quant_rows: input must be 16-byte aligned with a row stride that is a multiple of 8");
  H3S_CHECK_ARG((reinterpret_cast<uintptr_t>(x_i8) & 7) == 0, "convrot_quant_rows: output must be 8-byte aligned");
  const int row_bytes = 32 * rot_stride(hidden / kRotGroup) * static_cast<int>(sizeof(float));  // of shared memory, 33 KB at most
  auto launch = [&](auto kernel, int warps) {
    H3S_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kRotWarps * 32 * rot_stride(32) * static_cast<int>(sizeof(float))));
    H3S_CHECK_CUDA(launch_next(kernel, ceil_div(rows, warps), warps * 32, warps * row_bytes, stream, static_cast<const __nv_bfloat16 *>(x),
                               x_stride_row, rows, hidden, x_i8, x_scale, clear, words));
    return H3S_OK;
  };
  // Of wide rows shared memory holds few: as many as go in with one to a CTA, and more loads to each.  us for 4096 rows, four to a CTA with
  // six loads ahead / one with six / one with twelve: 5120 channels 28.7 / 23.4 / 21.6, 8192 64.9 / 49.1 / 42.0; 3072 12.9 / 13.0 / 13.4,
  // 1024 5.8 / 6.3 / 6.0.
  // But where one round of CTAs with four holds all rows, more than two for each SM, nothing is won by that, and a quarter of the CTAs
  // start sooner.  us with the GEMM behind it (8 heads), one / four to a CTA: 592 x 3328 21.6 / 20.6, 2304 x 3328 33.9 / 31.5, 888 x 4096
  // 26.0 / 24.3, 1776 x 4096 34.6 / 33.3, 592 x 5120 26.8 / 25.5, 1184 x 5120 28.0 / 26.3, 592 x 8192 35.7 / 33.3; beyond one round 1480 x
  // 5120 28.7 / 30.1, 888 x 8192 36.4 / 40.4.  By itself 64 x 8192 7.2 / 7.8, 300 x 5120 5.5 / 5.9.
  constexpr int kSharedPerSm = 228 * 1024, kReserved = 1024;  // of a CTA
  const int one_round = kSmCount * kRotWarps * (kSharedPerSm / (kRotWarps * row_bytes + kReserved));
  const bool one_to_a_cta = hidden > 3072 && (rows <= 2 * kSmCount || rows > one_round);
  return one_to_a_cta ? launch(convrot_quant_rows_kernel<12>, 1) : launch(convrot_quant_rows_kernel<6>, kRotWarps);
}

}  // namespace h3s

extern "C" {

int h3s_convrot_quant_rows(const void *x, int64_t x_stride_row, int rows, int hidden, int8_t *x_i8,
                           float *x_scale, h3s_stream_t stream) {
  return h3s::convrot_quant_rows(x, x_stride_row, rows, hidden, x_i8, x_scale, nullptr, 0, static_cast<cudaStream_t>(stream));
}

static int qkv_gemm_chunk_impl(const int8_t *x_i8, const float *x_scale, const int8_t *w_i8, const float *w_scale,
                               int rows, int hidden, int n_out, void *out_bf16, int64_t out_stride_head,
                               const float *q_norm, const float *k_norm, float epsilon, const void *rope,
                               int rope_dtype, const int64_t *rope_strides, int heads, int32_t *status,
                               h3s_stream_t stream, const char *who, const h3s_qkv_carriers *carriers = nullptr,
                               int norm_dtype = H3S_F32) {
  using namespace h3s;
  H3S_CHECK_ARG(x_i8 && x_scale && w_i8 && w_scale && (out_bf16 || carriers), "%s: NULL pointer", who);
  H3S_CHECK_ARG(rows > 0 && hidden > 0 && hidden % kGemmK == 0, "%s: hidden %d must be a positive multiple of 128", who, hidden);
  H3S_CHECK_ARG(n_out > 0 && n_out % H3S_HEAD_DIM == 0, "%s: n_out %d must be a multiple of 128", who, n_out);
  H3S_CHECK_ARG(carriers != nullptr ||
                    (out_stride_head >= static_cast<int64_t>(rows) * H3S_HEAD_DIM && out_stride_head % 8 == 0),
                "%s: out_stride_head %lld is smaller than rows*128", who, static_cast<long long>(out_stride_head));
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(x_i8) | reinterpret_cast<uintptr_t>(w_i8) | reinterpret_cast<uintptr_t>(out_bf16)) & 15) == 0,
                "%s: operands must be 16-byte aligned", who);
  if (carriers != nullptr) {
    const h3s_qkv_carriers &c = *carriers;
    H3S_CHECK_ARG(heads > 0 && n_out == 3 * heads * H3S_HEAD_DIM, "%s: n_out %d is not 3*heads*128 for %d heads", who, n_out, heads);
    H3S_CHECK_ARG(c.q8 && c.q_scale && c.q_summary && c.k_summary && c.v_stage && c.stats,
                  "%s: q8, q_scale, q_summary, k_summary, v_stage and stats are required", who);
    H3S_CHECK_ARG((c.k8 != nullptr) == (c.k_scale != nullptr) && (c.k8 != nullptr) != (c.k_stage != nullptr),
                  "%s: give either k8 + k_scale (K quantised per chunk) or k_stage (K staged for smoothing)", who);
    H3S_CHECK_ARG(c.summary_dtype >= H3S_F32 && c.summary_dtype <= H3S_F64, "%s: bad summary dtype %d", who, c.summary_dtype);
    H3S_CHECK_ARG(c.row_start >= 0 && c.row_start % H3S_Q_TILE == 0 && c.row_start + rows <= c.sequence_total,
                  "%s: chunk [%d,%d) must start on a multiple of 128 inside the sequence of %d", who, c.row_start,
                  c.row_start + rows, c.sequence_total);
    H3S_CHECK_ARG(rows % H3S_Q_TILE == 0 || c.row_start + rows == c.sequence_total,
                  "%s: only the final chunk may contain a partial tile", who);
    const uintptr_t all = reinterpret_cast<uintptr_t>(c.q8) | reinterpret_cast<uintptr_t>(c.k8) |
                          reinterpret_cast<uintptr_t>(c.k_stage) | reinterpret_cast<uintptr_t>(c.v_stage);
    H3S_CHECK_ARG((all & 15) == 0 && (reinterpret_cast<uintptr_t>(c.stats) & 7) == 0,
                  "%s: carriers and staging must be 16-byte aligned, stats 8-byte aligned", who);
  }
  if (q_norm != nullptr || k_norm != nullptr || rope != nullptr) {
    H3S_CHECK_ARG(q_norm != nullptr && k_norm != nullptr, "%s: both norm weights are needed", who);
    H3S_CHECK_ARG(heads > 0 && n_out == 3 * heads * H3S_HEAD_DIM, "%s: n_out %d is not 3*heads*128 for %d heads", who, n_out, heads);
    H3S_CHECK_ARG(epsilon >= 0.f, "%s: negative epsilon", who);
    H3S_CHECK_ARG(norm_dtype == H3S_F32 || norm_dtype == H3S_BF16, "%s: norm weights must be fp32 or bf16", who);
    if (rope != nullptr) {
      H3S_CHECK_ARG(rope_strides != nullptr, "%s: rope strides missing", who);
      H3S_CHECK_ARG(rope_dtype == H3S_F32 || rope_dtype == H3S_BF16, "%s: rope must be fp32 or bf16", who);
    }
  }
  const int cap = h3s_device_capability();
  if (cap < 0) return cap;
  if (cap / 10 != 10) return fail(H3S_EARCH, "%s: needs an sm_100 device, found sm_%d", who, cap);
  CUtensorMap ma, mb;
  int rc = make_tensor_map_u8_2d(&ma, x_i8, hidden, rows, hidden, kGemmK, kGemmM, "qkv_gemm_chunk A map");
  if (rc) return rc;
  rc = make_tensor_map_u8_2d(&mb, w_i8, hidden, n_out, hidden, kGemmK, kGemmN / 2, "qkv_gemm_chunk B map");
  if (rc) return rc;
  GemmParams prm;
  prm.x_scale = x_scale; prm.w_scale = w_scale; prm.out = static_cast<__nv_bfloat16 *>(out_bf16);
  prm.out_stride_head = out_stride_head; prm.status = status;
  prm.rows = rows; prm.n_out = n_out; prm.hidden = hidden;
  prm.m_pairs = ceil_div(rows, kGemmPairM); prm.n_tiles = ceil_div(n_out, kGemmN);
  prm.q_norm = q_norm; prm.k_norm = k_norm; prm.rope = rope; prm.rope_dtype = rope_dtype;
  prm.rope_stride_seq = rope ? rope_strides[0] : 0; prm.rope_stride_dim = rope ? rope_strides[1] : 0;
  prm.rope_stride_rot = rope ? rope_strides[2] : 0; prm.rope_stride_pair = rope ? rope_strides[3] : 0;
  prm.heads = heads; prm.epsilon = epsilon; prm.norm_dtype = norm_dtype;
  prm.wait_budget_ns = wait_budget_ns();
  prm.q8 = prm.k8 = nullptr; prm.q_scale = prm.k_scale = nullptr; prm.q_summary = prm.k_summary = nullptr;
  prm.k_stage = prm.v_stage = nullptr; prm.k_sum = nullptr; prm.v_amax_bits = nullptr;
  prm.summary_dtype = H3S_F32; prm.sequence_total = rows; prm.row_start = 0;
  prm.operand_kind = H3S_GEMM_I8; prm.row_scale = nullptr; prm.col_scale = nullptr; prm.bias = nullptr;
  prm.activation = H3S_ACT_NONE; prm.tile_n = kGemmN; prm.vector_columns = false; prm.dense_out = nullptr; prm.ldc = 0;
  if (carriers != nullptr) {
    const h3s_qkv_carriers &c = *carriers;
    prm.q8 = c.q8; prm.k8 = c.k8; prm.q_scale = c.q_scale; prm.k_scale = c.k_scale;
    prm.q_summary = c.q_summary; prm.k_summary = c.k_summary;
    prm.k_stage = static_cast<__nv_bfloat16 *>(c.k_stage); prm.v_stage = static_cast<__nv_bfloat16 *>(c.v_stage);
    // statistics scratch: double k_sum[heads*128]; uint32 v_amax_bits[heads*128] (the layout of h3s_column_stats)
    double *sums = static_cast<double *>(c.stats);
    prm.k_sum = c.k_stage != nullptr ? sums : nullptr;
    prm.v_amax_bits = reinterpret_cast<unsigned int *>(sums + heads * H3S_HEAD_DIM);
    prm.summary_dtype = c.summary_dtype; prm.sequence_total = c.sequence_total; prm.row_start = c.row_start;
  }
  int device = 0, sms = 0;
  H3S_CHECK_CUDA(cudaGetDevice(&device));
  H3S_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const int tiles = prm.m_pairs * prm.n_tiles;
  const int grid = 2 * (tiles < sms / 2 ? tiles : sms / 2);
  if (carriers != nullptr) {
    H3S_CHECK_CUDA(cudaFuncSetAttribute(qkv_gemm_kernel<kModeCarriers>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(GemmLayout<kModeCarriers>::kBytes)));
    // Not `launch_next`: its blocks would take SMs one by one from the rotation of the rows that stands before it, whose last
    // blocks share an SM four at a time (attention block of 33272 tokens 4995 us so, 4935 behind the complete rotation).
    qkv_gemm_kernel<kModeCarriers><<<grid, GemmWarps<kModeCarriers>::kThreads, GemmLayout<kModeCarriers>::kBytes, static_cast<cudaStream_t>(stream)>>>(ma, mb, prm);
    H3S_CHECK_CUDA(cudaGetLastError());
  } else {
    H3S_CHECK_CUDA(cudaFuncSetAttribute(qkv_gemm_kernel<kModeStaging>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(GemmLayout<kModeStaging>::kBytes)));
    H3S_CHECK_CUDA(launch_next(qkv_gemm_kernel<kModeStaging>, grid, GemmWarps<kModeStaging>::kThreads, GemmLayout<kModeStaging>::kBytes,
                               static_cast<cudaStream_t>(stream), ma, mb, prm));
  }
  return H3S_OK;
}

int h3s_qkv_gemm_chunk(const int8_t *x_i8, const float *x_scale, const int8_t *w_i8, const float *w_scale,
                       int rows, int hidden, int n_out, void *out_bf16, int64_t out_stride_head,
                       int32_t *status, h3s_stream_t stream) {
  return qkv_gemm_chunk_impl(x_i8, x_scale, w_i8, w_scale, rows, hidden, n_out, out_bf16, out_stride_head, nullptr,
                             nullptr, 0.f, nullptr, H3S_F32, nullptr, 0, status, stream, "qkv_gemm_chunk");
}

int h3s_qkv_gemm_chunk_norm_rope(const int8_t *x_i8, const float *x_scale, const int8_t *w_i8,
                                 const float *w_scale, int rows, int hidden, int heads, void *out_bf16,
                                 int64_t out_stride_head, const float *q_norm, const float *k_norm,
                                 float epsilon, const void *rope, int rope_dtype, const int64_t *rope_strides,
                                 int32_t *status, h3s_stream_t stream) {
  H3S_CHECK_ARG(q_norm != nullptr && k_norm != nullptr, "qkv_gemm_chunk_norm_rope: NULL norm weight");
  return qkv_gemm_chunk_impl(x_i8, x_scale, w_i8, w_scale, rows, hidden, 3 * heads * H3S_HEAD_DIM, out_bf16,
                             out_stride_head, q_norm, k_norm, epsilon, rope, rope_dtype, rope_strides, heads, status,
                             stream, "qkv_gemm_chunk_norm_rope");
}

// Columns of a dense tile.  Every pair of SMs takes as long as the most tiles that one of them gets, a round of tiles; narrower
// tiles may need no more rounds, or make up for one more.  A tile's time goes with its columns and a part that does not: per step of
// K its 128 rows of A are loaded whatever the width (96 bytes a clock and SM with 128 columns, 64 with 256), and what the MMAs leave
// idle the SM clock makes up for, as the power allows.  96 columns' worth of such time is where the line fits 52 shapes; the rule's
// choice is the fastest width of each or within 4 % of it.  us, 256 columns / the rule's, launches in a row:
//   fp8    64 x 3072 x 12288 32.7 / 17.6 (64), 300 x 3072 x 12288 33.7 / 19.8 (96), 700 x 3072 x 12288 34.0 / 23.8 (128), 1000 x 3072 x 12288
//          38.0 / 30.5 (192), 1000 x 12288 x 3072 34.2 / 31.3 (224), 2000 x 3072 x 12288 80.6 / 66.1 (192), 1500 x 3072 x 12288 42.2 (256)
//   bf16   64 x 1024 x 1024 10.0 / 6.9 (64), 900 x 3072 x 3072 21.2 / 17.4 (192), 2304 x 3072 x 3072 35.3 / 30.4 (192), 8000 x 3072 x 3072
//          128.5 / 120.9 (192), 33272 x 3072 x 3072 462.3 (256; 224: 477, 128: 603)
// Where A is all but nothing (up to 20 rows of 6 KB, 8 of 12 KB) every CTA waits for the same few lines of it at the same time, and 32 tiles
// and more beside one another take longer than 24.  us, 256 columns / as many as leave 24 tiles / 64: fp8 1 x 3072 x 12288 32.6 / 26.9
// (128) / 38.4, 8 rows 32.6 / 25.2 / 39.3, 12 rows 32.6 / 18.9 / 17.5; bf16 1 x 3072 x 3072 19.2 / 17.0 (128) / 23.2, 20 rows 19.2 / 13.8 / 21.2,
// 24 rows 19.2 / 12.0 / 11.3; 1 x 4096 x 1024 10.3 / 10.3 (192) / 11.9, 48 rows 10.3 / 9.4 / 10.3, 64 rows 10.3 / 9.0 / 7.5; 1 x 2048 x 2048
// 14.7 / 14.2 (96) / 16.3, 24 rows 14.7 / 11.4 / 13.4, 32 rows 14.7 / 9.3 / 9.0; with 264 columns 64 are the fastest throughout.
int h3s_dense_gemm_columns(int rows, int n_out, int k_bytes, int sms) {
  constexpr int kStep = 32, kLeast = 64, kFixed = 96, kTilesOfLittle = 24;
  constexpr int64_t kLittle = 128 * 1024;  // bytes of A that a row of tiles reads
  const int m_pairs = h3s::ceil_div(rows, h3s::kGemmPairM), pairs_of_sms = sms < 2 ? 1 : sms / 2;
  const bool little = static_cast<int64_t>(rows < h3s::kGemmPairM ? rows : h3s::kGemmPairM) * k_bytes < kLittle;
  int best = h3s::kGemmN;
  int64_t best_cost = 0;
  for (int width = h3s::kGemmN; width >= kLeast; width -= kStep) {
    const int columns = h3s::ceil_div(n_out, width);
    if (little && columns > kTilesOfLittle) break;
    const int64_t tiles = static_cast<int64_t>(m_pairs) * columns;
    const int64_t cost = (tiles + pairs_of_sms - 1) / pairs_of_sms * (kFixed + width);
    if (best_cost == 0 || cost < best_cost) { best = width; best_cost = cost; }
  }
  return best;
}

int h3s_dense_gemm(const void *a, int64_t lda_bytes, const void *b, int64_t ldb_bytes, int operand_kind, int rows,
                   int n_out, int k_bytes, const float *row_scale, const float *col_scale, const float *bias,
                   int activation, void *out_bf16, int64_t ldc, int32_t *status, h3s_stream_t stream) {
  using namespace h3s;
  H3S_CHECK_ARG(a != nullptr && b != nullptr && out_bf16 != nullptr, "dense_gemm: NULL pointer");
  H3S_CHECK_ARG(operand_kind >= H3S_GEMM_I8 && operand_kind <= H3S_GEMM_E4M3, "dense_gemm: unknown operand kind %d", operand_kind);
  H3S_CHECK_ARG(activation == H3S_ACT_NONE || activation == H3S_ACT_GELU_TANH, "dense_gemm: unknown activation %d", activation);
  H3S_CHECK_ARG(rows > 0 && n_out > 0 && n_out % 8 == 0, "dense_gemm: rows %d, n_out %d (a positive multiple of 8)", rows, n_out);
  H3S_CHECK_ARG(k_bytes > 0 && k_bytes % kGemmK == 0, "dense_gemm: the reduction length %d bytes must be a positive multiple of 128", k_bytes);
  H3S_CHECK_ARG(lda_bytes >= k_bytes && ldb_bytes >= k_bytes && lda_bytes % 16 == 0 && ldb_bytes % 16 == 0,
                "dense_gemm: operand row strides must be multiples of 16 bytes and cover the reduction length");
  H3S_CHECK_ARG(ldc >= n_out && ldc % 8 == 0, "dense_gemm: ldc %lld must be a multiple of 8 and at least n_out", static_cast<long long>(ldc));
  H3S_CHECK_ARG(((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(out_bf16)) & 15) == 0,
                "dense_gemm: operands and output must be 16-byte aligned");
  const int cap = h3s_device_capability();
  if (cap < 0) return cap;
  if (cap / 10 != 10) return fail(H3S_EARCH, "dense_gemm: needs an sm_100 device, found sm_%d", cap);
  CUtensorMap ma, mb;
  int rc = make_tensor_map_u8_2d(&ma, a, k_bytes, rows, lda_bytes, kGemmK, kGemmM, "dense_gemm A map");
  if (rc) return rc;
  int device = 0, sms = 0;
  H3S_CHECK_CUDA(cudaGetDevice(&device));
  H3S_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const int tile_n = h3s_dense_gemm_columns(rows, n_out, k_bytes, sms);
  rc = make_tensor_map_u8_2d(&mb, b, k_bytes, n_out, ldb_bytes, kGemmK, tile_n / 2, "dense_gemm B map");
  if (rc) return rc;
  GemmParams prm;
  memset(&prm, 0, sizeof(prm));
  prm.x_scale = row_scale; prm.status = status;
  prm.rows = rows; prm.n_out = n_out; prm.hidden = k_bytes;
  prm.m_pairs = ceil_div(rows, kGemmPairM); prm.n_tiles = ceil_div(n_out, tile_n); prm.tile_n = tile_n;
  prm.heads = 1; prm.wait_budget_ns = wait_budget_ns();
  prm.operand_kind = operand_kind; prm.row_scale = row_scale; prm.col_scale = col_scale; prm.bias = bias;
  prm.vector_columns = ((reinterpret_cast<uintptr_t>(col_scale) | reinterpret_cast<uintptr_t>(bias)) & 15) == 0;
  prm.activation = activation; prm.dense_out = static_cast<__nv_bfloat16 *>(out_bf16); prm.ldc = ldc;
  H3S_CHECK_CUDA(cudaFuncSetAttribute(qkv_gemm_kernel<kModeDense>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(GemmLayout<kModeDense>::kBytes)));
  const int tiles = prm.m_pairs * prm.n_tiles;
  H3S_CHECK_CUDA(launch_next(qkv_gemm_kernel<kModeDense>, 2 * (tiles < sms / 2 ? tiles : sms / 2), GemmWarps<kModeDense>::kThreads,
                             GemmLayout<kModeDense>::kBytes, static_cast<cudaStream_t>(stream), ma, mb, prm));
  return H3S_OK;
}

int h3s_qkv_gemm_chunk_carriers(const int8_t *x_i8, const float *x_scale, const int8_t *w_i8,
                                const float *w_scale, int rows, int hidden, int heads,
                                const h3s_qkv_carriers *carriers, const float *q_norm, const float *k_norm,
                                float epsilon, const void *rope, int rope_dtype, const int64_t *rope_strides,
                                int32_t *status, h3s_stream_t stream) {
  return h3s::qkv_gemm_carriers(x_i8, x_scale, w_i8, w_scale, rows, hidden, heads, carriers, q_norm, k_norm, H3S_F32, epsilon, rope,
                                rope_dtype, rope_strides, status, stream);
}

}  // extern "C"

int h3s::qkv_gemm_carriers(const int8_t *x_i8, const float *x_scale, const int8_t *w_i8, const float *w_scale, int rows, int hidden,
                           int heads, const h3s_qkv_carriers *carriers, const void *q_norm, const void *k_norm, int norm_dtype,
                           float epsilon, const void *rope, int rope_dtype, const int64_t *rope_strides, int32_t *status,
                           h3s_stream_t stream) {
  H3S_CHECK_ARG(carriers != nullptr, "qkv_gemm_chunk_carriers: NULL carrier description");
  return qkv_gemm_chunk_impl(x_i8, x_scale, w_i8, w_scale, rows, hidden, 3 * heads * H3S_HEAD_DIM, nullptr, 0,
                             static_cast<const float *>(q_norm), static_cast<const float *>(k_norm), epsilon, rope, rope_dtype,
                             rope_strides, heads, status, stream, "qkv_gemm_chunk_carriers", carriers, norm_dtype);
}
