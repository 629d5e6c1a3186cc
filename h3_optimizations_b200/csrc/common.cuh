// Shared host/device helpers for the h3sparse kernels (sm_100a only).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/h3sparse.h"

namespace h3s {

// Records the message returned by h3s_last_error() and returns `code`.
int fail(int code, const char *fmt, ...);

#define H3S_CHECK_ARG(cond, ...)                          \
  do {                                                    \
    if (!(cond)) return ::h3s::fail(H3S_EINVAL, __VA_ARGS__); \
  } while (0)

// The error is reported here, so the runtime's note of it goes too: a later cudaGetLastError() would take it for that of a
// launch of its own.
#define H3S_CHECK_CUDA(expr)                                                   \
  do {                                                                         \
    cudaError_t err__ = (expr);                                                \
    if (err__ != cudaSuccess) {                                                \
      (void)cudaGetLastError();                                                \
      return ::h3s::fail(H3S_ECUDA, "%s failed: %s", #expr,                    \
                         cudaGetErrorString(err__));                           \
    }                                                                          \
  } while (0)

// Upper bound of every device-side wait of the kernels launched from now on
// (h3s_set_wait_budget_ns).
unsigned long long wait_budget_ns();

// h3s_qkv_gemm_chunk_carriers with norm weights of `norm_dtype`, fp32 or bf16 (qkv_gemm.cu)
int qkv_gemm_carriers(const int8_t *x_i8, const float *x_scale, const int8_t *w_i8, const float *w_scale, int rows, int hidden,
                      int heads, const h3s_qkv_carriers *carriers, const void *q_norm, const void *k_norm, int norm_dtype,
                      float epsilon, const void *rope, int rope_dtype, const int64_t *rope_strides, int32_t *status,
                      h3s_stream_t stream);

// K (with smooth_k) and V of the projection from their staging and the totals in `c->scratch`
int staged_carriers(const h3s_layer_carriers *c, const void *k_stage, const void *v_stage, int heads, int sequence, bool smooth_k,
                    float v_bound, cudaStream_t stream);
// h3s_convrot_quant_rows, whose first launch of a call may also clear `words` 32-bit words
int convrot_quant_rows(const void *x, int64_t x_stride_row, int rows, int hidden, int8_t *x_i8, float *x_scale, uint32_t *clear, int words,
                       cudaStream_t stream);

constexpr int kSmCount = 148;  // of a B200, for the rules that deal out work

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// ---- launches that follow one another in a stream ----
//
// A kernel launched with `launch_next` may start while the kernel before it is still running: its blocks come as SMs get
// free, set themselves up and stop at `wait_for_previous` until that kernel is complete and its writes are seen.  So every
// thread of such a kernel calls it before it touches global memory, reads and writes alike; then a kernel is complete only
// after all those before it are, whatever their kind.  `let_next_start` tells that this block does not mind; it stands at the
// top, as the next kernel's blocks are only placed once every block of this one has been.  What is saved is the gap between
// two kernels and the set-up of the second.  us, the same kernels launched without / with it, in turn: MLP of 1000 x 3072 x 12288 (four
// kernels) 102 / 94, of 33272 rows (36) 2612 / 2567, of 33130 x 1024 x 4096 623 / 558; layer of 7 heads x 10384 tokens 133 / 131, of
// 24 x 33272 alike.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What an earlier kernel may have written is read by this, by `load_if`, through `written_before` or by TMA.  `__ldg`, and a load through
// a `const __restrict__` parameter, tell the compiler that the memory does not change while the kernel runs, which begins before the
// wait: it had moved the loads of the V quantiser's scales above it (long fp32 layers at full density were quantised by the scales of an
// earlier call; waiting costs those kernels 0.3 to 1 us).  An ordinary load that is volatile stays behind the wait.  Where `__ldg` is
// left, in the roles of a kernel behind barriers and loops, there is no way up.
template <typename T>
__device__ __forceinline__ T load_written(const T *p) {
  static_assert(sizeof(T) == 2 || sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) == 16, "one load");
  T value;
  if constexpr (sizeof(T) == 2) {
    asm volatile("ld.global.b16 %0, [%1];" : "=h"(reinterpret_cast<unsigned short &>(value)) : "l"(p));
  } else if constexpr (sizeof(T) == 4) {
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(reinterpret_cast<unsigned int &>(value)) : "l"(p));
  } else if constexpr (sizeof(T) == 8) {
    asm volatile("ld.global.b64 %0, [%1];" : "=l"(reinterpret_cast<unsigned long long &>(value)) : "l"(p));
  } else {
    uint4 &v = reinterpret_cast<uint4 &>(value);
    asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  }
  return value;
}

// A pointer of which nothing is known but that it comes from behind the wait: ordinary loads through it stay there too, in any order among
// themselves (router 24 x 16 rows of 32 scores 5.2 us, 5.7 with volatile loads; 3 x 256 of 512 21.1 and 22.1).
template <typename T>
__device__ __forceinline__ T *written_before(T *p) {
  asm volatile("" : "+l"(p) : : "memory");
  return p;
}

template <typename... Params, typename... Args>
inline cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, dim3 block, size_t shared_bytes, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = shared_bytes;
  config.stream = stream;
  config.attrs = &attribute;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);
}

// ---- element loads: 8 consecutive channels of one row, widened to fp32 ----

// 16 bytes, or zeros.  Volatile: where a block asks for many rows before it uses the first, the compiler must not move the loads to
// their uses.  us, statistics, Q, K and V of a layer on two streams, without / with it: 24 heads x 33272 tokens 288 / 269, fp32 464 / 427,
// 24 x 9872 95 / 90, 3 x 33272 59 / 47, 7 x 10384 51 / 38, 24 x 2304 46 / 32, 4 x 2304 fp32 28 / 21.
__device__ __forceinline__ uint4 load_if(const void *p, bool valid) {
  uint4 v;
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "mov.b32 %0, 0;\n\t"
      "mov.b32 %1, 0;\n\t"
      "mov.b32 %2, 0;\n\t"
      "mov.b32 %3, 0;\n\t"
      "@q ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n\t"
      "}\n"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
      : "l"(p), "r"(static_cast<int>(valid)));
  return v;
}

template <typename T>
struct Elem;

template <>
struct Elem<float> {
  static constexpr int kDtype = H3S_F32;
  struct Raw { float4 a, b; };  // 8 elements as loaded
  __device__ static Raw load_raw(const float *p) {
    Raw r;
    r.a = load_written(reinterpret_cast<const float4 *>(p));
    r.b = load_written(reinterpret_cast<const float4 *>(p) + 1);
    return r;
  }
  __device__ static Raw load_raw_if(const float *p, bool valid) {
    const uint4 a = load_if(p, valid), b = load_if(p + 4, valid);
    Raw r;
    r.a = make_float4(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w));
    r.b = make_float4(__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z), __uint_as_float(b.w));
    return r;
  }
  __device__ static Raw zero_raw() { Raw r; r.a = make_float4(0.f, 0.f, 0.f, 0.f); r.b = r.a; return r; }
  __device__ static void unpack(const Raw &r, float (&v)[8]) {
    v[0] = r.a.x; v[1] = r.a.y; v[2] = r.a.z; v[3] = r.a.w;
    v[4] = r.b.x; v[5] = r.b.y; v[6] = r.b.z; v[7] = r.b.w;
  }
  __device__ static void load8(const float *p, float (&v)[8]) { unpack(load_raw(p), v); }
  __device__ static float round_trip(float x) { return x; }
};

template <>
struct Elem<__nv_bfloat16> {
  static constexpr int kDtype = H3S_BF16;
  typedef uint4 Raw;  // 8 elements as loaded
  __device__ static Raw load_raw(const __nv_bfloat16 *p) { return load_written(reinterpret_cast<const uint4 *>(p)); }
  __device__ static Raw load_raw_if(const __nv_bfloat16 *p, bool valid) { return load_if(p, valid); }
  __device__ static Raw zero_raw() { return make_uint4(0u, 0u, 0u, 0u); }
  __device__ static void load8(const __nv_bfloat16 *p, float (&v)[8]) { unpack(load_raw(p), v); }
  __device__ static void unpack(const Raw &raw, float (&v)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  __device__ static float round_trip(float x) {
    return __bfloat162float(__float2bfloat16_rn(x));
  }
};

template <>
struct Elem<__half> {
  static constexpr int kDtype = H3S_F16;
  typedef uint4 Raw;  // 8 elements as loaded
  __device__ static Raw load_raw(const __half *p) { return load_written(reinterpret_cast<const uint4 *>(p)); }
  __device__ static Raw load_raw_if(const __half *p, bool valid) { return load_if(p, valid); }
  __device__ static Raw zero_raw() { return make_uint4(0u, 0u, 0u, 0u); }
  __device__ static void load8(const __half *p, float (&v)[8]) { unpack(load_raw(p), v); }
  __device__ static void unpack(const Raw &raw, float (&v)[8]) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&raw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(h[i]);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
    }
  }
  __device__ static float round_trip(float x) {
    return __half2float(__float2half_rn(x));
  }
};

// Packed fp32x2 arithmetic: one instruction for the two halves of a 64-bit register pair, each
// rounded as by itself.  The quantisers are bound by the instructions they issue (K of 24
// heads x 33272 tokens 75 -> 70 us); the GEMM epilogues, bound by latency, gain 1 to 3 %.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long &>(d))
      : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)),
        "l"(reinterpret_cast<unsigned long long &>(c)));
  return d;
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long &>(d))
      : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
  return d;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long &>(d))
      : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
  return d;
}

// the two bf16 of a word
__device__ __forceinline__ float2 bf16_pair(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// Correctly rounded a/b for many a and one b: with r = RN(1/b),
//   q0 = RN(a*r), e = a - b*q0 (exact in an FMA), q = RN(q0 + e*r)
// equals RN(a/b) (Markstein) unless b's significand is all ones, where RN(1/b)
// is not accurate enough; `exact` is false there and the IEEE divide is used.
struct SharedDivisor {
  float b, r;
  bool exact;
};

__device__ __forceinline__ SharedDivisor make_divisor(float divisor) {
  SharedDivisor d;
  d.b = divisor;
  d.r = __frcp_rn(divisor);
  d.exact = (__float_as_uint(divisor) & 0x007fffffu) != 0x007fffffu && fabsf(divisor) > 1.0e-30f &&
            fabsf(divisor) < 1.0e30f;
  return d;
}

// kExact is d.exact, tested ONCE by the caller around its whole element loop: with the
// test inside `divide` the compiler keeps the IEEE division sequence in the loop body
// next to the three-instruction path, which made the quantisers several times slower.
template <bool kExact>
__device__ __forceinline__ float divide(const SharedDivisor &d, float a) {
  if (!kExact) return __fdiv_rn(a, d.b);
  const float q0 = __fmul_rn(a, d.r);
  const float e = __fmaf_rn(-d.b, q0, a);
  return __fmaf_rn(e, d.r, q0);
}

template <bool kExact>
__device__ __forceinline__ float2 divide2(const SharedDivisor &d, float2 a) {
  if (!kExact) return make_float2(__fdiv_rn(a.x, d.b), __fdiv_rn(a.y, d.b));
  const float2 r = make_float2(d.r, d.r), minus_b = make_float2(-d.b, -d.b);
  const float2 q0 = mul2(a, r);
  return fma2(fma2(minus_b, q0, a), r, q0);
}

// trunc(q +- 0.5), the half with q's sign
__device__ __forceinline__ void round_codes(float2 q, uint32_t &first, uint32_t &second) {
  const float2 half = make_float2(__uint_as_float((__float_as_uint(q.x) & 0x80000000u) | 0x3f000000u),
                                  __uint_as_float((__float_as_uint(q.y) & 0x80000000u) | 0x3f000000u));
  q = add2(q, half);
  first = static_cast<uint32_t>(static_cast<int>(q.x));
  second = static_cast<uint32_t>(static_cast<int>(q.y));
}

// 8 E4M3 codes -> the same values as FP16 (exact: four significant bits, 2^-9 to 448)
__device__ __forceinline__ uint4 e4m3x8_to_half(const uint2 &codes) {
  const uint32_t in[2] = {codes.x, codes.y};
  uint32_t pair[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(pair[k]) : "h"(static_cast<uint16_t>(in[k >> 1] >> ((k & 1) * 16))));
  return make_uint4(pair[0], pair[1], pair[2], pair[3]);
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace h3s
