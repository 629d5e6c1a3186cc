// What the two tcgen05 attention kernels share: launch parameters, status codes, bounded waits
// and the output stores.
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace h3s {

// A code names one kind of wait; backend.py and h3sparse.h have their texts
enum AbortCode {
  kAbortQFull = 1, kAbortKvFull, kAbortKvEmpty, kAbortSFull, kAbortPFull, kAbortScoreSlot,
  kAbortPvDone, kAbortFinal, kAbortQFree, kAbortNextItem, kAbortPass, kAbortOFree, kAbortFirstMax, kAbortStaged,
  kAbortStatistics
};

// The words of the first launch that gives up, and their copy in pinned host memory (either may be null); one thread
__device__ __forceinline__ void report_status(int32_t *status, int32_t *status_mirror, int code, int number, int head, int tile) {
  if (status == nullptr || atomicCAS(status, 0, code) != 0) return;
  status[1] = number;
  status[2] = head;
  status[3] = tile;
  if (status_mirror == nullptr) return;
  volatile int32_t *mirror = status_mirror;
  mirror[1] = number;
  mirror[2] = head;
  mirror[3] = tile;
  __threadfence_system();
  mirror[0] = code;
}

constexpr float kIntBias = 12582912.0f;  // 1.5 * 2^23: float(kIntBias + s) has bits 0x4b400000 + s
constexpr uint32_t kIntBiasBits = 0x4b400000u;

struct AttnParams {
  const float *q_scale;
  const float *k_scale;
  const float *v_scale;
  const int32_t *route;  // (heads, q_stop-q_start, route_len) or null
  void *out;
  int32_t *status;
  int32_t *status_mirror;  // pinned host memory that gets the words too, or null (attn_half.cu)
  int64_t out_stride_h, out_stride_s;
  int route_len, q_start, q_stop;
  // A dense row's tile list may be cut into `parts` even parts, an item each (attn_half.cu); 1: not cut.  partial: per dense row and part 128 x 128 sums of P.V, 128 row sums and 128 reference points;
  // arrived: per dense row the number of parts that are in, zero at launch.
  int parts;
  float *partial;
  unsigned int *arrived;
  int heads, sequence, q_tiles, kv_tiles;
  int out_dtype;
  bool out_map;  // the output may go, and in attn_half.cu does go, through TMA stores
  // head-sharded runs: every output tile is also stored into these buffers
  // (the same slice of each peer GPU's full output, reached over NVLink with
  // plain stores), so no separate gather pass is needed
  void *peer_out[H3S_MAX_PEER_OUTPUTS];
  int n_peer_out;
  // Bound of the waits for TMA loads; a wait further down the pipeline (QK^T
  // result 2x, P 3x, P.V and free stages 4x) gets a multiple, so that when a
  // stage stalls the wait closest to the cause is the one that runs out first
  // and names it in the status words.
  unsigned long long wait_budget_ns;
  // self-test of the bounded waits (H3S_ATTN_TEST_DROP_KV_LOAD): the producer
  // never issues the K/V load of this iteration, so the wait for it runs out
  int drop_kv_load;                   // iteration index, -1 = none
  bool drop_last_v_load;              // H3S_ATTN_TEST_DROP_LAST_V_LOAD: that of every item's last tile (attn_half.cu)
};

// 1: `out` is memory of this device; 0: other memory that the device can write to (pinned host memory, managed
// memory, a peer's), which keeps plain stores; else a status (attn_tc.cu)
int output_home(const void *out, const char *who);

// Checks the arguments of an attention launch and fills `params` (attn_tc.cu).  `v` is the V
// carrier the kernel reads, E4M3 or its FP16 copy.
int fill_attn_params(AttnParams *params, const int8_t *q8, const int8_t *k8, const void *v, const float *q_scale,
                     const float *k_scale, const float *v_scale, const int32_t *route, int route_len, int q_start,
                     int q_stop, void *out, void *const *peer_out, int n_peer_out, int out_dtype, int64_t out_stride_h,
                     int64_t out_stride_s, int heads, int sequence, int flags, int32_t *status, const char *who);

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Every lane polls the barrier; the warp then agrees on the outcome so that
// the .sync.aligned tcgen05 instructions that follow stay convergent even if
// the abort word was raised between two lanes' polls.
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_word, int code,
                                          unsigned long long budget_ns) {
  if (__all_sync(0xffffffffu, ptx::mbar_test_wait(bar, parity))) return true;  // the usual case, kept short
  const bool ok = ptx::mbar_wait(bar, parity, abort_word, code, budget_ns);
  return __all_sync(0xffffffffu, ok);
}

template <typename OutT> __device__ __forceinline__ void store_out8(OutT *dst, const float (&v)[8]);
template <> __device__ __forceinline__ void store_out8<float>(float *dst, const float (&v)[8]) {
  reinterpret_cast<float4 *>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4 *>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
template <> __device__ __forceinline__ void store_out8<__nv_bfloat16>(__nv_bfloat16 *dst, const float (&v)[8]) {
  uint4 w;
  __nv_bfloat162 t;
  t = __floats2bfloat162_rn(v[0], v[1]); w.x = *reinterpret_cast<uint32_t *>(&t);
  t = __floats2bfloat162_rn(v[2], v[3]); w.y = *reinterpret_cast<uint32_t *>(&t);
  t = __floats2bfloat162_rn(v[4], v[5]); w.z = *reinterpret_cast<uint32_t *>(&t);
  t = __floats2bfloat162_rn(v[6], v[7]); w.w = *reinterpret_cast<uint32_t *>(&t);
  *reinterpret_cast<uint4 *>(dst) = w;
}
template <> __device__ __forceinline__ void store_out8<__half>(__half *dst, const float (&v)[8]) {
  uint4 w;
  __half2 t;
  t = __floats2half2_rn(v[0], v[1]); w.x = *reinterpret_cast<uint32_t *>(&t);
  t = __floats2half2_rn(v[2], v[3]); w.y = *reinterpret_cast<uint32_t *>(&t);
  t = __floats2half2_rn(v[4], v[5]); w.z = *reinterpret_cast<uint32_t *>(&t);
  t = __floats2half2_rn(v[6], v[7]); w.w = *reinterpret_cast<uint32_t *>(&t);
  *reinterpret_cast<uint4 *>(dst) = w;
}

// Copies the finished tile, staged in shared memory (row r at r*kRowBytes, 16-byte
// chunk c at chunk position c ^ (r & 15)), to the same slice of every peer GPU's
// output with plain stores over NVLink.  The whole CTA shares the copy, and each
// 16-byte chunk is sent to all peers back to back, so that the stores of one CTA
// are spread over every link at once instead of filling one destination after
// the other.
template <typename OutT>
__device__ __forceinline__ void scatter_to_peers(const AttnParams &prm, const unsigned char *stage, int head, int tq,
                                                 int threads) {
  constexpr int kRowBytes = H3S_HEAD_DIM * static_cast<int>(sizeof(OutT));
  constexpr int kChunksPerRow = kRowBytes / 16;
  const int64_t tile_offset = head * prm.out_stride_h * static_cast<int64_t>(sizeof(OutT));
  for (int idx = threadIdx.x; idx < H3S_Q_TILE * kChunksPerRow; idx += threads) {
    const int r = idx / kChunksPerRow, c = idx % kChunksPerRow;
    const int grow = tq * H3S_Q_TILE + r;
    if (grow < prm.sequence) {
      const uint4 value = *reinterpret_cast<const uint4 *>(stage + r * kRowBytes + ((c ^ (r & 15)) << 4));
      const int64_t at = tile_offset + static_cast<int64_t>(grow) * prm.out_stride_s * static_cast<int64_t>(sizeof(OutT)) + c * 16;
#pragma unroll
      for (int d = 0; d < H3S_MAX_PEER_OUTPUTS; ++d)
        if (d < prm.n_peer_out) *reinterpret_cast<uint4 *>(static_cast<unsigned char *>(prm.peer_out[d]) + at) = value;
    }
  }
}

// One warp writes `rows` rows of the staged tile, from `row0` on, as full contiguous lines.
template <typename OutT>
__device__ __forceinline__ void store_rows(const AttnParams &prm, const unsigned char *stage, int head, int tq,
                                           int row0, int rows, int lane) {
  constexpr int kRowBytes = H3S_HEAD_DIM * static_cast<int>(sizeof(OutT));
  constexpr int kChunksPerRow = kRowBytes / 16;
  unsigned char *base = static_cast<unsigned char *>(prm.out);
#pragma unroll 4
  for (int idx = lane; idx < rows * kChunksPerRow; idx += 32) {
    const int r = row0 + idx / kChunksPerRow, c = idx % kChunksPerRow;
    const int grow = tq * H3S_Q_TILE + r;
    if (grow < prm.sequence) {
      const uint4 value = *reinterpret_cast<const uint4 *>(stage + r * kRowBytes + ((c ^ (r & 15)) << 4));
      unsigned char *dst = base + (head * prm.out_stride_h + static_cast<int64_t>(grow) * prm.out_stride_s) *
                                      static_cast<int64_t>(sizeof(OutT)) + c * 16;
      *reinterpret_cast<uint4 *>(dst) = value;
    }
  }
}

}  // namespace h3s
