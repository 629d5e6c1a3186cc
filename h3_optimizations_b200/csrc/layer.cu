// Launch sequences of a whole layer call.  Nothing here runs on the GPU by itself: these
// calls issue the kernels of the other files in order, on the caller's two streams, so that
// a host in Python pays for one foreign call instead of ten to thirty.
//
// What it measured: host time bounds every call of up to about 10000 tokens and 8 heads; see
// the figures at B200SparseBackend.prepare and run_chunked_sparse_qkv, which call them.
#include <mutex>

#include "common.cuh"

namespace h3s {

// A recorded event is overwritten by the next record, so "record on one stream, wait on the
// other" has to be one step when several threads share a pair of streams and its events.
static std::mutex g_order_mutex;

static int order_after(cudaStream_t first, cudaStream_t then, void *event) {
  std::lock_guard<std::mutex> lock(g_order_mutex);
  H3S_CHECK_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(event), first));
  H3S_CHECK_CUDA(cudaStreamWaitEvent(then, static_cast<cudaEvent_t>(event), 0));
  return H3S_OK;
}

constexpr int64_t kStagedOneLaunchRows = 100000;

}  // namespace h3s

extern "C" {

int h3s_stream_order(h3s_stream_t first, h3s_stream_t then, void *event) {
  H3S_CHECK_ARG(event != nullptr, "stream_order: NULL event");
  return h3s::order_after(static_cast<cudaStream_t>(first), static_cast<cudaStream_t>(then), event);
}

int h3s_quant_qkv(const h3s_layer_carriers *c, const void *q, const void *k, const void *v, const int64_t *strides,
                  int dtype, int heads, int sequence, int smooth_k, float v_bound, int v_after_k, void *event,
                  h3s_stream_t stream, h3s_stream_t side_stream) {
  using namespace h3s;
  const bool forked = side_stream != stream;  // else one stream does it all, in the same order
  H3S_CHECK_ARG(c != nullptr && strides != nullptr && (event != nullptr || !forked), "quant_qkv: NULL argument");
  H3S_CHECK_ARG(q != nullptr && k != nullptr && v != nullptr, "quant_qkv: NULL input");
  cudaStream_t s = static_cast<cudaStream_t>(stream), side = static_cast<cudaStream_t>(side_stream);
  const float *mean = smooth_k ? c->k_mean : nullptr;
  int rc = forked ? order_after(s, side, event) : H3S_OK;
  if (rc) return rc;
  rc = h3s_column_stats(smooth_k ? k : nullptr, strides[2], strides[3], v, strides[4], strides[5], dtype, heads,
                        sequence, v_bound, smooth_k ? c->k_mean : nullptr, c->v_scale, c->scratch, side);
  if (rc) return rc;
  // Q needs no statistics and runs beside them; K joins when they are in
  rc = h3s_quant_qk_blocks(q, dtype, strides[0], strides[1], nullptr, c->q8, c->q_scale, c->q_summary,
                           c->summary_dtype, heads, sequence, 0, sequence, H3S_Q_TILE, s);
  if (rc) return rc;
  rc = forked ? order_after(side, s, event) : H3S_OK;
  if (rc) return rc;
  rc = h3s_quant_qk_blocks(k, dtype, strides[2], strides[3], mean, c->k8, c->k_scale, c->k_summary, c->summary_dtype,
                           heads, sequence, 0, sequence, H3S_KV_TILE, s);
  if (rc) return rc;
  if (v_after_k && forked) {
    rc = order_after(s, side, event);
    if (rc) return rc;
  }
  return h3s_quant_v_fp8_half(v, dtype, strides[4], strides[5], c->v_scale, c->v8, c->v16, heads, sequence, 0, sequence,
                              v_bound, side);
}

int h3s_project_qkv_norms(const h3s_layer_carriers *c, const void *x_bf16, int64_t x_stride_row, int sequence, int hidden,
                          int chunk_rows, int8_t *x_i8, float *x_scale, const int8_t *w_i8, const float *w_scale, int heads,
                          int smooth_k, void *k_stage, void *v_stage, const void *q_norm, const void *k_norm,
                          int norm_dtype, float epsilon, const void *rope, int rope_dtype, const int64_t *rope_strides, float v_bound,
                          int32_t *status, void *event, h3s_stream_t stream, h3s_stream_t side_stream) {
  using namespace h3s;
  H3S_CHECK_ARG(c != nullptr && event != nullptr, "project_qkv: NULL argument");
  H3S_CHECK_ARG(x_bf16 != nullptr && x_i8 != nullptr && x_scale != nullptr, "project_qkv: NULL input");
  H3S_CHECK_ARG(c->scratch != nullptr && heads > 0 && sequence > 0, "project_qkv: empty problem");
  H3S_CHECK_ARG(chunk_rows > 0 && chunk_rows % H3S_Q_TILE == 0, "project_qkv: chunk_rows %d must be a positive multiple of 128", chunk_rows);
  H3S_CHECK_ARG(rope == nullptr || rope_strides != nullptr, "project_qkv: rope strides missing");
  cudaStream_t s = static_cast<cudaStream_t>(stream), side = static_cast<cudaStream_t>(side_stream);
  h3s_qkv_carriers out;
  out.q8 = c->q8; out.q_scale = c->q_scale; out.q_summary = c->q_summary;
  out.k8 = smooth_k ? nullptr : c->k8; out.k_scale = smooth_k ? nullptr : c->k_scale; out.k_summary = c->k_summary;
  out.k_stage = smooth_k ? k_stage : nullptr; out.v_stage = v_stage; out.stats = c->scratch;
  out.summary_dtype = c->summary_dtype; out.sequence_total = sequence;
  const int words = static_cast<int>(h3s_column_stats_scratch_bytes(heads) / sizeof(uint32_t));
  const int64_t rope_size = rope_dtype == H3S_F32 ? 4 : 2;
  int rc = H3S_OK;
  for (int start = 0; start < sequence; start += chunk_rows) {
    const int rows = chunk_rows < sequence - start ? chunk_rows : sequence - start;
    rc = convrot_quant_rows(static_cast<const char *>(x_bf16) + start * x_stride_row * 2, x_stride_row, rows, hidden, x_i8, x_scale,
                            static_cast<uint32_t *>(c->scratch), start == 0 ? words : 0, s);
    if (rc) return rc;
    out.row_start = start;
    const void *rope_rows = rope == nullptr ? nullptr : static_cast<const char *>(rope) + start * rope_strides[0] * rope_size;
    rc = qkv_gemm_carriers(x_i8, x_scale, w_i8, w_scale, rows, hidden, heads, &out, q_norm, k_norm, norm_dtype, epsilon,
                           rope_rows, rope_dtype, rope_strides, status, s);
    if (rc) return rc;
  }
  // One launch for short sequences, in whose kernels and between whose kernels the chip waits more than it works: from the last projection
  // tile to the end 11.9 us for 12.9 at 24 heads x 2304 tokens, and the host issues three calls for nine; whole blocks of 4 x 900 139 ->
  // 129 us, 24 x 900 140 -> 130, 24 x 2304 168 and 167, 12 x 8000 372 and 371.  For long ones, kernels of their own are the faster: 24 x 33272 151 us for 169.  Replayed
  // from a graph, without the host, whole projections several / one: 24 x 900 41.2 / 41.3, 24 x 2304 80.3 / 79.0, 24 x 4500 154.0 / 154.4,
  // 24 x 6000 199.1 / 200.5, 4 x 36000 226 / 230, 24 x 8000 255 / 259, 24 x 16000 496 / 509.
  if (static_cast<int64_t>(heads) * sequence <= kStagedOneLaunchRows)
    return staged_carriers(c, k_stage, v_stage, heads, sequence, smooth_k != 0, v_bound, s);
  rc = h3s_column_stats_finalize(c->scratch, H3S_BF16, heads, sequence, v_bound, smooth_k ? c->k_mean : nullptr,
                                 c->v_scale, s);
  if (rc) return rc;
  const int64_t head = static_cast<int64_t>(sequence) * H3S_HEAD_DIM;
  // the two second-phase quantisers are independent and each leaves part of the memory
  // system idle: V runs on the second stream underneath K
  if (smooth_k) {
    rc = order_after(s, side, event);
    if (rc) return rc;
    rc = h3s_quant_qk_blocks(k_stage, H3S_BF16, head, H3S_HEAD_DIM, c->k_mean, c->k8, c->k_scale, nullptr, H3S_F32,
                             heads, sequence, 0, sequence, H3S_KV_TILE, s);
  }
  if (!rc) rc = h3s_quant_v_fp8_half(v_stage, H3S_BF16, head, H3S_HEAD_DIM, c->v_scale, c->v8, c->v16, heads, sequence, 0,
                                     sequence, v_bound, smooth_k ? side : s);
  if (!smooth_k) return rc;
  // joined wherever it was forked, and only there: a capture must not wait for a stream outside it
  const int joined = order_after(side, s, event);
  return rc ? rc : joined;
}

int h3s_project_qkv(const h3s_layer_carriers *c, const void *x_bf16, int64_t x_stride_row, int sequence, int hidden,
                    int chunk_rows, int8_t *x_i8, float *x_scale, const int8_t *w_i8, const float *w_scale, int heads,
                    int smooth_k, void *k_stage, void *v_stage, const float *q_norm, const float *k_norm,
                    float epsilon, const void *rope, int rope_dtype, const int64_t *rope_strides, float v_bound,
                    int32_t *status, void *event, h3s_stream_t stream, h3s_stream_t side_stream) {
  return h3s_project_qkv_norms(c, x_bf16, x_stride_row, sequence, hidden, chunk_rows, x_i8, x_scale, w_i8, w_scale, heads, smooth_k, k_stage,
                               v_stage, q_norm, k_norm, H3S_F32, epsilon, rope, rope_dtype, rope_strides, v_bound, status, event,
                               stream, side_stream);
}

int h3s_status_mirror(const int32_t *status, int32_t *host_mirror, void *event, h3s_stream_t stream) {
  H3S_CHECK_ARG(status != nullptr && host_mirror != nullptr && event != nullptr, "status_mirror: NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  H3S_CHECK_CUDA(cudaMemcpyAsync(host_mirror, status, 4 * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  H3S_CHECK_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(event), s));
  return H3S_OK;
}

}  // extern "C"
