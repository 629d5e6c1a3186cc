"""Chunked native-carrier QKV provider for the B200 backend.

Counterpart of the reference's ``ChunkedSparseQKVProjector``
(attention/sparse/chunked_qkv.py:205-366): the packed ``x (S, hidden)`` is
projected in 4096-row chunks straight into full-length quantised carriers, so
no full-precision Q/K/V of the whole sequence is handed to the backend.

Per chunk:  ConvRot (Hadamard-256) + per-row INT8 of the activations
            -> tcgen05 INT8 GEMM against the INT8 QKV weight whose epilogue
               writes the carriers: INT8 Q blocks, scales and tile means
               straight from the accumulators (Q is never stored in a wider
               format), K tile means, bf16 staging of K and V with their
               column sums / maxima accumulated on the way.
After the last chunk (K smoothing and the V scale need whole-sequence
statistics): the statistics are finalised, the staged K is quantised with the
mean removed and the staged V becomes the FP8-E4M3 carrier.  With
``smooth_k=False`` (what every chunked producer of the reference does,
chunked_qkv.py:289) K leaves the epilogue as INT8 blocks like Q and only V is
staged.  The default keeps the smoothing on, which is what the attention
kernel's accuracy figures are stated for.

The module handed to ``project`` must expose ``heads``, ``head_dim`` and the
INT8 weight in the rotated domain: ``qkv_weight_int8`` (3*H*128, hidden) with
rows ordered ``[Q heads | K heads | V heads]`` (fused_qkv.py:195,394) and
``qkv_weight_scale`` (3*H*128,) fp32.  When the module carries ``q_norm`` and
``k_norm`` (objects with ``weight`` (128,) and ``eps``) the per-head RMS norm of
Q and K runs in the GEMM epilogue, and with ``rope_freqs`` (1,S,1,48,2,2) the
split-half rotation as well (fused_qkv.py:225-289); a module without norms
(the benchmark configuration) is projected without either, and asking for the
rotation without norms is an error.
"""

from __future__ import annotations

import math

import torch

from . import _native, ops
from .carriers import ProjectedLayer
from .errors import FusedQKVError
from .router import KV_TILE, Q_TILE

CHUNK_ROWS = 4096
HEAD_DIM = 128
V_QUANT_BOUND = 448.0


_SIDE_STREAMS = {}


def _side_stream(device):
    key = device.index if device.index is not None else torch.cuda.current_device()
    if key not in _SIDE_STREAMS:
        _SIDE_STREAMS[key] = ops.SideStream(device)
    return _SIDE_STREAMS[key]


def _validate_chunk_rows(chunk_rows, q_tile=Q_TILE, kv_tile=KV_TILE):
    chunk_rows = int(chunk_rows)
    alignment = math.lcm(int(q_tile), int(kv_tile))
    if chunk_rows <= 0 or chunk_rows % alignment:
        raise FusedQKVError(
            "chunked Sparse Sage QKV rows must be a positive multiple of %d" % alignment
        )
    return chunk_rows


class ChunkedSparseQKVProjector:
    name = "chunked_b200_sparse_qkv"
    qk_format = "sparge_block_int8"

    def __init__(self, chunk_rows=CHUNK_ROWS, *, smooth_k=True, summary_dtype=torch.float32):
        self.chunk_rows = _validate_chunk_rows(chunk_rows)
        self.smooth_k = bool(smooth_k)
        self.summary_dtype = summary_dtype

    @property
    def installation_signature(self):
        return (self.name, self.qk_format, self.chunk_rows, ("sm_100a", _native.ABI_VERSION, self.smooth_k))

    # -- protocol ---------------------------------------------------------

    def try_project(self, module, x, rope_freqs, *, layer_index, transformer_options):
        if rope_freqs is not None and (getattr(module, "q_norm", None) is None or getattr(module, "k_norm", None) is None):
            return None
        if getattr(module, "qkv_weight_int8", None) is None or getattr(module, "qkv_weight_scale", None) is None:
            return None
        return self.project(module, x, rope_freqs, layer_index=layer_index, transformer_options=transformer_options)

    def project(self, module, x, rope_freqs, *, layer_index, transformer_options):
        del transformer_options
        weight = getattr(module, "qkv_weight_int8", None)
        scale = getattr(module, "qkv_weight_scale", None)
        if weight is None or scale is None:
            raise FusedQKVError("module does not expose qkv_weight_int8 / qkv_weight_scale")
        q_norm, k_norm = getattr(module, "q_norm", None), getattr(module, "k_norm", None)
        if (q_norm is None) != (k_norm is None):
            raise FusedQKVError("module must carry both q_norm and k_norm or neither")
        if rope_freqs is not None and q_norm is None:
            raise FusedQKVError("RoPE in the QKV epilogue needs the module's q_norm / k_norm")
        norm = None
        if q_norm is not None:
            if float(q_norm.eps) != float(k_norm.eps):
                raise FusedQKVError("q_norm and k_norm use different epsilons")
            norm = (q_norm.weight, k_norm.weight, float(q_norm.eps))
        return run_chunked_sparse_qkv(
            x, weight, scale, heads=int(module.heads), head_dim=int(module.head_dim),
            layer_index=layer_index, chunk_rows=self.chunk_rows, smooth_k=self.smooth_k,
            summary_dtype=self.summary_dtype, norm=norm, rope_freqs=rope_freqs,
        )


def run_chunked_sparse_qkv(x, w_i8, w_scale, *, heads, head_dim=HEAD_DIM, layer_index=0,
                           chunk_rows=CHUNK_ROWS, smooth_k=True, summary_dtype=torch.float32,
                           status=None, norm=None, rope_freqs=None):
    if not x.is_cuda or x.dtype != torch.bfloat16 or x.ndim != 2:
        raise FusedQKVError("chunked Sparse Sage QKV requires a rank-2 CUDA BF16 input")
    if torch.is_grad_enabled() and x.requires_grad:
        raise FusedQKVError("chunked Sparse Sage QKV is inference-only")
    if head_dim != HEAD_DIM:
        raise FusedQKVError("chunked Sparse Sage QKV requires H3 head_dim 128")
    chunk_rows = _validate_chunk_rows(chunk_rows)
    sequence, hidden = int(x.shape[0]), int(x.shape[1])
    n_out = 3 * heads * HEAD_DIM
    if sequence <= 0 or tuple(w_i8.shape) != (n_out, hidden) or w_i8.dtype != torch.int8:
        raise FusedQKVError("QKV weight must be int8 (3*heads*128, hidden) = (%d, %d)" % (n_out, hidden))
    if tuple(w_scale.shape) != (n_out,) or w_scale.dtype != torch.float32:
        raise FusedQKVError("QKV weight scale must be fp32 (%d,)" % n_out)
    device = x.device
    q_norm = k_norm = None
    epsilon = 0.0
    if norm is not None:
        q_norm, k_norm, epsilon = norm
        # bf16 weights go to the kernel as they are: two launches and two tensors fewer
        dtype = torch.bfloat16 if q_norm.dtype == k_norm.dtype == torch.bfloat16 else torch.float32
        q_norm = q_norm.detach().to(device=device, dtype=dtype).contiguous()
        k_norm = k_norm.detach().to(device=device, dtype=dtype).contiguous()
        if tuple(q_norm.shape) != (HEAD_DIM,) or tuple(k_norm.shape) != (HEAD_DIM,):
            raise FusedQKVError("q_norm / k_norm weights must have 128 elements")
    if rope_freqs is not None:
        if norm is None:
            raise FusedQKVError("RoPE in the QKV epilogue needs the q_norm / k_norm weights")
        if (rope_freqs.ndim != 6 or tuple(rope_freqs.shape[:3]) != (1, sequence, 1)
                or tuple(rope_freqs.shape[3:]) != (48, 2, 2) or rope_freqs.device != device):
            raise FusedQKVError("rope_freqs must be (1, %d, 1, 48, 2, 2) on the projection's device" % sequence)
        if rope_freqs.dtype not in (torch.float32, torch.bfloat16):
            rope_freqs = rope_freqs.float()
    if summary_dtype is None:  # as torch.empty takes it
        summary_dtype = torch.get_default_dtype()
    try:
        buffers = ops.LayerBuffers(heads, sequence, device, smooth_k=smooth_k, summary_dtype=summary_dtype)
        # every launch of the projection from one native call (24 heads x 2304 tokens, with
        # backend and out_proj: 344 -> 259 us)
        ops.project_qkv(x, w_i8.contiguous(), w_scale.contiguous(), buffers, _side_stream(device), _native.stream_ptr(device),
                        heads=heads, chunk_rows=chunk_rows, smooth_k=smooth_k, q_norm=q_norm, k_norm=k_norm,
                        epsilon=float(epsilon), rope=rope_freqs, status=status, v_bound=V_QUANT_BOUND)
    except _native.NativeError as exc:
        raise FusedQKVError("chunked QKV projection failed: layer=%d: %s" % (layer_index, exc)) from exc
    q_summary, k_summary = buffers.q_summary, buffers.k_summary
    buffers.release_call()
    return ProjectedLayer.over(
        buffers, v=None, q_summary=q_summary, k_summary=k_summary, output_dtype=x.dtype, head_dim=HEAD_DIM,
        layer_index=int(layer_index), smooth_k=bool(smooth_k))
