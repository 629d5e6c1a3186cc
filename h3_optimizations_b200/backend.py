"""The B200 sparse-attention backend: a drop-in for the reference's
``HybridSparseBackend`` (attention/sparse/backend.py:27-255) behind the same
duck-typed protocol the forward boundary calls
(attention_forward.py:99-128,148-246):

    prepare(q, k, v, *, layer_index, transformer_options) -> prepared
    prepare_projected(projected, *, layer_index, transformer_options) -> prepared
    execute(prepared) -> HND tensor (1,H,S,128) in the input dtype

``prepare`` runs, on torch's current stream and without a host sync:
column statistics (K mean, V amax) -> INT8 Q/K blocks with FP64 tile means ->
FP8 V carrier -> router.  ``execute`` launches the tcgen05 attention kernel.
There is no fallback of any kind: a device that is not sm_100, a missing
native library or a failed launch raises ``SparseSageError``.

Every wait inside the attention kernel is bounded; a wait that runs out makes
the kernel return early and leave a code in a per-device status word that the
backend hands to every launch.  Reading that word needs the stream to have
drained, so it is not done on the hot path: ``check_status()`` reads it (and
raises) whenever the caller synchronises anyway, ``forward_host`` calls it
before it returns, and the next ``prepare`` or ``prepare_projected`` on the device looks, without
blocking, at a mirror of the word in pinned host memory that a kernel which
gave up writes as well (with a copy behind every launch instead, the next
call's kernels began 8 us later).
"""

from __future__ import annotations

import torch

from . import _native, ops
from .carriers import PreparedFusedQKV, PreparedHybrid, PreparedLayer, PreparedSparse, ProjectedLayer, VCarrier, validate_prepared_fused_qkv
from .config import MODE_SAGE128_FUSED_QKV, HybridSparseConfig, resolve_video_budget
from .errors import FusedQKVError, SparseRouterError, SparseSageError
from .router import KV_TILE, Q_TILE, SparseTileRouter
from .runtime import get_runtime_snapshot

# Where one kernel makes all carriers of a layer, on one stream, and where kernels of their own do it on two.  Long layers do without the
# bookkeeping of jobs, and where a head has many KV tiles V goes beside the router, which takes longer the more they are.  Of the others a
# call that the host issues waits for the host first, and one kernel saves it a dozen calls; while that is so (``HOST_BOUND``) it is the faster.
# Replays have no host in them: up to a few rows it saves launches, from there on V is better off beside the router, until the
# router fills the chip by itself (``MANY_ROWS``).  us a call, two streams / one kernel, from the host (bf16, fp32) and replayed (bf16, fp32):
#   1 head x 3000    113 / 88   101 / 87    49.9 / 43.5  51.0 / 44.4      8 x 6000     102 / 87   102 / 100   86.0 / 89.1  97.1 / 98.0
#   4 x 4500          98 / 83    98 / 83    65.2 / 62.4  66.0 / 64.6      3 x 10500    102 / 94   102 / 97    91.8 / 91.2  97.1 / 101.9
#   2 x 9000         101 / 88   101 / 87    76.2 / 74.8  79.1 / 79.0      4 x 11900    119 / 119  129 / 136   115 / 122    125 / 134
#   4 x 6000         108 / 90   102 / 87    70.6 / 71.4  74.5 / 77.0      6 x 9000     118 / 122  135 / 134   116 / 120    129 / 132
#   8 x 4500          99 / 83    97 / 83    72.9 / 73.5  78.7 / 81.2      10 x 9000    171 / 172  194 / 201   165 / 167    188 / 189
#   24 x 2304        100 / 81    99 / 90    74.6 / 74.5  87.5 / 87.1      24 x 4500    150 / 149  184 / 183   144 / 144    169 / 169
#   24 x 3000         98 / 93   118 / 120   93.7 / 91.8  109 / 112        24 x 6000    211 / 209  249 / 252   202 / 199    234 / 231
#   16 x 4500        113 / 111  132 / 135   108 / 108    123 / 128        12 x 11900   300 / 298  340 / 344   291 / 284    323 / 319
# (heads of 13512 tokens: 4 of them 157 / 161, replayed 156 / 161; one of 33272 177 / 182, 180 / 183.)
ONE_STREAM_ROWS = 150_000
SHORT_HEAD_ROWS = 12_000
FEW_ROWS, MANY_ROWS = 20_000, 105_000  # of all heads
HOST_BOUND = 335_000_000  # rows of all heads, times the rows of one
# Bytes of a head's q, k and v from which ``forward_host`` ends with single heads: as long as they take to copy a chunk more is
# paid for by a shorter end, below that it costs the host's time.  us a call, pairs to the end / single heads at the end, 8 heads,
# bf16: 1212 tokens 818 / 1001, 4512 933 / 1046, 6512 1080 / 1130, 7512 1155 / 1181, 8512 1316 / 1313, 10512 1594 / 1555, 33272 4575 /
# 4374; fp32: 3512 1113 / 1157, 4512 1389 / 1389, 10512 2918 / 2845; 24 heads, bf16: 1212 2203 / 2384, 6512 2755 / 2769, 11512 4486 / 4458.
LONE_HEAD_BYTES = 6_500_000
# Output copies of ``forward_host`` are cut into pieces of this size.  A copy out that runs beside the next chunk's copies in
# slows them down, by how much depends on which of them it meets; between pieces the two directions are dealt out anew.
# us a call, whole / pieces of 3, 2, 1.6 and 1.25 MB: 24 heads x 9881 tokens 4189 / 3928, 3934, 3973, 3988; 12 x 8512 1940 / 1936, 1827,
# 1851, 1854; 24 x 6512 2995 / 3007, 2802, 2806, 2866; 4 x 33512 2545 / 2466, 2474, 2467, 2474; 8 x 33272 4486 / 4424, 4393, 4382, 4384;
# 8 x 4512 (2.3 MB a chunk) 930 / 936, 929, 915, 994; 24 x 11512 dense 4740 / 4704, 4687, 4683, 4681.
# A chunk of less than two pieces goes in one copy, as does the last one: there the host's time for a copy more (10 to 20 us) shows,
# 6 heads x 4923 fp32 (2.5 MB each) 1302 / 1431 in two.
COPY_OUT_BYTES = 1_600_000
V_QUANT_BOUND = 448.0  # FP32 accumulation (reference: sparse_sage.py:296)


def preflight():
    """Raise ``SparseSageError`` unless the native library loads and the
    current device is sm_100 (reference: sparse_sage.py:261-310)."""
    if not torch.cuda.is_available():
        raise SparseSageError("Hybrid Sparse Attention requires CUDA")
    try:
        capability = ops.device_capability()
    except _native.NativeError as exc:
        raise SparseSageError("B200 sparse backend is unavailable: %s" % exc) from exc
    if capability // 10 != 10:
        raise SparseSageError("B200 sparse backend requires sm_100; device is sm_%d" % capability)
    return capability


def one_carrier_kernel(heads, sequence, element_size):
    """Whether the carriers of a layer call on the current stream are made by one kernel."""
    rows = heads * sequence
    if rows > ONE_STREAM_ROWS or sequence > SHORT_HEAD_ROWS:
        return False
    if rows <= FEW_ROWS:
        return True
    replayed = torch.cuda.is_current_stream_capturing()
    if rows >= MANY_ROWS:
        return replayed or element_size == 2
    return not replayed and rows * sequence <= HOST_BOUND


class CapturedLayerCall:
    """``prepare`` + ``execute`` of one layer call on fixed input tensors, captured
    once into a CUDA graph.  A sampler calls the same layer with the same shapes
    and the same budget step after step; replaying the graph takes the host out
    of the step (four launches of most short layers, eight and half a dozen stream operations of the others otherwise) and
    closes the gaps between the small carrier kernels.  Every kernel still runs on
    every replay - statistics, carriers, router, attention (and, for a sharded
    owner, the exchange) - on whatever ``q``, ``k``, ``v`` hold at that moment; the
    output tensor and the carriers are the same buffers each time.  The device
    status word is not looked at between replays: call ``check_status()``.
    """

    def __init__(self, owner, q, k, v, *, layer_index, transformer_options, warmup=2):
        self.owner = owner
        # streams, status words, kernel attributes and exchange buffers come into being on the first
        # calls; none of that may happen inside the capture
        for _ in range(max(1, int(warmup))):
            owner.execute(owner.prepare(q, k, v, layer_index=layer_index, transformer_options=transformer_options))
        torch.cuda.synchronize(q.device)
        self.graph = torch.cuda.CUDAGraph()
        # thread-local error mode: a watchdog thread of a communication library may legally touch the
        # device while this thread captures
        with torch.cuda.graph(self.graph, capture_error_mode="thread_local"):
            self.prepared = owner.prepare(q, k, v, layer_index=layer_index, transformer_options=transformer_options)
            self.out = owner.execute(self.prepared)

    def replay(self):
        self.graph.replay()
        return self.out


class B200SparseBackend:
    name = "b200_sparse"
    requires_registered_sage = False
    requires_runtime_context = True
    approximate = True

    def __init__(self, config=None, *, router=None, projector=None, smooth_k=True, check_device=True):
        self.config = config or HybridSparseConfig()
        if not isinstance(self.config, HybridSparseConfig):
            raise TypeError("config must be HybridSparseConfig")
        if check_device:
            preflight()
        self.router = router if router is not None else SparseTileRouter(self.config)
        if (self.router.q_tile, self.router.kv_tile) != (Q_TILE, KV_TILE):
            raise SparseSageError(
                "router geometry %dQ x %dKV does not match the kernel's %dQ x %dKV"
                % (self.router.q_tile, self.router.kv_tile, Q_TILE, KV_TILE)
            )
        self.projector = projector
        if self.config.mode == MODE_SAGE128_FUSED_QKV and self.projector is None:
            from .projector import ChunkedSparseQKVProjector

            self.projector = ChunkedSparseQKVProjector()
        self.smooth_k = bool(smooth_k)
        self._status = {}  # device index -> (device int32[4], pinned mirror)

    # -- identity ---------------------------------------------------------

    @property
    def installation_signature(self):
        projector = self.projector
        return (
            self.name,
            self.config.signature,
            (type(self.router).__module__, type(self.router).__qualname__),
            ("sm_100a", Q_TILE, KV_TILE, "int8_qk", "fp8_e4m3_v", V_QUANT_BOUND, _native.ABI_VERSION),
            bool(self.smooth_k),
            None
            if projector is None
            else (
                type(projector).__module__,
                type(projector).__qualname__,
                getattr(projector, "name", None),
                getattr(projector, "installation_signature", None),
            ),
        )

    def as_status(self):
        return {
            "mode": self.config.mode,
            "video_budget": float(self.config.video_budget),
            "denser_early_late_steps": bool(self.config.denser_early_late_steps),
            "density_mode": self.config.density_mode,
            "sparge_attention": "h3sparse-abi-%d" % _native.ABI_VERSION,
            "sparse_architecture": "sm_100a",
            "sparse_q_tile": Q_TILE,
            "sparse_kv_tile": KV_TILE,
            "sparse_v_format": "fp8",
            "sparse_v_quant_bound": V_QUANT_BOUND,
            "sparse_extension_layout": "h3sparse",
            "approximate": True,
            "fused_qkv": self.projector is not None,
            "qkv_projector": getattr(self.projector, "name", None),
            "qkv_chunk_rows": getattr(self.projector, "chunk_rows", None),
            "smooth_k": bool(self.smooth_k),
        }

    # -- helpers ------------------------------------------------------------

    @staticmethod
    def _snapshot(transformer_options, sequence):
        snapshot = get_runtime_snapshot(transformer_options)
        if snapshot is None:
            raise SparseSageError("Sparse Attention requires an H3 runtime snapshot")
        if not snapshot.valid_layout:
            raise SparseSageError(
                "Sparse Attention requires a valid packed layout: %s"
                % (getattr(snapshot, "error", None) or "layout unavailable")
            )
        if int(snapshot.layout.seq_len) != int(sequence):
            raise SparseSageError(
                "runtime layout sequence %d does not match attention sequence %d"
                % (snapshot.layout.seq_len, sequence)
            )
        return snapshot

    @staticmethod
    def _metadata(mask_metadata, layer_index, heads):
        metadata = mask_metadata.as_dict()
        metadata.update(
            {
                "layer": int(layer_index),
                "sparse_sage_heads": int(heads),
                "total_q_video_tiles": int(mask_metadata.pure_video_q_tiles) * int(heads),
                "sparse_architecture": "sm_100a",
                "sparse_q_tile": Q_TILE,
                "sparse_kv_tile": KV_TILE,
                "sparse_v_format": "fp8",
                "sparse_accumulator": "f32",
                "sparse_v_quant_bound": V_QUANT_BOUND,
            }
        )
        return metadata

    @staticmethod
    def _sink(transformer_options, layer_index):
        recorder = (transformer_options or {}).get("h3_optimizations_attention_route")
        sink = getattr(recorder, "sink", None)
        return {} if sink is None else {"sink": sink(layer_index)}

    @staticmethod
    def _validate_qkv(q, k, v):
        if q.shape != k.shape or q.shape != v.shape:
            raise SparseSageError(
                "Sparse Sage requires equal self-attention Q/K/V shapes; got %s %s %s"
                % (tuple(q.shape), tuple(k.shape), tuple(v.shape))
            )
        if q.ndim != 4:
            raise SparseSageError("Sparse Sage expects HND rank-4 tensors")
        batch, heads, sequence, head_dim = q.shape
        if batch != 1:
            raise SparseSageError("released H3 expects attention batch 1; got %d" % batch)
        if head_dim != 128:
            raise SparseSageError("Sparse Sage requires head_dim 128; got %d" % head_dim)
        if q.dtype not in (torch.float16, torch.bfloat16, torch.float32) or q.dtype != k.dtype or q.dtype != v.dtype:
            raise SparseSageError("Sparse Sage Q/K/V require matching fp16, bf16 or fp32 dtypes")
        if q.device != k.device or q.device != v.device:
            raise SparseSageError("Sparse Sage Q/K/V devices differ")
        if any(t.stride(-1) != 1 for t in (q, k, v)):
            raise SparseSageError("Sparse Sage Q/K/V last dimension must be contiguous")
        if not q.is_cuda:
            raise SparseSageError("Sparse Sage requires CUDA")
        return heads, sequence

    def _side_stream(self, device):
        streams = self.__dict__.setdefault("_side_streams", {})
        key = device.index if device.index is not None else torch.cuda.current_device()
        if key not in streams:
            streams[key] = ops.SideStream(device)
        return streams[key]

    # -- device status word -------------------------------------------------

    ABORT_NAMES = {1: "Q tile load", 2: "K/V tile load", 3: "free K/V stage", 4: "QK^T result", 5: "P from the softmax warps",
                   6: "free score slot", 7: "P.V of an earlier tile", 8: "last P.V", 9: "Q rows in tensor memory",
                   10: "answer to the request for more work", 11: "end of a pass over the list", 12: "output sums being read",
                   13: "first row maxima", 14: "output tile staged", 15: "whole-sequence statistics"}
    # where another kernel than the attention waited, and what the words behind the code are
    ABORT_PLACES = {15: ("Layer carrier", "job %d, head %d, block %d of 128 rows")}

    def _status_slot(self, device):
        key = device.index if device.index is not None else torch.cuda.current_device()
        slot = self._status.get(key)
        if slot is None:
            word = torch.zeros(4, dtype=torch.int32, device=device)
            mirror = torch.zeros(4, dtype=torch.int32).pin_memory()
            slot = self._status[key] = (word, mirror)
        return slot

    @classmethod
    def _raise_for(cls, words, where):
        code, number, head, tile = (int(x) for x in words)
        if code != 0:
            kernel, places = cls.ABORT_PLACES.get(code, ("Sparse attention", "CTA %d, head %d, query tile %d"))
            raise SparseSageError(
                "%s kernel gave up waiting for %s (code %d) in %s (%s); the output of that launch is invalid"
                % (kernel, cls.ABORT_NAMES.get(code, "an unknown event"), code, places % (number, head, tile), where))

    def _poll_status(self, device):
        """Non-blocking look at the mirror of the earlier launches' status."""
        slot = self._status.get(device.index if device.index is not None else torch.cuda.current_device())
        if slot is not None:
            words = slot[1].tolist()
            if words[0] != 0:
                self._raise_for(words, "reported by an earlier launch")

    def check_status(self, device=None):
        """Synchronise with the device and raise ``SparseSageError`` if a
        bounded device wait ran out in any launch of a layer call since the last
        check.  Clears the word."""
        devices = list(self._status) if device is None else [torch.device(device).index]
        for key in devices:
            slot = self._status.get(key)
            if slot is None:
                continue
            words = slot[0].cpu().tolist()
            if words[0] == 0:
                words = slot[1].tolist()  # a kernel of another stream may have got to the mirror after both were cleared
            if words[0] != 0:
                slot[0].zero_()
                slot[1].zero_()
            self._raise_for(words, "found by check_status")

    # -- protocol -------------------------------------------------------------

    def prepare(self, q, k, v, *, layer_index, transformer_options):
        heads, sequence = self._validate_qkv(q, k, v)
        self._poll_status(q.device)
        snapshot = self._snapshot(transformer_options, sequence)
        video_budget = resolve_video_budget(
            self.config, snapshot.step_index, snapshot.total_steps, layer_index
        )
        try:
            geometry = self.router.geometry(snapshot.layout)
            retained = self.router._retained(video_budget, geometry)
            need_route = retained < geometry.pure_video_kv_tiles
            # One kernel makes all carriers of most short layers.  Else every carrier has its own, on two streams: the column
            # statistics (K mean, V scale) run on the second one while the Q quantiser, which needs neither, starts at once on the
            # current one; the K quantiser joins when the statistics are in, and the V carrier is held back until the K quantiser
            # is through, so that this memory-bound kernel runs beside the router, which leaves the memory system idle.  Every
            # buffer is allocated on the current stream, which both chains rejoin before returning.
            stream = _native.stream_ptr(q.device)
            side = self._side_stream(q.device)  # there from the first call on: a capture must not bring it into being
            if one_carrier_kernel(heads, sequence, q.element_size()):
                side = None
            buffers = ops.LayerBuffers(heads, sequence, q.device, smooth_k=self.smooth_k,
                                       summary_dtype=torch.float64 if need_route else None)
            try:
                if side is None:
                    word, mirror = self._status_slot(q.device)
                    ops.prepare_layer(q, k, v, buffers, stream, smooth_k=self.smooth_k, status=word, status_mirror=mirror,
                                      v_bound=V_QUANT_BOUND)
                else:
                    ops.quant_qkv(q, k, v, buffers, side, stream, smooth_k=self.smooth_k, v_after_k=need_route,
                                  v_bound=V_QUANT_BOUND)
                if need_route:
                    route = self.router.build_route_from_summaries(
                        buffers.q_summary, buffers.k_summary, snapshot.layout, video_budget,
                        **self._sink(transformer_options, layer_index),
                    )
                else:
                    route = self.router.build_route(
                        q, k, snapshot.layout, video_budget, **self._sink(transformer_options, layer_index)
                    )
            finally:
                # on every exit path the main stream is ordered after the second one, so the
                # allocator cannot hand these buffers to someone else while it still runs
                if side is not None:
                    side.join(stream)
        except SparseRouterError as exc:
            raise SparseSageError("sparse routing failed: %s" % exc) from exc
        except _native.NativeError as exc:
            raise SparseSageError("carrier preparation failed: layer=%d: %s" % (layer_index, exc)) from exc
        buffers.release_call()
        metadata = self._metadata(route.metadata, layer_index, heads)
        metadata["smooth_k"] = self.smooth_k
        return PreparedHybrid(sparse=PreparedLayer.over(
            buffers, route=route, output_dtype=q.dtype, output_shape=tuple(q.shape), layer_index=int(layer_index), metadata=metadata))

    def prepare_projected(self, projected, *, layer_index, transformer_options):
        try:
            validate_prepared_fused_qkv(projected)
        except FusedQKVError as exc:
            raise SparseSageError(str(exc)) from exc
        snapshot = self._snapshot(transformer_options, projected.sequence)
        video_budget = resolve_video_budget(
            self.config, snapshot.step_index, snapshot.total_steps, layer_index
        )
        heads, sequence = int(projected.heads), int(projected.sequence)
        lazy = isinstance(projected, ProjectedLayer)
        device = projected.device if lazy else projected.q_int8.device
        if device.type != "cuda":
            raise SparseSageError("fused H3 Sparse Sage requires CUDA")
        self._poll_status(device)
        try:
            route = self.router.build_route_from_summaries(
                projected.q_summary, projected.k_summary, snapshot.layout, video_budget,
                **self._sink(transformer_options, layer_index),
            )
            # after the route: a route sink may have been handed the carriers meanwhile
            buffers = projected.untouched() if lazy else None
            prepacked = True
            if buffers is None:
                v_carrier, v_scale = VCarrier.of(projected), projected.v_scale
                prepacked = v_carrier.codes is not None
                if not prepacked:
                    v_carrier, v_scale = ops.quant_v_fp8(projected.v, None, V_QUANT_BOUND)
        except SparseRouterError as exc:
            raise SparseSageError("sparse routing failed: %s" % exc) from exc
        except _native.NativeError as exc:
            raise SparseSageError("carrier preparation failed: layer=%d: %s" % (layer_index, exc)) from exc
        metadata = self._metadata(route.metadata, layer_index, heads)
        metadata.update(
            {
                "qkv_projection": "fused_int8",
                "smooth_k": bool(projected.smooth_k),
                "prepacked_fp8_v": prepacked,
            }
        )
        if buffers is not None:
            return PreparedHybrid(sparse=PreparedLayer.over(
                buffers, route=route, output_dtype=projected.output_dtype, output_shape=(1, heads, sequence, projected.head_dim),
                layer_index=int(projected.layer_index), metadata=metadata))
        sparse = PreparedSparse(
            q_int8=projected.q_int8, k_int8=projected.k_int8, v_carrier=v_carrier,
            q_scale=projected.q_scale, k_scale=projected.k_scale, v_scale=v_scale, route=route,
            output_dtype=projected.output_dtype, output_shape=(1, heads, sequence, projected.head_dim),
            layer_index=int(projected.layer_index), sequence=sequence, heads=heads, metadata=metadata,
        )
        return PreparedHybrid(sparse=sparse)

    def execute(self, prepared, out=None, peer_out_ptrs=None):
        """Run the attention kernel on prepared carriers.  ``out`` (optional) is
        an HND ``(1, H, S, 128)`` tensor or view to write into;
        ``peer_out_ptrs`` (head-sharded runs, see ``sharding.HeadShardedBackend``)
        are the device addresses of the same head slice inside the peers'
        outputs, which receive every tile as well."""
        sparse = prepared.sparse
        route = sparse.route
        geometry = route.geometry
        buffers = sparse.untouched() if isinstance(sparse, PreparedLayer) else None
        device = sparse.q_int8.device if buffers is None else buffers.device
        word, mirror = self._status_slot(device)
        try:
            out_dtype = sparse.output_dtype
            if buffers is not None:
                return ops.sparse_attention_of(
                    buffers, route.indices, q_start=geometry.pure_video_q_start, q_stop=geometry.pure_video_q_stop, out=out,
                    out_dtype=out_dtype, status=word, status_mirror=mirror, peer_out_ptrs=peer_out_ptrs)
            v = VCarrier.of(sparse)
            return ops.sparse_attention(
                sparse.q_int8, sparse.k_int8, v.codes, sparse.q_scale, sparse.k_scale,
                sparse.v_scale, route.indices,
                q_start=geometry.pure_video_q_start, q_stop=geometry.pure_video_q_stop,
                out=out, out_dtype=out_dtype, status=word, status_mirror=mirror, peer_out_ptrs=peer_out_ptrs, v_half=v.half,
            )
        except _native.NativeError as exc:
            raise SparseSageError(
                "Sparse attention kernel failed: layer=%d sequence=%d heads=%d dtype=%s: %s"
                % (sparse.layer_index, sparse.sequence, sparse.heads, sparse.output_dtype, exc)
            ) from exc

    def capture(self, q, k, v, *, layer_index, transformer_options):
        """This layer call as a replayable CUDA graph (see ``CapturedLayerCall``)."""
        return CapturedLayerCall(self, q, k, v, layer_index=layer_index, transformer_options=transformer_options)

    def execute_projected(self, module, prepared):
        """Attention followed by the block's ``out_proj`` on the tensor cores:
        returns ``(S, hidden)`` as the forward boundary allows a backend to do
        (attention_forward.py:99-128; the reference's streamed backend does it in
        attention/sparse/sparse_sage_streamed.py:1454-1472).  The attention output
        is written token-major, so its ``(S, heads*128)`` view feeds the GEMM
        without a copy.  Returns ``None`` - the caller then runs ``execute`` and
        the module's own ``out_proj`` - when the projection is not a plain bf16
        Linear on the attention's device."""
        linear = getattr(module, "out_proj", None)
        weight = getattr(linear, "weight", None)
        sparse = prepared.sparse
        if (weight is None or weight.ndim != 2 or weight.dtype != torch.bfloat16
                or weight.dtype != sparse.output_dtype
                or weight.device != (sparse.device if isinstance(sparse, PreparedLayer) else sparse.q_int8.device)
                or weight.shape[1] != sparse.heads * 128 or weight.shape[0] % 8 or weight.stride(1) != 1):
            return None
        out_hnd = self.execute(prepared)                                   # (1, H, S, 128) view of (S, H, 128)
        rows = out_hnd.permute(0, 2, 1, 3).reshape(sparse.sequence, sparse.heads * 128)
        if rows.data_ptr() != out_hnd.data_ptr():                          # never a copy with this backend's buffers
            rows = rows.contiguous()
        bias = getattr(linear, "bias", None)
        try:
            result = ops.dense_gemm(rows, weight, bias=None if bias is None else bias.detach().float().contiguous())
        except _native.NativeError as exc:
            raise SparseSageError("output projection failed: layer=%d: %s" % (sparse.layer_index, exc)) from exc
        return result

    def forward(self, q, k, v, *, layer_index, transformer_options):
        """``prepare`` + ``execute`` for a batch: every sparse backend of the
        reference is limited to batch 1 (attention/sparse/sparse_sage.py:448-449)
        and so are ``prepare`` / ``execute`` here; batch elements are independent,
        so this entry walks them one after the other (one route per element) and
        returns ``(B, H, S, 128)``."""
        if q.ndim != 4 or q.shape != k.shape or q.shape != v.shape:
            raise SparseSageError("forward expects equal rank-4 HND Q/K/V; got %s %s %s"
                                  % (tuple(q.shape), tuple(k.shape), tuple(v.shape)))
        # a batch is written in place (gathering the elements afterwards moved every output twice)
        whole = torch.empty(q.shape, dtype=q.dtype, device=q.device) if q.shape[0] > 1 else None
        outputs = []
        for b in range(q.shape[0]):
            prepared = self.prepare(q[b:b + 1], k[b:b + 1], v[b:b + 1], layer_index=layer_index,
                                    transformer_options=transformer_options)
            outputs.append(self.execute(prepared, out=None if whole is None else whole[b:b + 1]))
        return whole if whole is not None else outputs[0] if outputs else torch.cat(outputs, dim=0)

    # -- host-resident activations -------------------------------------------

    def forward_host(self, q, k, v, out=None, *, layer_index, transformer_options, heads_per_chunk=None):
        """``prepare`` + ``execute`` for Q/K/V that live in (pinned) HOST memory.

        Heads are independent on the whole path, so the call walks the heads in
        chunks and overlaps three things on three streams: the host-to-device
        copy of chunk c+1, the kernels of chunk c (on the current stream) and
        the device-to-host copy of the output of chunk c-1.  The PCIe input copy
        is the longest of the three, so the call takes about as long as that
        copy alone.  Returns ``out`` (host, HND ``(1, H, S, 128)``; allocated
        pinned when not given).  With a route sink installed the heads are not
        split (the sink expects one call per layer).  How many heads go through
        at a time decides into how many parts the attention kernel cuts the rows that
        see every key, and so the order of their FP32 sums: the last bits of a head may
        differ between chunk sizes, and from those of a whole layer.  The call returns once the
        output is in host memory and raises if a launch reported an expired
        device wait."""
        if q.is_cuda or k.is_cuda or v.is_cuda:
            raise SparseSageError("forward_host expects host tensors; use prepare/execute for device tensors")
        if q.shape != k.shape or q.shape != v.shape or q.ndim != 4 or q.shape[0] != 1 or q.shape[3] != 128:
            raise SparseSageError("forward_host expects equal (1, H, S, 128) Q/K/V; got %s %s %s"
                                  % (tuple(q.shape), tuple(k.shape), tuple(v.shape)))
        if not (q.is_contiguous() and k.is_contiguous() and v.is_contiguous()):
            raise SparseSageError("forward_host expects contiguous HND host tensors")
        _, heads, sequence, _ = q.shape
        if out is None:
            out = torch.empty(q.shape, dtype=q.dtype).pin_memory()
        elif out.shape != q.shape or out.dtype != q.dtype or out.is_cuda or not out.is_contiguous():
            raise SparseSageError("forward_host: out must be a contiguous host tensor shaped and typed like q")
        recorder = (transformer_options or {}).get("h3_optimizations_attention_route")
        whole = getattr(recorder, "sink", None) is not None
        head_bytes = sequence * 128 * q.element_size()
        bounds = [(0, heads)] if whole else self._head_chunks(heads, heads_per_chunk, 3 * head_bytes)
        chunk = max((b - a for a, b in bounds), default=1)
        device = torch.device("cuda", torch.cuda.current_device())
        main = torch.cuda.current_stream(device)
        state = self._host_pipeline(device, chunk, sequence, q.dtype, min(3, len(bounds)))
        h2d, d2h, slots = state["h2d"], state["d2h"], state["slots"]
        h2d.wait_stream(main)
        d2h.wait_stream(main)
        for index, (a, b) in enumerate(bounds):
            slot = slots[index % len(slots)]
            n = b - a
            with torch.cuda.stream(h2d):
                if index >= len(slots):
                    h2d.wait_event(slot["computed"])  # the kernels of the chunk that used this slot are done
                for name, src in (("q", q), ("k", k), ("v", v)):
                    slot[name][:, :n].copy_(src[:, a:b], non_blocking=True)
                slot["loaded"].record(h2d)
            main.wait_event(slot["loaded"])
            if index >= len(slots):
                main.wait_event(slot["stored"])  # its previous output has left the device
            prepared = self.prepare(slot["q"][:, :n], slot["k"][:, :n], slot["v"][:, :n],
                                    layer_index=layer_index, transformer_options=transformer_options)
            self.execute(prepared, out=slot["out"][:, :n])
            slot["computed"].record(main)
            with torch.cuda.stream(d2h):
                d2h.wait_event(slot["computed"])
                if b < heads and n * head_bytes >= 2 * COPY_OUT_BYTES:
                    self._copy_out(out[:, a:b], slot["out"][:, :n])
                else:
                    out[:, a:b].copy_(slot["out"][:, :n], non_blocking=True)
                slot["stored"].record(d2h)
        main.wait_stream(d2h)
        main.wait_stream(h2d)
        main.synchronize()  # the result lives in host memory: it is complete when the call returns
        self.check_status(device)
        return out

    @staticmethod
    def _head_chunks(heads, heads_per_chunk, head_bytes=LONE_HEAD_BYTES):
        """The heads ``forward_host`` takes through at a time, as (first, stop).  By itself it takes two where that leaves
        at least four chunks, so that copy-in, kernels and copy-out overlap, and ends with single heads where a head's q, k and v
        (``head_bytes``) are many: what the last chunk's kernels and copy-out take comes on top of the copies in."""
        if heads_per_chunk is not None or heads < 8 or head_bytes < LONE_HEAD_BYTES:
            if heads_per_chunk is None:
                heads_per_chunk = 2 if heads >= 8 else 1
            chunk = max(1, min(int(heads_per_chunk), heads))
            return [(a, min(a + chunk, heads)) for a in range(0, heads, chunk)]
        pairs = (heads - 1) // 2
        return [(2 * i, 2 * i + 2) for i in range(pairs)] + [(a, a + 1) for a in range(2 * pairs, heads)]

    @staticmethod
    def _copy_out(to, source):
        """One chunk's output to host memory, in pieces of ``COPY_OUT_BYTES`` or a little more."""
        pieces = max(1, int(to.numel() * to.element_size() / COPY_OUT_BYTES))
        for part, rows in zip(to.view(-1, 128).tensor_split(pieces), source.view(-1, 128).tensor_split(pieces)):
            part.copy_(rows, non_blocking=True)

    def _host_pipeline(self, device, chunk, sequence, dtype, n_slots):
        key = (device.index, int(chunk), int(sequence), dtype, int(n_slots))
        cache = self.__dict__.setdefault("_host_pipelines", {})
        state = cache.get(key)
        if state is None:
            cache.clear()  # one geometry at a time: the staging buffers are large
            shape = (1, chunk, sequence, 128)
            slots = []
            for _ in range(n_slots):
                slot = {name: torch.empty(shape, dtype=dtype, device=device) for name in ("q", "k", "v", "out")}
                slot.update({name: torch.cuda.Event() for name in ("loaded", "computed", "stored")})
                slots.append(slot)
            state = {"h2d": torch.cuda.Stream(device), "d2h": torch.cuda.Stream(device), "slots": slots}
            cache[key] = state
        return state

    def reference_lut(self, prepared):
        """The route in the reference's delta-LUT encoding ``(lut, valid)``."""
        sparse = prepared.sparse
        lut, valid, _ = self.router._lut(sparse.route, sparse.q_int8.device, sparse.heads)
        return lut, valid
