"""Carrier data contracts (reference: attention/sparse/fused_qkv.py:30-154,
attention/sparse/sparse_sage.py:401-417)."""

from __future__ import annotations

from dataclasses import InitVar, dataclass, field

import torch

from .errors import FusedQKVError
from .router import KV_TILE, Q_TILE

HEAD_DIM = 128


class VCarrier:
    """The E4M3 codes of V and, while nobody else holds them, the FP16 copy that was written with
    them.  Whoever is handed the codes may write to them, so the copy is dropped then and the
    attention call makes its own (about 50 us at 24 heads x 33272 tokens)."""

    __slots__ = ("codes", "half")

    def __init__(self, codes, half=None):
        self.codes = codes
        self.half = half

    @classmethod
    def of(cls, prepared):
        """The pair that ``prepared`` holds; its codes alone where it is no class of this module."""
        pair = getattr(prepared, "_v", None)
        return pair if isinstance(pair, cls) else cls(prepared.v_carrier)

    def __reduce__(self):
        return VCarrier, (self.codes, self.half)

    @classmethod
    def field(cls):
        """``v_carrier`` of a class that keeps its codes in a pair (``_v``)."""

        def get(prepared):
            prepared._v.half = None
            return prepared._v.codes

        def put(prepared, codes):
            prepared._v = codes if isinstance(codes, cls) else cls(codes)

        return property(get, put)


@dataclass
class PreparedFusedQKV:
    """Output of a QKV projector: INT8 Q/K carriers with per-block scales and
    tile means, plus V either floating HND (``v``) or already packed
    (``v_carrier`` e4m3 ``(1,H,128,pad128(S))`` + ``v_scale`` ``(1,H,128)``;
    ``v_half``: its FP16 copy, see ``VCarrier``, which may also be given as ``v_carrier``)."""

    q_int8: torch.Tensor
    q_scale: torch.Tensor
    k_int8: torch.Tensor
    k_scale: torch.Tensor
    v: torch.Tensor | None
    q_summary: torch.Tensor
    k_summary: torch.Tensor
    output_dtype: torch.dtype
    sequence: int
    heads: int
    head_dim: int
    layer_index: int
    smooth_k: bool = False
    v_carrier: torch.Tensor | None = None
    v_scale: torch.Tensor | None = None
    v_half: InitVar[torch.Tensor | None] = None

    def __post_init__(self, v_half):
        if v_half is not None:
            self._v.half = v_half


PreparedFusedQKV.v_carrier = VCarrier.field()


def _carrier_spec(prepared):
    """What each tensor of a ``PreparedFusedQKV`` must look like, as rows of
    ``(field, tensor, shape, dtype | None, message)``, in the order they are checked."""
    sequence, heads, head_dim = int(prepared.sequence), int(prepared.heads), int(prepared.head_dim)
    q_blocks, k_blocks = -(-sequence // Q_TILE), -(-sequence // KV_TILE)
    full = (1, heads, sequence, head_dim)
    rows = [
        ("q_int8", prepared.q_int8, full, None, "fused H3 Q/K carrier shape is invalid"),
        ("k_int8", prepared.k_int8, full, None, "fused H3 Q/K carrier shape is invalid"),
        ("q_int8", prepared.q_int8, None, torch.int8, "fused H3 Q/K carriers must be INT8"),
        ("k_int8", prepared.k_int8, None, torch.int8, "fused H3 Q/K carriers must be INT8"),
    ]
    v = VCarrier.of(prepared)
    if v.codes is None:
        if prepared.v is None:
            raise FusedQKVError("fused H3 V is missing")
        rows.append(("v", prepared.v, full, prepared.output_dtype, "fused H3 V carrier is invalid"))
    else:
        padded = -(-sequence // 128) * 128
        rows.append(("v_carrier", v.codes, (1, heads, head_dim, padded), None,
                     "prepacked H3 FP8 V carrier shape is invalid"))
        rows.append(("v_carrier", v.codes, None, torch.float8_e4m3fn, "prepacked H3 V carrier must be E4M3 FP8"))
        if v.half is not None:
            rows.append(("v_half", v.half, (1, heads, head_dim, padded), torch.float16,
                         "FP16 copy of the prepacked H3 FP8 V is invalid"))
        if prepared.v_scale is None:
            raise FusedQKVError("prepacked H3 FP8 V requires V scale")
        rows.append(("v_scale", prepared.v_scale, (1, heads, head_dim), None, "prepacked H3 V scale shape is invalid"))
        rows.append(("v_scale", prepared.v_scale, None, torch.float32, "prepacked H3 V scale must be FP32"))
    rows += [
        ("q_scale", prepared.q_scale, (1, heads, q_blocks), None, "fused H3 Q scale shape is invalid"),
        ("k_scale", prepared.k_scale, (1, heads, k_blocks), None, "fused H3 K scale shape is invalid"),
        ("q_scale", prepared.q_scale, None, torch.float32, "fused H3 Q/K scales must be float32"),
        ("k_scale", prepared.k_scale, None, torch.float32, "fused H3 Q/K scales must be float32"),
        ("q_summary", prepared.q_summary, (1, heads, q_blocks, head_dim), None, "fused H3 Q router summary shape is invalid"),
        ("k_summary", prepared.k_summary, (1, heads, k_blocks, head_dim), None, "fused H3 K router summary shape is invalid"),
    ]
    return rows


def validate_prepared_fused_qkv(prepared):
    """Check a projector's output against the carrier contract
    (attention/sparse/fused_qkv.py:95-154: same conditions, same
    ``FusedQKVError`` texts) and hand it back.  The conditions are a table
    (``_carrier_spec``) walked once; device and contiguity are checked over
    every tensor the table names.  Carriers that nobody has been handed yet are
    as ``ops.LayerBuffers`` laid them out."""
    if isinstance(prepared, ProjectedLayer) and prepared.untouched() is not None:
        return prepared
    if int(prepared.head_dim) != HEAD_DIM:
        raise FusedQKVError("fused H3 QKV requires head_dim 128")
    seen = {}
    for name, tensor, shape, dtype, message in _carrier_spec(prepared):
        if shape is not None and tuple(tensor.shape) != shape:
            raise FusedQKVError(message)
        if dtype is not None and tensor.dtype != dtype:
            raise FusedQKVError(message)
        seen[name] = tensor
    home = prepared.q_int8.device
    if any(tensor.device != home for tensor in seen.values()):
        raise FusedQKVError("fused H3 QKV carrier devices differ")
    # V in floating point may be a strided view of the projection; everything else is dense
    if any(not tensor.is_contiguous() for name, tensor in seen.items() if name != "v"):
        raise FusedQKVError("fused H3 QKV carriers must be contiguous")
    return prepared


@dataclass
class PreparedSparse:
    """Everything one attention launch needs (the counterpart of
    ``PreparedSparseSage``): carriers, scales, the packed route and metadata.
    ``lut`` / ``valid_block_num`` in the reference's delta encoding are
    produced on demand by ``B200SparseBackend.reference_lut``."""

    q_int8: torch.Tensor
    k_int8: torch.Tensor
    v_carrier: torch.Tensor
    q_scale: torch.Tensor
    k_scale: torch.Tensor
    v_scale: torch.Tensor
    route: object  # router.SparseRoute
    output_dtype: torch.dtype
    output_shape: tuple
    layer_index: int
    sequence: int
    heads: int
    metadata: dict = field(default_factory=dict)
    v_half: InitVar[torch.Tensor | None] = None  # FP16 copy of v_carrier, see VCarrier

    def __post_init__(self, v_half):
        if v_half is not None:
            self._v.half = v_half


PreparedSparse.v_carrier = VCarrier.field()


def _unfilled(cls):
    return object.__new__(cls)


class _OverBuffers:
    """The lazy part of a class whose carriers are those of an ``ops.LayerBuffers`` (``over``).  Its tensors come into being
    when they are asked for; until then (``untouched``) nobody can have written to them or put others in their place.
    Objects over the same buffers share the pair of codes and FP16 copy as such, through the buffers."""

    _LAZY = frozenset(("q_int8", "k_int8", "q_scale", "k_scale", "v_scale", "_v"))
    _copied_as = None  # the class of a copy

    @classmethod
    def over(cls, buffers, **rest):
        prepared = object.__new__(cls)
        prepared.__dict__.update(rest, sequence=buffers.sequence, heads=buffers.heads, _buffers=buffers)
        return prepared

    def __getattr__(self, name):  # of what the instance does not hold (yet)
        buffers = self.__dict__.get("_buffers")
        if buffers is None or name not in _OverBuffers._LAZY:
            raise AttributeError("%r object has no attribute %r" % (type(self).__name__, name))
        if name == "_v":
            value = getattr(buffers, "v_pair", None)
            if value is None:
                value = buffers.v_pair = VCarrier(buffers.tensor("v_carrier"), buffers.v_half)
                buffers.v_half = None
        else:
            value = buffers.tensor(name)
        self.__dict__[name] = value
        return value

    @property
    def device(self):
        """Where the carriers are, without asking for one."""
        buffers = self.__dict__.get("_buffers")
        return self.q_int8.device if buffers is None else buffers.device

    def untouched(self):
        """The buffers, if no tensor of them has been handed out or replaced."""
        buffers = self.__dict__.get("_buffers")
        if buffers is None or buffers.v_half is None or not _OverBuffers._LAZY.isdisjoint(self.__dict__):
            return None
        return buffers

    def __reduce_ex__(self, protocol):
        """A copy is of the plain class.  A shallow one shares the tensors, and the pair of codes and FP16 copy as such."""
        state = {name: getattr(self, name) for name in _OverBuffers._LAZY}
        state.update((name, value) for name, value in self.__dict__.items() if name != "_buffers")
        return _unfilled, (self._copied_as,), state


class PreparedLayer(_OverBuffers, PreparedSparse):
    """A ``PreparedSparse`` over an ``ops.LayerBuffers``."""

    _copied_as = PreparedSparse


class ProjectedLayer(_OverBuffers, PreparedFusedQKV):
    """A ``PreparedFusedQKV`` over an ``ops.LayerBuffers``: what a backend of this package is handed by its projector, and
    hands on to the attention kernel by addresses.  Short blocks are bound by the host, which made seven tensors, looked at each
    of them at both ends and took them apart again for the launches: 24 heads x 900 tokens 181 -> 140 us, 24 x 2304 188 -> 168."""

    _copied_as = PreparedFusedQKV

    @property
    def v_scale(self):  # the plain class has a default, which would be found before ``__getattr__``
        held = self.__dict__
        return held["v_scale"] if "v_scale" in held else self.__getattr__("v_scale")

    @v_scale.setter
    def v_scale(self, value):
        self.__dict__["v_scale"] = value

    def untouched(self):
        """The buffers, if besides their tensors also what describes them, and the tile means, is as the contract wants it."""
        buffers = super().untouched()
        if buffers is None or (self.sequence, self.heads, self.head_dim) != (buffers.sequence, buffers.heads, HEAD_DIM):
            return None
        for means, tile in ((self.q_summary, Q_TILE), (self.k_summary, KV_TILE)):
            if (means.shape != (1, buffers.heads, -(-buffers.sequence // tile), HEAD_DIM) or means.device != buffers.device
                    or not means.is_contiguous()):
                return None
        return buffers


@dataclass
class PreparedHybrid:
    sparse: PreparedSparse
