"""One decoder block per native call (``csrc/layer.cu``): the same kernels as op by op, on the current
stream, without the host time of launching each from Python. CUDA, bf16, one rank (no tensor parallelism);
:class:`forgetrain_b200.models.minicpm4.MiniCPM4` runs the op-by-op sequence everywhere else.

Sequence of the reference's block: exports/train_engine_0.5B/src/training_engine_tensor/
forward.py:81-217, backward.py:125-393.
"""
from __future__ import annotations

import ctypes
import math

import torch

from . import _lib, attention, gemm

P = _lib.ptr
_PTR, _INT, _FLOAT = ctypes.c_void_p, ctypes.c_int, ctypes.c_float


def _struct(name: str, pointers: str, ints: str, floats: str):
    fields = [(n, _PTR) for n in pointers.split()] + [(n, _INT) for n in ints.split()] + \
        [(n, _FLOAT) for n in floats.split()]
    return type(name, (ctypes.Structure,), {"_fields_": fields})


# field for field the structs of csrc/layer.h
FtLayerFwd = _struct(
    "FtLayerFwd", "res x w_an w_qkv w_o w_fn w_fc1 w_2 cos sin pos h_in n1 rs1 qkv attn lse o h_mid n2 rs2 "
    "y1 act f status", "T S H n_groups g D F", "eps r scale")
FtLayerBwdFfn = _struct(
    "FtLayerBwdFfn", "dh y1 act n2 h_mid rs2 w_2 w_fc1 w_fn g_2 g_fc1 g_fn dy1 dn2 partial status",
    "T H F accumulate", "r")
FtLayerBwdAttn = _struct(
    "FtLayerBwdAttn", "dh attn lse qkv n1 h_in rs1 w_o w_qkv w_an cos sin pos g_o g_qkv g_an dattn dqkv acc "
    "delta dn1 partial status", "T S H n_groups g D accumulate", "r scale")


def _offsets(*nbytes: int) -> list[int]:
    """Starts of consecutive 256-byte aligned pieces, and the total."""
    out, at = [], 0
    for n in nbytes:
        out.append(at)
        at += (n + 255) & ~255
    out.append(at)
    return out


class BlockSaved:
    """What the backward of a block needs. ``keep`` holds h_in (when the block added its input up), n1,
    qkv, n2, rstd 1, rstd 2 and the log-sum-exp at ``offs``; ``attn``, ``y1`` and ``act`` are dropped
    (None) when they are recomputed."""
    __slots__ = ("keep", "offs", "h_in", "h_mid", "attn", "y1", "act", "T")


class Block:
    """Geometry of the decoder blocks of one model and the calls for them."""

    def __init__(self, spec, heads_per_group: int, n_groups: int):
        self.H, self.F, self.D = spec.hidden_size, spec.ffn_hidden_size, spec.head_dim
        self.G, self.g = n_groups, heads_per_group
        self.nq, self.nqkv = n_groups * heads_per_group * self.D, n_groups * (heads_per_group + 2) * self.D
        self.eps, self.r = spec.norm_epsilon, spec.mup_residual_scale
        self.scale = 1.0 / math.sqrt(self.D)
        # geometries the kernels of this sequence take; others raise from the op that does not take them
        self.supported = self.D in (64, 128) and self.F % 128 == 0 and \
            self.H in (256, 512, 1024, 2048, 4096, 8192)

    def takes(self, x: torch.Tensor, seq: int) -> bool:
        return (self.supported and x.is_cuda and x.dtype == torch.bfloat16 and x.is_contiguous()
                and x.shape[1] == self.H and seq % 256 == 0 and seq > 0 and x.data_ptr() % 16 == 0)

    def _keep_offsets(self, T: int, adds: bool) -> list[int]:
        return _offsets(T * self.H * 2 if adds else 0, T * self.H * 2, T * self.nqkv * 2, T * self.H * 2, T * 4,
                        T * 4, T * self.G * self.g * 4)

    def forward(self, w, res, x, cos, sin, pos, seq: int, keep_attn: bool, keep_mlp: bool):
        """``w``: attention-norm, qkv, output, FFN-norm, FC1, FC2 weights. Returns the block's middle
        ``h_mid``, the feed-forward branch and what the backward needs."""
        T, dev, H = x.shape[0], x.device, self.H
        sv = BlockSaved()
        sv.T = T
        sv.offs = o = self._keep_offsets(T, res is not None)
        sv.keep = torch.empty(o[7], dtype=torch.uint8, device=dev)
        k = sv.keep.data_ptr()
        sv.h_mid = torch.empty_like(x)
        f = torch.empty_like(x)       # also the attention branch, which is dead before f is written
        attn = torch.empty(T, self.nq, dtype=torch.bfloat16, device=dev)
        y1 = torch.empty(T, 2 * self.F, dtype=torch.bfloat16, device=dev)
        act = torch.empty(T, self.F, dtype=torch.bfloat16, device=dev)
        sv.h_in = x if res is None else None
        fp = f.data_ptr()
        a = FtLayerFwd(None if res is None else res.data_ptr(), x.data_ptr(), *[t.data_ptr() for t in w],
                       cos.data_ptr(), sin.data_ptr(), None if pos is None else pos.data_ptr(),
                       None if res is None else k, k + o[1], k + o[4], k + o[2], attn.data_ptr(), k + o[6], fp,
                       sv.h_mid.data_ptr(), k + o[3], k + o[5], y1.data_ptr(), act.data_ptr(), fp,
                       _lib.status_word(dev).data_ptr(), T, seq, H, self.G, self.g, self.D, self.F, self.eps,
                       self.r, self.scale)
        _lib.check_rc(_lib.lib().ft_layer_fwd(ctypes.byref(a), _lib.stream()), "ft_layer_fwd")
        sv.attn = attn if keep_attn else None
        sv.y1, sv.act = (y1, act) if keep_mlp else (None, None)
        return sv.h_mid, f, sv

    def piece(self, sv: BlockSaved, i: int, dtype, *shape) -> torch.Tensor:
        n = math.prod(shape) * dtype.itemsize
        return sv.keep[sv.offs[i]:sv.offs[i] + n].view(dtype).view(shape)

    def unpack(self, sv: BlockSaved, into, seq: int):
        """The same as separate tensors, in the attributes of ``into`` (the op-by-op sequence's record)."""
        T, bf, f32 = sv.T, torch.bfloat16, torch.float32
        into.h_in = sv.h_in if sv.h_in is not None else self.piece(sv, 0, bf, T, self.H)
        into.n1_full, into.qkv = self.piece(sv, 1, bf, T, self.H), self.piece(sv, 2, bf, T, self.nqkv)
        into.n2_full = self.piece(sv, 3, bf, T, self.H)
        into.rs1, into.rs2 = self.piece(sv, 4, f32, T), self.piece(sv, 5, f32, T)
        into.h_mid, into.attn, into.y1, into.act = sv.h_mid, sv.attn, sv.y1, sv.act
        if sv.attn is not None:
            B = T // seq
            into.lse = self.piece(sv, 6, f32, B, self.G * self.g, seq)
        return into

    def backward_ffn(self, sv: BlockSaved, dh, w, g, accumulate: bool, side) -> None:
        """Feed-forward half, ``dh`` in place. ``w``: FC2, FC1, FFN-norm weights; ``g``: their gradients;
        ``side``: stream of the weight-gradient GEMMs or None."""
        T, dev, H, F = sv.T, dh.device, self.H, self.F
        y1, act = sv.y1, sv.act
        if y1 is None:
            y1, act = gemm.linear_swiglu_fwd(self.piece(sv, 3, torch.bfloat16, T, H), w[1])
        sv.y1 = sv.act = None
        k, o = sv.keep.data_ptr(), sv.offs
        L = _lib.lib()
        parts = L.ft_rmsnorm_bwd_partials(_INT(T), _INT(H))
        q = _offsets(T * 2 * F * 2, T * H * 2, parts * H * 4)
        scratch = torch.empty(q[3], dtype=torch.uint8, device=dev)
        s = scratch.data_ptr()
        a = FtLayerBwdFfn(dh.data_ptr(), y1.data_ptr(), act.data_ptr(), k + o[3], sv.h_mid.data_ptr(), k + o[5],
                          *[t.data_ptr() for t in w], *[t.data_ptr() for t in g], s, s + q[1], s + q[2],
                          _lib.status_word(dev).data_ptr(), T, H, F, int(accumulate), self.r)
        _lib.check_rc(L.ft_layer_bwd_ffn(ctypes.byref(a), _PTR(side.cuda_stream if side is not None else None),
                                         _lib.stream()), "ft_layer_bwd_ffn")

    def backward_attn(self, sv: BlockSaved, dh, w, g, cos, sin, pos, seq: int, accumulate: bool, side) -> None:
        """Attention half, ``dh`` in place. ``w``: output, qkv, attention-norm weights; ``g``: their gradients."""
        T, dev, H, bf = sv.T, dh.device, self.H, 2
        k, o = sv.keep.data_ptr(), sv.offs
        attn, lse = sv.attn, k + o[6]
        if attn is None:
            attn, again = attention.attention_fwd(self.piece(sv, 2, torch.bfloat16, T, self.nqkv), T // seq, self.G,
                                                  self.g, self.D)
            lse = again.data_ptr()
        sv.attn = None
        L = _lib.lib()
        parts = L.ft_rmsnorm_bwd_partials(_INT(T), _INT(H))
        q = _offsets(T * self.nq * bf, T * self.nqkv * bf, T * self.nqkv * 4, 2 * T * self.G * self.g * 4, T * H * bf,
                     parts * H * 4)
        scratch = torch.empty(q[6], dtype=torch.uint8, device=dev)
        s = scratch.data_ptr()
        a = FtLayerBwdAttn(dh.data_ptr(), attn.data_ptr(), lse, k + o[2], k + o[1],
                           sv.h_in.data_ptr() if sv.h_in is not None else k, k + o[4],
                           *[t.data_ptr() for t in w], cos.data_ptr(), sin.data_ptr(),
                           None if pos is None else pos.data_ptr(), *[t.data_ptr() for t in g],
                           s, s + q[1], s + q[2], s + q[3], s + q[4], s + q[5], _lib.status_word(dev).data_ptr(),
                           T, seq, H, self.G, self.g, self.D, int(accumulate), self.r, self.scale)
        _lib.check_rc(L.ft_layer_bwd_attn(ctypes.byref(a), _PTR(side.cuda_stream if side is not None else None),
                                          _lib.stream()), "ft_layer_bwd_attn")
