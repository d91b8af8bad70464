"""Whole decoder blocks in one native call (csrc/layer.cu, ops/layer.py): the ctypes mirrors against the C
structs, and the calls against the op-by-op sequence."""
from __future__ import annotations

import ctypes
import re
from pathlib import Path

import pytest
import torch

HEADER = Path(__file__).resolve().parent.parent / "forgetrain_b200" / "csrc" / "layer.h"


@pytest.mark.parametrize("name", ["FtLayerFwd", "FtLayerBwdFfn", "FtLayerBwdAttn"])
def test_the_mirror_has_the_fields_of_the_struct(name):
    from forgetrain_b200.ops import layer
    body = re.search(rf"struct {name} \{{(.*?)\n\}};", HEADER.read_text(), re.S).group(1)
    want = []
    for decl in re.sub(r"//[^\n]*", "", body).split(";"):
        m = re.match(r"\s*(?:const )?(void|int|float)\b\s*(.*)", decl.strip(), re.S)
        for field in (m.group(2).split(",") if m else ()):
            kind = ctypes.c_void_p if "*" in field else {"int": ctypes.c_int, "float": ctypes.c_float}[m.group(1)]
            want.append((field.replace("*", "").strip(), kind))
    assert want == getattr(layer, name)._fields_


def test_pieces_do_not_overlap_and_are_aligned():
    from forgetrain_b200.ops.layer import _offsets
    sizes = [0, 1000, 256, 4, 0, 77]
    o = _offsets(*sizes)
    assert all(a % 256 == 0 for a in o)
    assert all(o[i] + sizes[i] <= o[i + 1] for i in range(len(sizes)))


def test_block_calls_are_for_one_rank_on_the_gpu():
    from forgetrain_b200.config import load_model_spec
    from forgetrain_b200.models.minicpm4 import MiniCPM4
    from forgetrain_b200.models.params import ParamStore
    spec = load_model_spec("tiny")
    m = MiniCPM4(spec, ParamStore(spec, "cpu", torch.float32))
    assert m._block is None and not m._block_takes((torch.zeros(256, spec.hidden_size),), 1, None)


def test_unpacking_gives_every_tensor_the_op_by_op_backward_reads():
    from forgetrain_b200.config import load_model_spec
    from forgetrain_b200.models.minicpm4 import LayerSaved
    from forgetrain_b200.ops.layer import Block, BlockSaved
    spec = load_model_spec("tiny")
    b = Block(spec, spec.heads_per_group, spec.num_query_groups)
    T, H = 512, spec.hidden_size
    sv = BlockSaved()
    sv.T, sv.offs = T, b._keep_offsets(T, True)
    sv.keep = torch.zeros(sv.offs[7], dtype=torch.uint8)
    sv.h_in = None
    sv.h_mid = sv.attn = sv.y1 = sv.act = torch.zeros(1)
    into = b.unpack(sv, LayerSaved(), 256)
    assert all(getattr(into, n) is not None for n in LayerSaved.__slots__)
    assert into.lse.shape == (2, spec.num_attention_heads, 256) and into.n1_full.shape == (T, H)
    assert into.qkv.shape == (T, spec.qkv_dim) and into.rs1.shape == into.rs2.shape == (T,)


# head dims 64 and 128; tied tables; position ids that restart; recomputation; weight gradients in line and on
# a stream of their own; a second, accumulated micro-batch
@pytest.mark.gpu
@pytest.mark.parametrize("model,seq,docs,recompute,side", [
    ("tiny", 256, False, False, True), ("0.5b", 512, True, False, True), ("0.5b", 256, False, True, False),
    ("8b", 256, True, True, True)])
def test_block_calls_against_the_op_by_op_sequence(model, seq, docs, recompute, side):
    from forgetrain_b200.config import load_model_spec
    from forgetrain_b200.models.minicpm4 import MiniCPM4
    from forgetrain_b200.models.params import ParamStore
    from forgetrain_b200.ops import _lib
    spec = load_model_spec(model, num_layers=2, vocab_size=1024, seq_length=seq, max_position_embeddings=seq)
    gen = torch.Generator(device="cuda").manual_seed(0)
    ids = torch.randint(0, 1024, (2, seq + 1), generator=gen, device="cuda")
    pos = (torch.arange(seq, device="cuda") % 100).expand(2, seq) if docs else None
    got = []
    for whole in (True, False):
        store = ParamStore(spec, "cuda", torch.bfloat16)
        store.init_random(0, "normal", 0.02)
        m = MiniCPM4(spec, store, recompute_attn=recompute, recompute_mlp=recompute)
        assert m._block is not None
        if not whole:
            m._block = None
        if side:
            m.wgrad_stream = torch.cuda.Stream()
        seen = []
        logits = m.forward(ids[:, :-1].contiguous(), pos).clone()
        for accumulate in (False, True):
            loss = m.forward_backward(ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), None, 0.5, accumulate,
                                      seen.append, pos)
        torch.cuda.synchronize()
        got.append((logits, float(loss), {n: g.clone() for n, g in store.grads.items()}, seen))
    _lib.check_status()
    (la, xa, ga, sa), (lb, xb, gb, sb) = got
    assert torch.equal(la, lb) and xa == xb and sa == sb
    for n in gb:
        # dQ and split weight gradients are summed in arrival order: bf16 roundings of d qkv may flip (2^-9)
        assert float((ga[n] - gb[n]).norm()) <= 0.01 * float(gb[n].norm()), n
    last = f"layers.{spec.num_layers - 1}.feed_forward."
    for n in ("w2.weight", "wfc1.weight"):      # in front of the first attention backward: fp32 sums only
        assert float((ga[last + n] - gb[last + n]).norm()) <= 1e-5 * float(gb[last + n].norm()), n


@pytest.mark.gpu
def test_diagnostics_and_unsupported_inputs_take_the_op_by_op_sequence():
    from forgetrain_b200.config import load_model_spec
    from forgetrain_b200.models.minicpm4 import MiniCPM4
    from forgetrain_b200.models.params import ParamStore
    spec = load_model_spec("tiny", num_layers=2, vocab_size=512, seq_length=256, max_position_embeddings=256)
    store = ParamStore(spec, "cuda", torch.bfloat16)
    store.init_random(0, "normal", 0.02)
    m = MiniCPM4(spec, store)
    ids = torch.randint(0, 512, (1, 257), device="cuda")
    m.diagnostics = {}
    m.forward_backward(ids[:, :-1].contiguous(), ids[:, 1:].contiguous())
    assert "d_fc1_last" in m.diagnostics and torch.isfinite(store.flat_grads).all()
    with pytest.raises(ValueError, match="seq"):        # still refused, by the op that does not take it
        m.forward(ids[:, :128].contiguous())
