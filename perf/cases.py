"""The work this engine is timed on: training steps and evaluation passes through its public calls.

A case is a dict of plain values. ``do`` says which call is made:

* ``train``      ``Trainer.train_step``: forward, loss, backward, gradient norm and clip, AdamW, over
                 ``accum`` micro-batches of ``batch`` x ``seq`` tokens;
* ``logits``     ``Trainer.forward_logits``: the forward pass of an evaluation loop;
* ``attention``  ``ops.attention_fwd`` + ``ops.attention_bwd`` on an interleaved QKV buffer.

Model shapes are the built-in specs, with the number of layers cut where a whole 8B optimizer state
would not fit one GPU; the vocabulary is the spec's or any other multiple of 8. Token ids are uniform
and the weights N(0, 0.02), as in ``bench.py``.
"""
from __future__ import annotations

import math

import torch

from forgetrain_b200 import ops
from forgetrain_b200.config import load_model_spec
from forgetrain_b200.engine_config import from_spec
from forgetrain_b200.parallel.topology import Topology
from forgetrain_b200.trainer import Trainer

LAYERS = {"tiny": 4, "0.5b": 24, "8b": 2}
VOCAB = {"tiny": 4096, "0.5b": 73448, "8b": 73448}


def _case(name, do, model, batch, seq, **more):
    c = {"do": do, "model": model, "layers": LAYERS[model], "vocab": VOCAB[model], "batch": batch, "seq": seq,
         "accum": 1, "docs": False, "recompute": False, "graph": False, "mtp": 0}
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the plumbing model (tied tables), micro-batch 2: launch latency and host work only
        _case("train-tiny-2x256", "train", "tiny", 2, 256),
        # the 0.5B model on one short text: a fine-tuning step that is far from filling the GPU
        _case("train-0.5b-1x512", "train", "0.5b", 1, 512),
        # the same scale of work replayed from the whole-step CUDA graph, the switch for small steps
        _case("train-0.5b-1x1024-graph", "train", "0.5b", 1, 1024, graph=True),
        # packed documents: position ids restart, a fifth of the targets masked, an odd batch and length
        _case("train-0.5b-3x1280-docs", "train", "0.5b", 3, 1280, docs=True),
        # a global batch taken as accumulated micro-batches
        _case("train-0.5b-4x1x2048-accum", "train", "0.5b", 1, 2048, accum=4),
        # multi-token prediction with one extra layer, the reference's other training objective
        _case("train-0.5b-2x2048-mtp", "train", "0.5b", 2, 2048, mtp=1),
        # the benchmark step: sequence 4096, micro-batch 4
        _case("train-0.5b-4x4096", "train", "0.5b", 4, 4096),
        # 8B geometry (head dim 128, hidden 4096): wide GEMMs
        _case("train-8b-1x4096", "train", "8b", 1, 4096, layers=4),
        # 8B geometry, long sequence, activations recomputed to save memory
        _case("train-8b-1x8192-recompute", "train", "8b", 1, 8192, recompute=True),
        # evaluation: one short text, and a batch of full sequences
        _case("logits-0.5b-1x256", "logits", "0.5b", 1, 256),
        _case("logits-0.5b-4x4096", "logits", "0.5b", 4, 4096),
        # attention by itself, 8B heads at the long sequence of the kernel benchmark
        _case("attention-8b-4x8192", "attention", "8b", 4, 8192),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    do = rng.choice(["train", "train", "train", "train", "logits", "logits", "attention"])
    model = rng.choice(["tiny", "0.5b", "0.5b", "0.5b", "8b"]) if do != "attention" else rng.choice(["0.5b", "8b"])
    seq = 256 * _log_int(rng, 1, 32)
    batch = _log_int(rng, 1, 12)
    more = {}
    if do != "attention":
        more["vocab"] = VOCAB[model] if rng.random() < 0.5 else 8 * _log_int(rng, 512, 9181)
        more["docs"] = rng.random() < 0.3
        if model == "8b":
            more["layers"] = rng.randint(1, 4)
    if do == "train":
        option = rng.choice(["", "", "accum", "recompute", "graph", "mtp"])
        if option == "accum":
            more["accum"] = rng.randint(2, 6)
        elif option == "mtp" and model == "0.5b":
            more["mtp"] = 1
        elif option in ("recompute", "graph"):
            more[option] = True
    # no case is more work than the benchmark step; it and the long attention bound the range
    while True:
        c = _case("", do, model, batch, seq, **more)
        most = _BENCH if do != "attention" else _LONG
        if work(c)["flops"] <= work(most)["flops"] and c["accum"] * batch * seq <= 32768:
            return c
        if batch > 1:
            batch -= 1
        elif c["accum"] > 2:
            more["accum"] -= 1
        else:
            seq -= 256


_BENCH = _case("", "train", "0.5b", 4, 4096)
_LONG = _case("", "attention", "8b", 4, 8192)


def _spec(case):
    return load_model_spec(case["model"], num_layers=case["layers"], vocab_size=case["vocab"],
                           seq_length=case["seq"], max_position_embeddings=case["seq"])


def _micro_batch(case, gen, dev):
    B, S = case["batch"], case["seq"]
    ids = torch.randint(0, case["vocab"], (B, S + 1), generator=gen, device=dev)
    mb = {"tokens": ids[:, :-1].contiguous(), "labels": ids[:, 1:].contiguous(),
          "loss_mask": torch.ones(B, S, device=dev)}
    if case["docs"]:
        # documents of 1 to S tokens: a position id is the distance to the start of its document
        at = torch.arange(S, device=dev).expand(B, S)
        first = (torch.rand(B, S, generator=gen, device=dev) < 4.0 / S) | (at == 0)
        mb["position_ids"] = (at - torch.where(first, at, 0).cummax(dim=1).values).to(torch.int32)
        mb["loss_mask"] = (torch.rand(B, S, generator=gen, device=dev) >= 0.2).float()
    return mb


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    if case["do"] == "attention":
        sp = load_model_spec(case["model"])
        T = case["batch"] * case["seq"]
        qkv = torch.randn(T, sp.qkv_dim, generator=gen, device=dev).to(torch.bfloat16)
        dout = torch.randn(T, sp.q_dim, generator=gen, device=dev).to(torch.bfloat16)
        return {"case": case, "qkv": qkv, "dout": dout,
                "geometry": (case["batch"], sp.num_query_groups, sp.heads_per_group, sp.head_dim)}
    spec = _spec(case)
    # the spec's own learning-rate schedule (2000 warm-up steps for the 0.5B and 8B models)
    cfg = from_spec(spec, dtype="bf16", init_scheme="normal", init_std=0.02, recompute_attn=case["recompute"],
                    recompute_mlp=case["recompute"], full_step_cuda_graph=case["graph"],
                    mtp_num_layers=case["mtp"])
    trainer = Trainer(spec, cfg, Topology(device=dev), seq_length=case["seq"],
                      micro_batch_size=case["batch"], seed=seed)
    batches = [_micro_batch(case, gen, dev) for _ in range(case["accum"])]
    if case["graph"]:    # eager warm-up steps, then the one that captures: once per run of a program
        for _ in range(cfg.step_cuda_graph_warmup + 1):
            trainer.train_step(batches)
    return {"case": case, "trainer": trainer, "batches": batches}


def run(state):
    do = state["case"]["do"]
    if do == "attention":
        qkv, geometry = state["qkv"], state["geometry"]
        out, lse = ops.attention_fwd(qkv, *geometry)
        return out, lse, ops.attention_bwd(state["dout"], qkv, out, lse, *geometry)
    trainer = state["trainer"]
    if do == "logits":
        batch = state["batches"][0]
        return trainer.forward_logits(batch["tokens"], batch.get("position_ids"))
    step = trainer.train_step(state["batches"])
    opt = trainer.opt
    return {"loss": step["loss"], "grad_norm": step["grad_norm"], "grads": trainer.store.flat_grads,
            "params": trainer.store.flat_params, "master": opt.master, "exp_avg": opt.exp_avg}


def work(case):
    sp = load_model_spec(case["model"], num_layers=case["layers"], vocab_size=case["vocab"])
    B, S = case["batch"], case["seq"]
    T = B * S
    attn = 2.0 * T * S * sp.q_dim                # causal: half of Q K^T and of P V
    if case["do"] == "attention":
        # five products backward (S again, dP, dQ, dK, dV) for two forward; qkv and the output gradient are
        # read, output, log-sum-exp and the gradient of qkv written
        return {"bytes": 2.0 * T * (2 * sp.qkv_dim + 2 * sp.q_dim) + 4.0 * T * sp.num_attention_heads,
                "flops": 3.5 * attn}
    h = sp.hidden_size
    layer = 2.0 * T * h * (sp.qkv_dim + sp.q_dim + 3 * sp.ffn_hidden_size)
    head = 2.0 * T * h * sp.vocab_size
    params = sp.num_parameters(case["mtp"])
    if case["do"] == "logits":
        # weights and ids in, logits out; only the embedding rows that are looked up are needed
        table = 0 if sp.tie_embeddings else sp.vocab_size * h
        return {"bytes": 2.0 * (params - table) + 2.0 * T * (h + sp.vocab_size),
                "flops": sp.num_layers * (layer + attn) + head}
    one = (sp.num_layers + case["mtp"]) * (3 * layer + 3.5 * attn) + (1 + case["mtp"]) * 3 * head
    one += case["mtp"] * 3 * 4.0 * T * h * h
    # bf16 weights in and out, fp32 gradients out, master weights and both moments in and out
    return {"bytes": params * (2 + 2 + 4 + 24.0), "flops": case["accum"] * one}


def tolerance(case):
    # bf16 activations and gradients through 2 to 25 layers. Against the same pass with every value in
    # fp32 the gradients of the 0.5B and 8B models are off by 0.020 to 0.022 (2-norm; 1.7 for the largest
    # single value, which is small itself), the tiny model's by 0.006, the logits by 0.017; two runs on the
    # same inputs are 0.009 apart (0.021 a few steps later), through the order of fp32 sums.
    if case["do"] == "attention":
        return {"rel": 0.01, "max": 0.3}
    if case["do"] == "logits":
        return {"rel": 0.025, "max": 0.4}
    return {"rel": 0.03, "max": 0.9}
