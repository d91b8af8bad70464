"""Programmatic dependent launches (csrc/launch.h): every kernel launched that way waits for the kernel in
front of it, kernels that wait for other ranks are not, and a chain of short kernels keeps its order."""
from __future__ import annotations

import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "forgetrain_b200" / "csrc"


def kernels(text):
    text = re.sub(r"__(?:launch_bounds|cluster_dims)__\([^)]*\)", "", text)
    for m in re.finditer(r"__global__\s+void\s+(\w+)\s*\([^;{]*\)\s*\{", text):
        yield m.group(1), text[m.end():text.index("\n}\n", m.end())]


def test_every_dependently_launched_kernel_waits_before_it_reads():
    launched, bodies = set(), {}
    for f in CSRC.glob("*.cu"):
        text = f.read_text()
        launched |= {m.group(1) for m in re.finditer(r"launch_pdl(?:_cluster)?\(\s*(\w+)", text)}
        bodies.update(kernels(text))
    assert len(launched) > 15
    for name in launched:
        body = bodies[name]
        assert body.index("pdl_trigger();") < body.index("pdl_wait();"), name
        # nothing in front of the wait touches global memory: set-up of barriers, TMEM and indices only
        head = body[:body.index("pdl_wait();")]
        for word in ("tma_load", "tma_store", "atomicAdd", "reinterpret_cast<const bf16x8", "__ldg"):
            assert word not in head, (name, word)


def test_kernels_that_wait_for_other_ranks_are_launched_plainly():
    for f in ("comm.cu", "gemm_tp_sm100.cu"):
        text = (CSRC / f).read_text()
        assert "pdl" not in text and "<<<" in text


@pytest.mark.gpu
def test_a_chain_of_short_kernels_keeps_its_order():
    """Each op reads what the one in front has just written into a reused buffer: bitwise the result of
    the same calls with a synchronisation after each."""
    from forgetrain_b200 import ops
    T, H = 256, 256
    x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
    w = (torch.randn(H, H, device="cuda") * 0.1).to(torch.bfloat16)
    nw = torch.ones(H, device="cuda", dtype=torch.bfloat16)

    def chain(sync):
        h = x.clone()
        for _ in range(60):
            _, n, rstd = ops.add_rmsnorm_fwd(None, h, nw, 1e-5)
            sync()
            y = ops.linear_fwd(n, w)
            sync()
            dw = torch.empty(H, device="cuda")
            d = ops.rmsnorm_bwd(y, h, nw, rstd, None, dw, False)
            sync()
            h = ops.linear_dgrad(d, w)
            sync()
        return h

    assert torch.equal(chain(lambda: None), chain(torch.cuda.synchronize))
