"""AdamW kernel, one vector per thread: sizes around a CTA's 1024 elements, segments that begin anywhere."""
from __future__ import annotations

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("n,ends", [(4, [4]), (1024, [1024]), (1028, [1, 1023, 1028]), (4096, [1024, 2048, 4096]),
                                    (10240, [7, 8, 1000, 1025, 5001, 5002, 9999, 10240]), (2052, [2049, 2052])])
def test_adamw_against_the_statement_per_segment(n, ends):
    from forgetrain_b200.ops import cuda_ops as C
    from forgetrain_b200.ops import reference as R
    p, g = torch.randn(n, device="cuda"), torch.randn(n, device="cuda")
    m, v = torch.randn(n, device="cuda") * 0.1, torch.rand(n, device="cuda") * 0.1
    wd = [0.1 * (i % 3) for i in range(len(ends))]
    lrm = [1.0 / (1 + i) for i in range(len(ends))]
    rp, rm, rv, rb = p.clone(), m.clone(), v.clone(), torch.empty(n, device="cuda", dtype=torch.bfloat16)
    a = 0
    for e, w, q in zip(ends, wd, lrm):
        R.adamw_step(rp[a:e], rm[a:e], rv[a:e], g[a:e], rb[a:e], 1e-2 * q, 0.9, 0.95, 1e-8, w, 3, 0.7)
        a = e
    hyper = torch.tensor([1e-2, 0.9, 0.95, 1e-8, 1 - 0.9 ** 3, 1 - 0.95 ** 3, 0.7, 0.0], device="cuda")
    b = torch.empty(n, device="cuda", dtype=torch.bfloat16)
    C.adamw_flat(p, m, v, g, b, hyper, torch.tensor(ends, device="cuda"), torch.tensor(wd, device="cuda"),
                 torch.tensor(lrm, device="cuda"))
    for x, y in ((p, rp), (m, rm), (v, rv)):
        assert torch.allclose(x, y, rtol=2e-6, atol=2e-7)      # a few roundings of fp32 sums of O(1) values
    assert torch.allclose(b.float(), rb.float(), rtol=2 ** -8, atol=1e-6)
