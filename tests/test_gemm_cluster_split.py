"""GEMM whose reduction is split inside a thread-block cluster (csrc/gemm_sm100.cu, ``EPI_CLUSTER``): the rows a
CTA sums on the CPU, the kernel on a GPU at the edges of tiles, clusters and K ranges."""
from __future__ import annotations

import pytest
import torch


@pytest.mark.parametrize("ncta", range(1, 9))
def test_the_cluster_sums_every_row_once(ncta):
    per = -(-128 // ncta)                      # sum_partials: rows [rank * per, min(.., 128)), eight warps
    seen = [r for rank in range(ncta) for warp in range(8)
            for r in range(rank * per + warp, min(rank * per + per, 128), 8)]
    assert sorted(seen) == list(range(128))


# one tile; rows and columns that end inside a tile (columns inside a group of four lanes' vectors too: 1036, 300); as
# many k-steps as CTAs; K ranges of unequal length with a partial last k-step
@pytest.mark.gpu
@pytest.mark.parametrize("ncta", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("T,N,K", [(128, 128, 512), (200, 1032, 520), (136, 264, 1000), (512, 1024, 4096)])
def test_cluster_split_against_fp32(T, N, K, ncta):
    from forgetrain_b200.ops import gemm

    def rel(a, b):
        return float((a.float() - b).norm() / b.norm())

    bn = 1000 + ncta
    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    y = gemm.linear_fwd(x, w, alpha=0.5, bn=bn)
    assert rel(y, 0.5 * (x.float() @ w.float().t())) < 0.004       # 2^-9 relative rounding of each value
    assert torch.equal(y, gemm.linear_fwd(x, w, alpha=0.5, bn=bn))   # summed in rank order, whatever the timing
    # reduction over K here too, both operands MN-major: dy is [K, N], x is [K, T]
    dy, x2 = torch.randn(K, N, device="cuda").to(torch.bfloat16), torch.randn(K, T, device="cuda").to(torch.bfloat16)
    ref = dy.float().t() @ x2.float()
    dw = gemm.linear_wgrad(dy, x2, bn=bn)
    assert rel(dw, ref) < 1e-5
    gemm.linear_wgrad(dy, x2, out=dw, accumulate=True, bn=bn)
    assert rel(dw, 2 * ref) < 1e-5
    w3 = (torch.randn(K, N, device="cuda") * 0.05).to(torch.bfloat16)
    assert rel(gemm.linear_dgrad(x, w3, bn=bn), x.float() @ w3.float()) < 0.004


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(256, 1024, 8192), (512, 1024, 4096), (1000, 1032, 4096)])
def test_split_reductions_are_no_less_exact_and_the_forward_pass_is_not_split(T, N, K):
    from forgetrain_b200.ops import gemm

    def err(a, ref):
        return float((a.double() - ref).norm() / ref.norm())

    dy = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(K, N, device="cuda") * 0.05).to(torch.bfloat16)
    ref = dy.double() @ w.double()
    # both are dominated by the bf16 rounding of the result
    assert err(gemm.linear_dgrad(dy, w), ref) < 1.02 * err(gemm.linear_dgrad(dy, w, bn=256), ref)
    x = torch.randn(T, N, device="cuda").to(torch.bfloat16)
    ref = dy.double().t() @ x.double()          # [K, N] over T tokens: fp32 result, chains no longer than before
    before = gemm.linear_wgrad(dy, x, bn=256)
    assert err(gemm.linear_wgrad(dy, x), ref) < 1.1 * err(before, ref)
    wt = w.t().contiguous()
    assert torch.equal(gemm.linear_fwd(dy, wt), gemm.linear_fwd(dy, wt, bn=256))
    # a row of the forward result does not depend on how many rows there are
    assert torch.equal(gemm.linear_fwd(dy, wt)[:128], gemm.linear_fwd(dy[:128], wt))


# rows / columns that end inside a tile, an odd number of 64-wide boxes, a partial one, fewer k-steps than stages
@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(128, 64, 64), (200, 72, 192), (384, 328, 128), (512, 1280, 1024), (130, 136, 1000),
                                   (136, 1288, 4096)])
def test_narrow_tiles_are_bitwise_the_wide_ones(T, N, K):
    from forgetrain_b200.ops import gemm
    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    assert torch.equal(gemm.linear_fwd(x, w, alpha=0.5, bn=64), gemm.linear_fwd(x, w, alpha=0.5, bn=256))
    w2 = (torch.randn(K, N, device="cuda") * 0.05).to(torch.bfloat16)
    assert torch.equal(gemm.linear_dgrad(x, w2, bn=64), gemm.linear_dgrad(x, w2, bn=256))
