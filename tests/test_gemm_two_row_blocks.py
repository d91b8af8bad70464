"""GEMM tiles of two 128-row blocks (csrc/gemm_sm100.cu, ``MT == 2``): the work decomposition on the
CPU, the kernel on a GPU at the edges of its tiles."""
from __future__ import annotations

import pytest
import torch

from gemm_schedule_model import G


def units(M, N, k_iters, splitk, ctas):
    """Row blocks and K range of every work unit, as ``cut_tail`` and ``decode_tile<2>`` cut them."""
    m_tiles, n_tiles = -(-M // 256), -(-N // 256)
    total = m_tiles * n_tiles * splitk
    rem = total % ctas
    cut = splitk == 1 and ctas >= 2 and rem > 0 and 2 * rem <= ctas
    split_from, total_units = (total - rem, total + rem) if cut else (total, total)
    group = G["GEMM_GROUP_M"] // 2
    for u in range(total_units):
        half, t = -1, u
        if u >= split_from:
            half, t = (u - split_from) & 1, split_from + ((u - split_from) >> 1)
        ks, r = divmod(t, m_tiles * n_tiles)
        g, inside = divmod(r, group * n_tiles)
        gm = min(m_tiles - g * group, group)
        mt, nt = g * group + inside % gm, inside // gm
        base, extra = divmod(k_iters, splitk)
        kb, kn = ks * base + min(ks, extra), base + (ks < extra)
        blocks = [2 * mt, 2 * mt + 1] if half < 0 else [2 * mt + half]
        yield blocks, nt, kb, kn


@pytest.mark.parametrize("M,N,k_iters,splitk,ctas", [(256, 256, 4, 1, 148), (300, 520, 7, 1, 148),
                                                      (16384, 1280, 3, 1, 148), (4096, 8192, 2, 1, 148),
                                                      (1280, 1024, 64, 7, 148), (73448, 1024, 1, 1, 148),
                                                      (2304, 300, 5, 1, 11), (256, 256, 1, 1, 1)])
def test_every_row_block_is_covered_once_for_every_k_step(M, N, k_iters, splitk, ctas):
    seen = set()
    for blocks, nt, kb, kn in units(M, N, k_iters, splitk, ctas):
        assert kn > 0
        for b in blocks:
            for k in range(kb, kb + kn):
                assert (b, nt, k) not in seen
                seen.add((b, nt, k))
    assert len(seen) == 2 * -(-M // 256) * -(-N // 256) * k_iters


# rows / columns that end inside a block, a last row block that lies outside the matrix as a whole (384), a
# tail wave cut into single blocks (2560 x 4096: 160 tiles on 148 CTAs), one k-step, and fewer k-steps than stages
@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(256, 256, 64), (384, 200, 72), (1000, 1032, 1024), (2560, 4096, 192),
                                   (136, 1288, 328)])
def test_two_row_blocks_against_fp32(T, N, K):
    from forgetrain_b200.ops import gemm

    def rel(a, b):
        return float((a.float() - b).norm() / b.norm())

    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16)
    dy = torch.randn(T, N, device="cuda").to(torch.bfloat16)
    # bf16 outputs: 2^-9 relative rounding of each value; fp32 ones: sums of up to 2560 products
    assert torch.equal(gemm.linear_fwd(x, w, bn=512), gemm.linear_fwd(x, w, bn=256))
    assert torch.equal(gemm.linear_dgrad(dy, w, bn=512), gemm.linear_dgrad(dy, w, bn=256))
    assert rel(gemm.linear_fwd(x, w, alpha=0.25, bn=512), 0.25 * (x.float() @ w.float().t())) < 0.004
    ref = dy.float().t() @ x.float()
    dw = gemm.linear_wgrad(dy, x, bn=512)
    assert rel(dw, ref) < 1e-5
    gemm.linear_wgrad(dy, x, out=dw, accumulate=True, bn=512, splitk=min(3, (T + 63) // 64))
    assert rel(dw, 2 * ref) < 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("T,F,K", [(4096, 8192, 2048), (4000, 8192, 2056), (768, 16384, 4096)])
def test_fc1_swiglu_with_two_row_blocks_is_bitwise_the_two_kernels(T, F, K):
    from forgetrain_b200.ops import cuda_ops, gemm
    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * 0.05).to(torch.bfloat16)
    y, act = gemm.linear_swiglu_fwd(x, w)
    assert torch.equal(y, gemm.linear_fwd(x, w, bn=256))
    assert torch.equal(act, cuda_ops.swiglu_fwd(y))


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.02, 0.3, 4.0])
@pytest.mark.parametrize("T,F,K", [(128, 128, 64), (1000, 1024, 256), (2560, 8192, 2048)])
def test_fused_activation_is_bitwise_the_divided_one_for_small_and_huge_gates(T, F, K, scale):
    """Gates up to several hundred in magnitude (underflowing and saturated sigmoids), millions of values:
    those near the middle of two bf16 numbers have to take the divided form."""
    from forgetrain_b200.ops import cuda_ops, gemm
    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * scale).to(torch.bfloat16)
    y, act = gemm.linear_swiglu_fwd(x, w)
    assert torch.equal(act, cuda_ops.swiglu_fwd(y))


# 64 gate + 64 up columns per tile: a row block that ends inside a tile, one tile, as many as there are CTAs at most
@pytest.mark.gpu
@pytest.mark.parametrize("T,F,K", [(128, 128, 64), (200, 1024, 264), (256, 4096, 1024), (1100, 1024, 256)])
def test_narrow_fc1_swiglu_is_bitwise_the_two_kernels(T, F, K):
    from forgetrain_b200.ops import cuda_ops, gemm
    x = torch.randn(T, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(2 * F, K, device="cuda") * 0.1).to(torch.bfloat16)
    y, act = gemm.linear_swiglu_fwd(x, w, alpha=0.5)
    assert torch.equal(y, gemm.linear_fwd(x, w, alpha=0.5, bn=256))
    assert torch.equal(act, cuda_ops.swiglu_fwd(y))
