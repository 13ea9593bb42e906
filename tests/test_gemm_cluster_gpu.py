"""GEMMs of few output tiles (a cluster of CTAs per tile, csrc/gemm_cluster_sm100.cu) against 64-bit products: every operand
orientation and epilogue at sizes around the tile (128 x 64 and 128 x 128), the K block (64) and the split of the reduction.

Tolerance: fp32 sums of K products of bf16 values: K 2^-24 of the sum of magnitudes at most, below 2^-13 relative for the
sizes here; bf16 results are rounded once more (2^-9), those behind an activation or a second operand twice.
"""
import pytest
import torch

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 64), (127, 64, 72), (129, 72, 128), (128, 128, 1024),      # one or two tiles; a K that is no whole block
    (512, 1024, 1024), (512, 512, 4096), (300, 776, 2000),            # split over two, four, eight CTAs
    (1000, 1472, 1472), (2048, 1160, 200),                            # nearly a tile per SM
])
def test_cluster_gemm(M, N, K):
    torch.manual_seed(M + N + K)
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    a, w, bias, res = bf(M, K), bf(N, K) * 0.05, bf(N), bf(M, N)
    want = a.double() @ w.double().t()
    assert rel(F.gemm(a, w), want) < 2.0 ** -8
    assert rel(F.gemm(a, w, bias=bias, residual=res), want + bias.double() + res.double()) < 2.0 ** -8
    pre = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    y = F.gemm(a, w, bias=bias.float(), act=F.ACT_GELU, preact_out=pre)
    assert rel(pre, want + bias.double()) < 2.0 ** -8
    assert rel(y, torch.nn.functional.gelu(want + bias.double(), approximate="tanh")) < 2.0 ** -7
    old = bf(M, N)
    out = old.clone()
    F.gemm(a, w, out=out, accumulate=True, alpha=0.5)
    assert rel(out, 0.5 * want + old.double()) < 2.0 ** -8
    grad, x = bf(M, N), bf(M, K)
    dx = grad.double() @ w.double()
    assert rel(F.gemm(grad, w, b_mn=True, act=F.ACT_DRELU, aux=x), dx * (x > 0)) < 2.0 ** -8
    if M % 8 == 0 or M == 1:                                          # a leading dimension in units of 8
        mg = torch.randn(N, K, device=DEV)
        start = mg.double()
        F.gemm(grad, a, out=mg, a_mn=True, b_mn=True, accumulate=True)
        assert rel(mg, start + grad.double().t() @ a.double()) < 2.0 ** -13
        if N % 8 == 0:
            wt = w.t().contiguous()                                   # B stored [K][N], A stored [K][M]
            if M % 8 == 0:
                assert rel(F.gemm(a.t().contiguous(), wt, a_mn=True, b_mn=True), want) < 2.0 ** -8
                assert rel(F.gemm(a.t().contiguous(), w, a_mn=True), want) < 2.0 ** -8
    assert native.check_status() == 0


def test_cluster_gemm_draws_the_dropout_mask_of_the_other_kernels():
    torch.manual_seed(3)
    M, N, K = 256, 512, 1024
    a, w = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    y = F.gemm(a, w, dropout_p=0.3, seed=11)
    plain = F.gemm(a, w)
    masked = native.ext().elementwise(F.EW_DROPOUT, plain, None, None, 0.3, 11)
    assert torch.equal(y == 0, masked == 0) and rel(y, masked.double()) < 2.0 ** -8


def test_cluster_gemm_is_repeatable():
    torch.manual_seed(4)
    a, w = torch.randn(512, 4096, device=DEV).bfloat16(), torch.randn(512, 4096, device=DEV).bfloat16()
    assert torch.equal(F.gemm(a, w), F.gemm(a, w))


@pytest.mark.parametrize("M,N,K", [(300, 24, 2000), (130, 16, 64), (513, 8, 512)])
@pytest.mark.parametrize("shift", [1, 2, 4])
def test_narrow_outputs_with_operands_off_a_boundary(M, N, K, shift):
    """Column views that do not start on 16 bytes (refused where 32 columns are whole)."""
    torch.manual_seed(N + shift)
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    view = lambda t: t[:, shift:shift + N]
    a, w, res, x, pre = bf(M, K), bf(N, K) * 0.05, view(bf(M, 64)), view(bf(M, 64)), view(bf(M, 64))
    want = a.double() @ w.double().t()
    assert rel(F.gemm(a, w, residual=res), want + res.double()) < 2.0 ** -8
    assert rel(F.gemm(a, w, act=F.ACT_DRELU, aux=x), want * (x > 0)) < 2.0 ** -8
    y = F.gemm(a, w, act=F.ACT_RELU, preact_out=pre)
    assert rel(pre, want) < 2.0 ** -8 and rel(y, want.relu()) < 2.0 ** -8
    with pytest.raises(RuntimeError, match="gemm"):
        F.gemm(a, bf(40, K), residual=bf(M, 64)[:, shift:shift + 40])
