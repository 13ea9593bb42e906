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
    (1000, 1472, 1472), (2048, 1160, 200),                            # nearly a tile per SM; a forward on SM pairs
])
def test_gemms_of_a_small_layer(M, N, K):
    """Forward, input gradient and weight gradient at the sizes of small layers, whichever kernel takes each."""
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


def padded(rows, cols, dtype=torch.bfloat16, fill=None):
    """A [rows, cols] view of a matrix with a longer pitch (a multiple of 8), the columns behind it marked, and the whole."""
    whole = torch.full((rows, (cols + 7) // 8 * 8 + 8), 77.0, device=DEV, dtype=dtype)
    if fill is not None:
        whole[:, :cols] = fill
    return whole[:, :cols], whole


# Every pair of tile width and slices, and N that is no multiple of four: the last columns go by elements.
PLANS = {(127, 70, 64): (64, 1), (39, 40, 64): (64, 1), (130, 70, 136): (64, 2), (130, 70, 1032): (64, 4), (127, 131, 4104): (64, 8),
         (901, 1157, 64): (128, 1), (519, 1030, 1032): (128, 2), (901, 776, 1032): (128, 2), (130, 1157, 1032): (128, 4),
         (261, 773, 1032): (128, 4), (130, 515, 4104): (128, 8), (39, 776, 4104): (128, 8)}


@pytest.mark.parametrize("M,N,K", PLANS)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_every_plan_and_epilogue_of_the_cluster_gemm(M, N, K, a_mn, b_mn):
    """Element by element, in buffers with a pitch above N.  The fp32 sum of K products is off by at most K 2^-23 of the sum of
    their magnitudes; a bf16 result by 2^-8 of the values that are rounded on the way to it (result, pre-activation).  The
    activations use the hardware tanh, good to 2^-10.9 absolutely."""
    torch.manual_seed(M + N + K)
    gen = lambda r, c, scale=1.0: torch.randn(r, c, device=DEV) * scale
    a, _ = padded(*((K, M) if a_mn else (M, K)), fill=gen(*((K, M) if a_mn else (M, K))))
    b, _ = padded(*((K, N) if b_mn else (N, K)), fill=gen(*((K, N) if b_mn else (N, K)), 0.05))
    bias, (res, _), (x, _) = torch.randn(N, device=DEV), padded(M, N, fill=gen(M, N)), padded(M, N, fill=gen(M, N))
    A, B = (a.t() if a_mn else a).double(), (b if b_mn else b.t()).double()
    prod, slack = A @ B, K * 2.0 ** -23 * (A.abs() @ B.abs())
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def run(dtype=torch.bfloat16, start=None, act=F.ACT_NONE, with_bias=None, residual=None, aux=None, pre=None, **kw):
        out, whole = padded(M, N, dtype, start)
        address = lambda t: 0 if t is None else t.data_ptr()
        plan = native.ext().gemm_route(M, N, K, dtype == torch.float32, bool(kw.get("accumulate")), act, address(with_bias),
                                       address(aux), address(pre), address(residual), 0.0, sms)
        assert tuple(plan) == (2, *PLANS[M, N, K])
        F.gemm(a, b, out=out, a_mn=a_mn, b_mn=b_mn, act=act, bias=with_bias, residual=residual, aux=aux, preact_out=pre, **kw)
        assert bool((whole[:, N:] == 77.0).all())
        return out.double()

    def near(got, want, *rounded, extra=0.0):
        tol = slack + extra + 2.0 ** -8 * sum((r.abs() for r in rounded), torch.zeros_like(want))
        assert bool(((got - want).abs() <= tol + 1e-30).all())

    want = prod + bias.double() + res.double()
    near(run(with_bias=bias, residual=res), want, want)
    want = prod + bias.bfloat16().double() + res.double()
    near(run(with_bias=bias.bfloat16(), residual=res), want, want)
    pre, pre_whole = padded(M, N)
    want = prod + bias.double()
    gelu = torch.nn.functional.gelu(want, approximate="tanh")
    near(run(act=F.ACT_GELU, with_bias=bias, pre=pre), gelu, gelu, extra=slack + 2.0 ** -10 * want.abs())
    near(pre.double(), want, want)
    assert bool((pre_whole[:, N:] == 77.0).all())
    want = prod * (x > 0)
    near(run(act=F.ACT_DRELU, aux=x), want, want)
    xd = x.double().requires_grad_(True)
    d, = torch.autograd.grad(torch.nn.functional.gelu(xd, approximate="tanh").sum(), xd)
    want = prod * d
    near(run(act=F.ACT_DGELU, aux=x), want, want, extra=0.2 * slack + 2.0 ** -9 * (1 + x.double().square()) * prod.abs())
    start = torch.randn(M, N, device=DEV)
    near(run(torch.float32, start, accumulate=True), prod + start.double(), extra=2.0 ** -23 * (prod.abs() + start.abs()))
    old = start.bfloat16()
    want = 0.5 * prod + old.double()
    near(run(start=old, accumulate=True, alpha=0.5), want, want)
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
