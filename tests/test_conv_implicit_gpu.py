"""k x k convolutions whose patches are gathered inside the GEMM, at the edges of what they take, against 64-bit torch.

Operands are bf16 and enter the tensor core exactly; sums are fp32.  Outputs in bf16 carry one rounding (2^-9 relative), the
fp32 filter gradient the rounding of its sum (below 2^-14 for up to 2^18 terms in blocks of 16).
"""
import pytest
import torch
import torch.nn.functional as TF

from superscaler_b200.ops import conv as C
from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu


def _rel(a, e):
    return float((a.detach().double() - e).norm() / e.norm())


@pytest.mark.parametrize("N,H,W,Cin,Cout,k,stride,pad,plan", [
    (16, 28, 28, 320, 640, 3, 1, 1, 3),      # rows a multiple of the tile; the filter gradient keeps its patch matrix
    (3, 56, 56, 512, 512, 3, 1, 1, 3),       # 9408 pixels: last tile ragged
    (61, 7, 7, 1280, 1280, 3, 1, 1, 7),      # tiles span several images; all three passes
    (40, 14, 14, 328, 264, 3, 1, 1, 3),      # channel blocks of 64 reach past the last channel
    (64, 28, 28, 640, 640, 3, 2, 1, 5),      # strided: input gradient through col2im
    (33, 17, 23, 640, 640, 3, 1, 1, 7),      # odd image sides
    (20, 28, 28, 512, 512, 5, 1, 2, 7),      # 5 x 5
    (24, 28, 28, 512, 640, 3, 1, 0, 7),      # no padding: the gradient's map has positive reach on both sides
    (2, 14, 14, 64, 64, 3, 1, 1, 0),         # too small: patch matrix
])
def test_convolution_passes(N, H, W, Cin, Cout, k, stride, pad, plan):
    assert native.ext().conv_plan(N, H, W, Cin, Cout, k, k, stride, pad) == plan
    g = torch.Generator(device="cuda").manual_seed(N * 1000 + Cin)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    x = r(N, H, W, Cin).bfloat16().requires_grad_(True)
    w = torch.nn.Parameter((r(Cout, k * k * Cin) * (k * k * Cin) ** -0.5).bfloat16())
    w.main_grad = torch.ones(Cout, k * k * Cin, device="cuda")
    y = C.conv2d(x, w, k, k, stride, pad)
    dy = r(*y.shape).bfloat16()
    y.backward(dy)
    xd, wd = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    xp, w4 = TF.pad(xd, (0, 0, pad, pad, pad, pad)), wd.view(Cout, k, k, Cin)
    Ho, Wo = y.shape[1:3]
    want = 0
    for i in range(k):
        for j in range(k):
            want = want + xp[:, i:i + stride * (Ho - 1) + 1:stride, j:j + stride * (Wo - 1) + 1:stride] @ w4[:, i, j].t()
    dx, dw = torch.autograd.grad(want, (xd, wd), dy.double())
    assert _rel(y, want.detach()) < 2.0 ** -8
    assert _rel(x.grad, dx) < (2.0 ** -8 if plan & 2 else 2.0 ** -7)     # col2im adds bf16-rounded taps
    assert _rel(w.main_grad - 1.0, dw) < 2.0 ** -12                       # accumulated onto ones: one more rounding
    assert native.check_status() == 0


@pytest.mark.parametrize("N,H,W,Cin,Cout,k,stride,pad", [
    (61, 7, 7, 1280, 1280, 3, 1, 1),         # all three passes gather from the activation
    (16, 28, 28, 320, 640, 3, 1, 1),         # the filter gradient builds its patch matrix in the backward
    (2, 14, 14, 64, 64, 3, 1, 1),            # patch matrix throughout
])
@pytest.mark.parametrize("filter_grad", [True, False])
def test_input_may_change_before_the_backward(N, H, W, Cin, Cout, k, stride, pad, filter_grad):
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()
    leaf, w = r(N, H, W, Cin).requires_grad_(True), r(Cout, k * k * Cin)
    w.requires_grad_(filter_grad)
    got = []
    for change in (False, True):
        x = leaf * 1
        y = C.conv2d(x, w, k, k, stride, pad)
        if change:
            x.zero_()
        got.append(torch.autograd.grad(y, (leaf, w) if filter_grad else (leaf,), torch.ones_like(y)))
    for a, b in zip(*got):
        assert torch.equal(a, b)
