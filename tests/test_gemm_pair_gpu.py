"""The GEMM on pairs of SMs (csrc/gemm2_sm100.cu) where its tiles and its epilogues end: outputs that are no whole tiles, row
pitches above N, fp32 outputs that are written or added to, against 64-bit products.

Tolerance, element by element: the fp32 sum of K products is off by at most K 2^-23 of the sum of their magnitudes; the value that
is added to rounds once more (2^-24 of the result), a bf16 result by 2^-8.
"""
import pytest
import torch

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def padded(rows, cols, dtype=torch.bfloat16):
    """A random [rows, cols] view of a matrix with a longer pitch, the columns behind it marked, and the whole."""
    whole = torch.full((rows, (cols + 7) // 8 * 8 + 8), 77.0, device=DEV, dtype=dtype)
    whole[:, :cols] = torch.randn(rows, cols, device=DEV)
    return whole[:, :cols], whole


def operands(M, N, K, a_mn, b_mn):
    torch.manual_seed(M + N + K)
    a, _ = padded(*((K, M) if a_mn else (M, K)))
    b, _ = padded(*((K, N) if b_mn else (N, K)))
    x, y = (a.t() if a_mn else a).double(), (b.t() if b_mn else b).double()
    return a, b, x @ y.t(), (x.abs() @ y.abs().t()) * (K * 2.0 ** -23)


def check(got, whole, want, bound):
    assert (whole[:, got.shape[1]:] == 77).all()
    assert float(((got.double() - want).abs() - bound).max()) <= 0
    assert native.check_status() == 0


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [
    (9472, 256, 64, False, False),                                   # whole tiles, one K block
    (2557, 1096, 200, False, False), (2312, 1300, 136, True, True),   # rows, columns and reduction end inside
    (1901, 1286, 264, False, True), (1904, 1217, 72, True, False),    # the last 64 columns by elements: 6 and 1 left
])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("bias", [False, True])
def test_fp32_outputs(M, N, K, a_mn, b_mn, accumulate, bias):
    a, b, want, bound = operands(M, N, K, a_mn, b_mn)
    d, whole = padded(M, N, torch.float32)
    bb = torch.randn(N, device=DEV) if bias else None
    if bias:
        want = want + bb.double()
    if accumulate:
        want = want + d.double()
    F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, bias=bb, accumulate=accumulate)
    check(d, whole, want, bound + 2.0 ** -22 * (want.abs() + 4))
