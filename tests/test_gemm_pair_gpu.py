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


# Tiles of 256 x 512: (M, N, K, fp32) with both halves whole, the second half cut or empty, rows and reduction that end inside.
WIDE = [(2048, 4608, 8192, False), (1901, 4456, 8264, False), (2040, 4200, 8200, False), (2044, 4360, 8192, False),
        (1904, 4424, 16456, True)]


@pytest.mark.parametrize("M,N,K,fp32", WIDE)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_wide_tiles(M, N, K, fp32, a_mn, b_mn):
    assert native.ext().gemm_pair_columns(M, N, K, fp32, 148) == 512
    a, b, want, bound = operands(M, N, K, a_mn, b_mn)
    d, whole = padded(M, N, torch.float32 if fp32 else torch.bfloat16)
    if fp32:
        want = want + d.double()
    F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, accumulate=fp32)
    check(d, whole, want, bound + (2.0 ** -22 if fp32 else 2.0 ** -8) * (want.abs() + 2.0 ** -20))


@pytest.mark.parametrize("M,N,K", [(2048, 4608, 8192), (1901, 4452, 8264)])
@pytest.mark.parametrize("kind", ["bias_residual_dropout", "gelu_preact", "dgelu", "accumulate"])
def test_wide_tile_epilogues(M, N, K, kind):
    """Against the kernel with one CTA per tile: the same products in the same order of the reduction, the same epilogue."""
    a, b, _, _ = operands(M, N, K, False, False)
    a = a * 0.02
    bias, rows = torch.randn(N, device=DEV).bfloat16(), [padded(M, N)[0] for _ in range(2)]
    results = []
    for mode in (0, 1):
        native.ext().gemm_set_pair_mode(mode)
        try:
            d = rows[1].clone() if kind == "accumulate" else torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
            pre = torch.zeros(M, (N + 7) // 8 * 8, device=DEV, dtype=torch.bfloat16)[:, :N]
            call = dict(bias_residual_dropout=dict(bias=bias, residual=rows[0], dropout_p=0.1, seed=5), accumulate=dict(accumulate=True),
                        gelu_preact=dict(bias=bias, act=F.ACT_GELU, preact_out=pre), dgelu=dict(act=F.ACT_DGELU, aux=rows[0]))[kind]
            if kind == "bias_residual_dropout" and N % 8:
                d = torch.empty(M, N + 4, device=DEV, dtype=torch.bfloat16)[:, :N]
                call.pop("dropout_p")
            elif N % 8:
                d = torch.empty(M, N + 4, device=DEV, dtype=torch.bfloat16)[:, :N].copy_(rows[1])
            F.gemm(a, b, out=d, **call)
            results.append((d.clone(), pre.clone()))
        finally:
            native.ext().gemm_set_pair_mode(1)
    assert native.check_status() == 0
    for one, pair in zip(*results):
        assert torch.equal(one, pair)


# Tiles of 224, 192 and 160 columns, whose last 64 columns are 32 (or none): N at and around the ends of tiles.
NARROW = [(12544, 640, 200, 224), (12541, 645, 136, 224), (9472, 384, 192, 192), (9470, 381, 72, 192), (9472, 320, 64, 160),
          (9400, 317, 200, 160)]


@pytest.mark.parametrize("M,N,K,columns", NARROW)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("fp32", [False, True])
def test_narrow_tiles(M, N, K, columns, a_mn, b_mn, fp32):
    assert native.ext().gemm_pair_columns(M, N, K, fp32, 148) == columns
    if a_mn:
        M = M // 8 * 8
    a, b, want, bound = operands(M, N, K, a_mn, b_mn)
    d, whole = padded(M, N, torch.float32 if fp32 else torch.bfloat16)
    if fp32:
        want = want + d.double()
    bias = torch.randn(N, device=DEV).bfloat16() if not fp32 else None
    if bias is not None:
        want = want + bias.double()
    F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, bias=bias, accumulate=fp32)
    check(d, whole, want, bound + (2.0 ** -22 if fp32 else 2.0 ** -8) * (want.abs() + 4))
