"""The GEMM on pairs of SMs (csrc/gemm2_sm100.cu) where its tiles and its epilogues end: outputs that are no whole tiles, row
pitches above N, every width of a tile, fp32 outputs that are written or added to.

Operands are small whole numbers: products, their sums (below 2^24) and what they are added to are exact in fp32, so an fp32 output
has to equal the 64-bit result and a bf16 output its one rounding.  Epilogues with activations are compared bit for bit with the
kernel with one CTA per tile: the same products in the same order of the reduction, the same arithmetic behind it.
"""
import pytest
import torch

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"
LAYOUTS = [(False, False), (False, True), (True, True), (True, False)]


def view(values, lines=False):
    """`values` as a view of a matrix with a longer pitch (whole lines of 128 bytes, or off them), the columns behind it marked."""
    rows, cols = values.shape
    pitch = (cols + 63) // 64 * 64 + 64 if lines else (cols + 63) // 64 * 64 + 8
    whole = torch.full((rows, pitch), 77.0, device=DEV, dtype=values.dtype)
    whole[:, :cols] = values
    return whole[:, :cols], whole


def whole_numbers(rows, cols, most, dtype=torch.bfloat16):
    return torch.randint(-most, most + 1, (rows, cols), device=DEV).to(dtype)


def operands(M, N, K, a_mn, b_mn, lines=False, random=False):
    torch.manual_seed(M + N + K)
    make = (lambda *s: torch.randn(*s, device=DEV).bfloat16()) if random else (lambda *s: whole_numbers(*s, 2))
    a, _ = view(make(K, M) if a_mn else make(M, K), lines)
    b, _ = view(make(K, N) if b_mn else make(N, K), lines)
    if random:
        return a, b, None
    x, y = (a.t() if a_mn else a).double(), (b.t() if b_mn else b).double()
    return a, b, x @ y.t()


def columns(M, N, K, fp32, b_mn, lines=False):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert native.ext().gemm_route(M, N, K, fp32, False, 0, 0, 0, 0, 0, 0.0, sms)[0] == 1
    return native.ext().gemm_pair_columns(M, N, K, fp32, sms, b_mn, lines)


def check(got, whole, want):
    assert torch.equal(got, want.to(got.dtype))              # (exact in fp32: one rounding to bf16)
    assert (whole[:, got.shape[1]:] == 77).all()
    assert native.check_status() == 0


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [
    (9472, 512, 64, False, False), (9472, 512, 128, True, True),       # whole tiles, one K block and two
    (2557, 1782, 200, False, False), (2312, 1670, 136, True, True),    # rows, columns and reduction end inside
    (1901, 2214, 264, False, True), (1904, 2177, 72, True, False),     # the last 64 columns by elements: 38 and 1 left
])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("bias", [False, True])
def test_fp32_outputs(M, N, K, a_mn, b_mn, accumulate, bias):
    assert columns(M, N, K, True, b_mn) == 256
    a, b, want = operands(M, N, K, a_mn, b_mn)
    d, whole = view(whole_numbers(M, N, 1000, torch.float32))
    bb = whole_numbers(1, N, 50, torch.float32)[0] if bias else None
    if bias:
        want = want + bb.double()
    if accumulate:
        want = want + d.double()
    F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, bias=bb, accumulate=accumulate)
    check(d, whole, want)


# Tiles of 256 x 512: (M, N, K, fp32) with both halves whole, the second half cut or empty, rows and reduction that end inside.
WIDE = [(2048, 4608, 8192, False), (1901, 4456, 8264, False), (2040, 4200, 8200, False), (2044, 4360, 8192, False),
        (1904, 4424, 16456, True)]


@pytest.mark.parametrize("M,N,K,fp32", WIDE)
@pytest.mark.parametrize("a_mn,b_mn", LAYOUTS)
def test_wide_tiles(M, N, K, fp32, a_mn, b_mn):
    assert columns(M, N, K, fp32, b_mn) == 512
    a, b, want = operands(M, N, K, a_mn, b_mn)
    d, whole = view(whole_numbers(M, N, 1000, torch.float32 if fp32 else torch.bfloat16))
    if fp32:
        want = want + d.double()
    F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, accumulate=fp32)
    check(d, whole, want)


# Tiles of 224, 192 and 160 columns, whose last 64 columns are 32 (or none): N at and around the ends of tiles.
NARROW = [(12544, 640, 200, 224), (12541, 645, 136, 224), (9472, 384, 192, 192), (9470, 381, 72, 192), (9472, 320, 64, 160),
          (9400, 317, 200, 160)]


@pytest.mark.parametrize("M,N,K,width", NARROW)
@pytest.mark.parametrize("a_mn,b_mn", LAYOUTS)
@pytest.mark.parametrize("fp32", [False, True])
def test_narrow_tiles(M, N, K, width, a_mn, b_mn, fp32):
    assert columns(M, N, K, fp32, b_mn, lines=True) == width
    a, b, want = operands(M, N, K, a_mn, b_mn, lines=True)
    d, whole = view(whole_numbers(M, N, 1000, torch.float32 if fp32 else torch.bfloat16))
    bias = whole_numbers(1, N, 50)[0] if not fp32 else None
    want = want + (d if fp32 else bias).double()
    F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, bias=bias, accumulate=fp32)
    check(d, whole, want)


@pytest.mark.parametrize("M,N,K,width", [(2048, 4608, 8192, 512), (1901, 4452, 8264, 512), (2557, 1782, 200, 256), *NARROW])
@pytest.mark.parametrize("kind", ["bias_residual_dropout", "residual", "gelu_preact", "dgelu", "drelu", "accumulate", "fp32_gelu", "fp32_residual"])
@pytest.mark.parametrize("a_mn,b_mn", LAYOUTS[:3])
def test_epilogues(M, N, K, width, kind, a_mn, b_mn):
    """(an fp32 output takes the wide tile from longer reductions on: 256 columns here)"""
    fp32 = kind.startswith("fp32")
    assert columns(M, N, K, fp32, b_mn, lines=True) == (width if not fp32 or width != 512 else 256)
    if kind == "bias_residual_dropout" and N % 8:
        pytest.skip("dropout takes a dense output, whose rows have to start on 16 bytes")
    a, b, _ = operands(M, N, K, a_mn, b_mn, lines=True, random=True)
    a.mul_(0.02)
    bias, rows, old = torch.randn(N, device=DEV).bfloat16(), view(torch.randn(M, N, device=DEV).bfloat16())[0], torch.randn(M, N, device=DEV)
    call = dict(bias_residual_dropout=dict(bias=bias, residual=rows, dropout_p=0.1, seed=5), residual=dict(residual=rows),
                gelu_preact=dict(bias=bias, act=F.ACT_GELU), dgelu=dict(act=F.ACT_DGELU, aux=rows), drelu=dict(act=F.ACT_DRELU, aux=rows),
                accumulate=dict(accumulate=True), fp32_gelu=dict(bias=bias, act=F.ACT_GELU), fp32_residual=dict(residual=rows))[kind]
    results = []
    for mode in (0, 1):
        native.ext().gemm_set_pair_mode(mode)
        try:
            d, whole = view(old if fp32 else old.bfloat16())
            pre, pre_whole = view(torch.zeros(M, N, device=DEV, dtype=torch.bfloat16))
            if kind == "bias_residual_dropout":
                d = whole = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
            F.gemm(a, b, out=d, a_mn=a_mn, b_mn=b_mn, **call, **(dict(preact_out=pre) if kind == "gelu_preact" else {}))
            results.append((whole, pre_whole))
        finally:
            native.ext().gemm_set_pair_mode(1)
    assert native.check_status() == 0
    for one, pair in zip(*results):
        assert torch.equal(one, pair)


@pytest.mark.parametrize("p", [0.004, 0.1, 0.5, 0.998])
@pytest.mark.parametrize("M,N,K,route", [(300, 776, 128, 2), (2000, 64, 512, 0), (2560, 1792, 64, 1), (9472, 320, 64, 1)])
def test_dropout_mask_is_the_elementwise_kernels(M, N, K, route, p):
    """Whichever kernel takes the product, at the smallest and largest probabilities too."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert native.ext().gemm_route(M, N, K, False, False, 0, 0x1000, 0, 0, 0, p, sms)[0] == route
    zeros = lambda r: torch.zeros(r, K, device=DEV, dtype=torch.bfloat16)
    y = F.gemm(zeros(M), zeros(N), bias=torch.ones(N, device=DEV).bfloat16(), dropout_p=p, seed=123)
    want = native.ext().elementwise(F.EW_DROPOUT, torch.ones(M, N, device=DEV).bfloat16(), None, None, p, 123)
    assert torch.equal(y, want)
    kept = max(1, int((1 - p) * 256 + 0.5)) / 256                             # in steps of 1 / 256
    assert abs(float((want != 0).float().mean()) - kept) < 6 * (0.25 / (M * N)) ** 0.5
