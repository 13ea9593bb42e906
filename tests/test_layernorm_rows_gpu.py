"""LayerNorm forward for rows held in the registers of a warp: lengths that do not fill the last vector of every lane, values kept
as fp32 and packed (csrc/layernorm.cu), against 64-bit LayerNorm.  Tolerance: one rounding to bf16 (2^-9) of every result."""
import pytest
import torch

from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H", [8, 248, 256, 264, 768, 1016, 1472, 1800, 2048, 2056, 3080, 4096, 4104])
@pytest.mark.parametrize("rows", [1, 7, 2369, 5003])
@pytest.mark.parametrize("with_residual", [False, True])
def test_layernorm_forward_row_lengths(H, rows, with_residual):
    torch.manual_seed(H + rows)
    x = (torch.randn(rows, H, device=DEV) * 2 + 3).bfloat16()
    r = torch.randn(rows, H, device=DEV).bfloat16() if with_residual else None
    g, b = torch.randn(H, device=DEV), torch.randn(H, device=DEV)
    out = native.ext().layernorm_fwd(x, r, g, b, 1e-5)
    xs = x
    if with_residual:
        xs = out[3]
        assert torch.equal(xs, (x.float() + r.float()).bfloat16())
    d = xs.double()
    want = torch.nn.functional.layer_norm(d, (H,), g.double(), b.double(), 1e-5)
    assert float((out[0].double() - want).norm()) <= 2.0 ** -8 * float(want.norm())
    assert float((out[1].double() - d.mean(-1)).abs().max()) < 1e-5
    rstd = 1.0 / torch.sqrt(d.var(-1, unbiased=False) + 1e-5)
    assert float(((out[2].double() - rstd) / rstd).abs().max()) < 1e-4


@pytest.mark.parametrize("H,rows", [(8, 7104), (248, 7105), (264, 7106), (512, 9001),              # a warp per row, three at a time
                                    (1288, 2220), (1472, 2221), (1536, 2370),                      # three warps per row
                                    (1544, 1776), (1800, 1777), (2048, 1778), (2048, 5003),        # four
                                    (776, 7104), (960, 7105), (1024, 7999), (1032, 4440), (1280, 5003),  # two and three, of two rounds
                                    (512, 7103), (1536, 2219), (2048, 1775), (1024, 7103)])        # one row short of it
@pytest.mark.parametrize("offset", [3.0, 300.0])
def test_layernorm_forward_of_many_rows(H, rows, offset):
    """Mean and 1/std from parts of a row.  fp32 sums of values near `offset`: off by 2^-22 offset at most per value, hence the mean by
    that, the sum of squares about it by its square; results round to bf16 once (2^-9)."""
    torch.manual_seed(H + rows)
    x = (torch.randn(rows, H, device=DEV) * 2 + offset).bfloat16()
    flat = torch.randn(2 * H + 1, device=DEV)
    for g, b in ((flat[:H], flat[H:2 * H]), (flat[1:H + 1], flat[H + 1:])):      # on and off a 16-byte boundary
        y, mean, rstd = native.ext().layernorm_fwd(x, None, g, b, 1e-5)[:3]
        d = x.double()
        mu = d.mean(-1)
        want = torch.nn.functional.layer_norm(d, (H,), g.double(), b.double(), 1e-5)
        r = 1.0 / torch.sqrt(d.var(-1, unbiased=False) + 1e-5)
        assert float((mean.double() - mu).abs().max()) <= 2.0 ** -20 * offset
        assert float(((rstd.double() - r) / r).abs().max()) <= 2.0 ** -18
        slip = 2.0 ** -20 * offset * r[:, None] * g.double().abs()
        assert float(((y.double() - want).abs() - 2.0 ** -8 * (want.abs() + b.double().abs()) - slip).max()) <= 0


@pytest.mark.parametrize("H,rows", [(8, 7104), (264, 7105), (512, 9001), (520, 4000), (776, 7104), (1000, 7999), (1024, 8000), (1032, 4440),
                                    (1280, 5003), (1288, 2220), (1536, 2370), (1544, 1776), (1800, 2500), (2048, 5003), (3000, 300)])
@pytest.mark.parametrize("with_residual", [False, True])
def test_layernorm_forward_of_a_row_does_not_depend_on_how_many_there_are(H, rows, with_residual):
    """Which kernel takes a call depends on the number of rows; the result of a row does not, in any bit."""
    torch.manual_seed(H)
    x = (torch.randn(rows, H, device=DEV) * 2 + 1).bfloat16()
    res = torch.randn(rows, H, device=DEV).bfloat16() if with_residual else None
    flat = torch.randn(2 * H + 1, device=DEV)
    for g, b in ((flat[:H], flat[H:2 * H]), (flat[1:H + 1], flat[H + 1:])):      # on and off a 16-byte boundary
        call = lambda a, e: native.ext().layernorm_fwd(x[a:e], None if res is None else res[a:e], g, b, 1e-5)[:3]
        whole = call(0, rows)
        for a, e in ((0, 1), (8, 19), (rows // 2, rows // 2 + 700), (0, min(rows, 2400)), (rows - 300, rows)):
            for part, want in zip(call(a, e), whole):
                assert torch.equal(part, want[a:e])
