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
