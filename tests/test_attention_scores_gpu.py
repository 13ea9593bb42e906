"""Flash attention on scores that are not small and alike."""
import math

import pytest
import torch

from superscaler_b200.ops import functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("HD", [64, 128])
@pytest.mark.parametrize("blocks", [2, 5])
def test_rows_of_one_value_are_exact(HD, blocks):
    """All values of a sequence equal one vector, so every output row is that vector, whatever the scores.  A row has one
    key of score 0 in the first block and one above it by up to 8 (log2) in the last; the other keys lie 40 below and weigh
    less than 2^-30 in all.  Both keys are their block's maximum, so their probabilities are exactly one when they are
    rounded to bf16, and sums and products are fp32: the result is off by less than 2^-18 before it is rounded to bf16, which
    returns the vector itself.  A probability rounded away from one (by up to 2^-9) would show."""
    S, rows = 128 * blocks, 128 * blocks
    g = torch.Generator(device="cuda").manual_seed(HD + blocks)
    q = torch.zeros(rows, HD, device="cuda")
    q[:, 0] = (torch.arange(rows, device="cuda") % 128 + 1) / 16.0        # score of the late key: up to 8
    q[:, 1] = 1.0
    k = torch.zeros(S, HD, device="cuda")
    k[:, 1] = -40.0
    k[17, 1] = 0.0
    k[S - 50] = 0.0
    k[S - 50, 0] = 1.0
    v = torch.randn(HD, generator=g, device="cuda").expand(S, HD)
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16().contiguous()
    o = F.flash_attention(q, k, v, 1, 1, rows, S, HD, scale=math.log(2.0))
    assert torch.equal(o, v[:1].expand(rows, HD))


@pytest.mark.parametrize("SQ,SK,HD,causal", [(64, 128, 64, False), (192, 256, 128, False), (100, 77, 64, False),
                                             (64, 64, 128, True), (321, 321, 64, True)])
def test_samples_keep_their_nans(SQ, SK, HD, causal):
    """Blocks that reach past the end of a sample must not bring in what the next one holds: with NaNs and infinities in the
    second of three samples the results of the others stay what they are with zeros in it."""
    B, NH = 3, 2
    g = torch.Generator(device="cuda").manual_seed(SQ)
    w = NH * HD
    made = [torch.randn(B, n, w, generator=g, device="cuda") for n in (SQ, SK, SK, SQ)]
    out = []
    for bad in (0.0, float("nan"), float("inf")):
        q, k, v, do = (t.clone() for t in made)
        for t in (q, k, v, do):
            t[1] = bad
        q, k, v, do = (t.view(-1, w).bfloat16() for t in (q, k, v, do))
        for t in (q, k, v):
            t.requires_grad_(True)
        y = F.flash_attention(q, k, v, B, NH, SQ, SK, HD, causal=causal)
        y.backward(do)
        out.append([t.detach().view(B, -1, w)[[0, 2]] for t in (y, q.grad, k.grad, v.grad)])
    for other in out[1:]:
        for a, e in zip(other, out[0]):
            assert torch.isfinite(a).all()
            # dq is summed over the key blocks in the order they finish: fp32 sums, then one rounding to bf16
            assert float((a.double() - e.double()).norm()) <= 2.0 ** -9 * float(e.double().norm())
