"""Flash attention on scores that are not small and alike, on samples that must not mix, and on more work items than SMs."""
import math

import pytest
import torch

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native
from test_attention_tiles_gpu import TOL, _oracle

pytestmark = pytest.mark.gpu


def _split(heads, SQ, SK, causal):
    """True where the forward deals the key blocks of a query tile to two slots, False where it works on pairs of tiles."""
    return native.ext().attn_fwd_split(heads, SQ, SK, causal, torch.cuda.get_device_properties(0).multi_processor_count)


@pytest.mark.parametrize("HD", [64, 128])
@pytest.mark.parametrize("blocks", [2, 5])
@pytest.mark.parametrize("NH", [1, 80, 120])             # (which form of the forward each takes: see below)
def test_rows_of_one_value_are_exact(HD, blocks, NH):
    """All values of a sequence equal one vector, so every output row is that vector, whatever the scores.  A row has one
    key of score 0 in the first block and one above it by up to 8 (log2) in the last; the other keys lie 40 below and weigh
    less than 2^-30 in all.  Both keys are their block's maximum, so their probabilities are exactly one when they are
    rounded to bf16, and sums and products are fp32: the result is off by less than 2^-18 before it is rounded to bf16, which
    returns the vector itself.  A probability rounded away from one (by up to 2^-9) would show."""
    S, rows = 128 * blocks, 128 * blocks
    assert _split(NH, rows, S, False) == ((NH, blocks) in {(1, 2), (1, 5), (80, 5)})
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
    q, k, v = (t.bfloat16().repeat(1, NH) for t in (q, k, v))
    o = F.flash_attention(q, k, v, 1, NH, rows, S, HD, scale=math.log(2.0))
    assert torch.equal(o, v[:1].expand(rows, NH * HD))


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


@pytest.mark.parametrize("S,HD,causal,p,bias", [
    (700, 64, True, 0.0, False),
    (700, 128, True, 0.1, False),
    (515, 64, False, 0.1, True),
    (515, 128, False, 0.0, False),
])
@pytest.mark.parametrize("gain", [8.0, 32.0])
@pytest.mark.parametrize("rising", [1, 32])              # rows of every 32 whose maximum rises with the keys
@pytest.mark.parametrize("B,NH", [(2, 2), (8, 4)])       # split keys; split keys if causal, else pairs of tiles
def test_late_maxima(S, HD, causal, p, bias, gain, rising, B, NH):
    """Keys ordered along one direction that some queries follow and the others oppose: their running maximum grows in
    every block, by more than 2^8 in probability.  The forward stays within the tolerance of small scores (fp32 scores of
    some 2^8 are off by 2^-16).  In the backward dS = P (dP - delta) cancels where one key takes the whole row, and what
    remains is the rounding of O in delta: e_r = 2^-9 |dO_r O_r| for row r, which enters dq_r with a weighted mean of keys
    and dk with q_r."""
    assert _split(B * NH, S, S, causal) == (B * NH == 4 or (B * NH == 32 and causal))
    seed = 5
    g = torch.Generator(device="cuda").manual_seed(S + HD)
    w, n = NH * HD, B * S
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    u = torch.nn.functional.normalize(r(HD), dim=0).repeat(NH)
    ramp = torch.linspace(-1.0, 1.0, S, device="cuda").repeat(B)[:, None]
    sign = torch.where(torch.arange(n, device="cuda") % 32 < rising, 1.0, -1.0)[:, None]
    q = (0.1 * gain * r(n, w) + gain * sign * u).bfloat16()
    k = (0.1 * r(n, w) + math.sqrt(HD) * ramp * u).bfloat16()
    v, do = r(n, w).bfloat16(), r(n, w).bfloat16()
    for t in (q, k, v):
        t.requires_grad_(True)
    bt = r(NH, 2 * S - 1).requires_grad_(True) if bias else None
    y = F.flash_attention(q, k, v, B, NH, S, S, HD, causal=causal, dropout_p=p, seed=seed, bias_table=bt)
    y.backward(do)
    o, dq, dk, dv, db = _oracle(q.detach(), k.detach(), v.detach(), do, B, NH, S, S, HD, causal, None, p, seed,
                                bt.detach() if bias else None)
    heads = lambda t: t.double().view(n, NH, HD)
    e = 2.0 ** -9 * (heads(do) * heads(o)).norm(dim=-1)                       # [tokens, heads]
    scale = HD ** -0.5
    slack = {"dq": scale * float(e.norm() * heads(k.detach()).norm(dim=-1).max()),
             "dk": scale * float((e * heads(q.detach()).norm(dim=-1)).norm())}
    err = lambda a, b: float((a.double() - b).norm())
    assert err(y.detach(), o) <= TOL * float(o.norm())
    assert err(v.grad, dv) <= TOL * float(dv.norm())
    assert err(q.grad, dq) <= TOL * float(dq.norm()) + 2 * slack["dq"]
    assert err(k.grad, dk) <= TOL * float(dk.norm()) + 2 * slack["dk"]
    if bias:
        assert err(bt.grad, db) <= TOL * float(db.norm()) + 2 * float(e.norm())


@pytest.mark.parametrize("HD,p", [(64, 0.0), (128, 0.1)])
@pytest.mark.parametrize("gain,rising", [(8.0, 1), (32.0, 1), (32.0, 32)])
def test_late_maxima_in_causal_pairs(HD, p, gain, rising):
    """Pairs of query tiles of unequal length under the mask: more heads than those above."""
    test_late_maxima(700, HD, True, p, False, gain, rising, 8, 12)


@pytest.mark.parametrize("NH", [2, 120])                 # split keys; pairs of tiles
@pytest.mark.parametrize("HD", [64, 128])
@pytest.mark.parametrize("first", [0, 1])                # the even or the odd key blocks: one slot or the other
@pytest.mark.parametrize("bad", [-math.inf, math.inf, math.nan])
def test_scores_that_are_not_finite_in_one_slot(NH, HD, first, bad):
    """Whole key blocks of scores -inf (rows with a first component of one) or +inf (minus one), a single NaN key: rows come out
    as softmax gives them, NaN where that is NaN, and the others stay what they are."""
    S = 640
    assert _split(NH, S, S, False) == (NH == 2)
    g = torch.Generator(device="cuda").manual_seed(HD)
    q, k, v = (torch.randn(S, HD, generator=g, device="cuda").bfloat16() for _ in range(3))
    q[:, 0] = 1.0
    if bad == math.inf:
        q[::3, 0] = -1.0                                 # their scores of those keys are -inf: no weight
    k[:, 0] = 0.0
    if math.isnan(bad):
        k[128 * first + 5, 0] = bad
    else:
        for b in range(first, 5, 2):
            k[128 * b:128 * (b + 1), 0] = bad
    s = (q.double() @ k.double().t()) / math.sqrt(HD)
    want = torch.softmax(s, -1) @ v.double()
    o = F.flash_attention(*(t.repeat(1, NH) for t in (q, k, v)), 1, NH, S, S, HD).double().view(S, NH, HD)
    ok = torch.isfinite(want).all(-1)
    assert bool(ok.any()) == (not math.isnan(bad)) and bool(torch.isnan(o[~ok]).all())
    err = (o[ok] - want[ok][:, None]).norm()
    assert float(err) <= TOL * float(want[ok].norm()) * math.sqrt(NH)


@pytest.mark.parametrize("SQ,SK,HD,causal,lens,p,bias", [
    (130, 130, 64, True, False, 0.1, False),
    (300, 300, 128, True, False, 0.1, False),
    (300, 300, 64, False, True, 0.1, True),
    (130, 300, 128, False, True, 0.0, False),
    (300, 130, 64, False, True, 0.0, False),
    (127, 127, 64, True, False, 0.1, False),
    (257, 257, 128, True, False, 0.0, False),
    (255, 130, 64, False, True, 0.1, False),
    (384, 96, 128, False, False, 0.5, False),
    (256, 256, 64, False, True, 0.1, True),
])
def test_more_items_than_sms(SQ, SK, HD, causal, lens, p, bias):
    """320 heads: every CTA of the persistent forward takes several items, some of them empty (a sample without keys)."""
    B, NH, seed = 20, 16, 31
    g = torch.Generator(device="cuda").manual_seed(SQ + SK + HD)
    w = NH * HD
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    q, k, v, do = (r(B * n, w).bfloat16() for n in (SQ, SK, SK, SQ))
    for t in (q, k, v):
        t.requires_grad_(True)
    bt = r(NH, SQ + SK - 1).requires_grad_(True) if bias else None
    ln = None
    if lens:
        ln = torch.randint(1, SK + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
        ln[3] = ln[10] = 0
        ln[11] = SK
    y = F.flash_attention(q, k, v, B, NH, SQ, SK, HD, causal=causal, kv_lens=ln, dropout_p=p, seed=seed, bias_table=bt)
    y.backward(do)
    want = _oracle(q.detach(), k.detach(), v.detach(), do, B, NH, SQ, SK, HD, causal, ln, p, seed,
                   bt.detach() if bias else None)
    got = [y.detach(), q.grad, k.grad, v.grad] + ([bt.grad] if bias else [])
    for a, e in zip(got, want):
        e = e.double()
        assert torch.isfinite(a).all()
        assert float((a.double() - e).norm()) <= TOL * float(e.norm()) + HD * 2.0 ** -24 * float(do.double().norm())
    assert native.check_status() == 0


@pytest.mark.parametrize("S", [31, 32, 33, 64, 65, 96, 97, 160, 225])
@pytest.mark.parametrize("HD,causal,lens", [(64, True, False), (128, True, False), (64, False, True), (128, False, True)])
def test_warps_without_queries_or_keys(S, HD, causal, lens):
    """Lengths around the 32 queries and 32 keys of a backward warp, which passes over what it does not see."""
    B, NH, seed, p = 2, 2, 9, 0.1
    g = torch.Generator(device="cuda").manual_seed(S)
    w = NH * HD
    q, k, v, do = (torch.randn(B * S, w, generator=g, device="cuda").bfloat16() for _ in range(4))
    for t in (q, k, v):
        t.requires_grad_(True)
    ln = torch.tensor([S, max(1, S - 40)], dtype=torch.int32, device="cuda") if lens else None
    y = F.flash_attention(q, k, v, B, NH, S, S, HD, causal=causal, kv_lens=ln, dropout_p=p, seed=seed)
    y.backward(do)
    want = _oracle(q.detach(), k.detach(), v.detach(), do, B, NH, S, S, HD, causal, ln, p, seed, None)
    for a, e in zip([y.detach(), q.grad, k.grad, v.grad], want):
        e = e.double()
        assert float((a.double() - e).norm()) <= TOL * float(e.norm()) + HD * 2.0 ** -24 * float(do.double().norm())
    assert native.check_status() == 0
