"""Flash attention at the edges of its tiles (128 queries / keys, 256-query work items) against 64-bit attention with
the same counter-based dropout mask.

Tolerance: the probabilities enter P.V, and dS the gradient products, as bf16 (relative error 2^-9 each), and the results
are rounded to bf16 once more, so the 2-norm of the error stays below three such roundings of the result's 2-norm; 2^-6 leaves room for
the cancellation in dS = P (dP - delta).  Where that difference vanishes (a single visible key) the fp32 rounding of its
two sums over the head remains: HD 2^-24 of the incoming gradient.
"""
import math

import pytest
import torch

from superscaler_b200.ops import functional as F

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -6


def _fmix32(x):
    x = x ^ (x >> 16)
    x = (x * 0x85EBCA6B) & 0xFFFFFFFF
    x = x ^ (x >> 13)
    x = (x * 0xC2B2AE35) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _hash64(seed, ctr):
    m = (1 << 64) - 1
    z = (seed + ctr * 0x9E3779B97F4A7C15) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return z ^ (z >> 31)


def _keep_mask(seed, bh, sq, sk, p):
    """Kept entries [sq, sk] and the scale of the kept values: byte q % 4 of the hash of (key, query quad) below keep8."""
    keep8 = max(1, min(256, int((1.0 - p) * 256.0 + 0.5)))
    q, k = torch.arange(sq)[:, None], torch.arange(sk)[None, :]
    h = _fmix32((((k * ((sq + 3) // 4) + q // 4) * 0x9E3779B1) + (_hash64(seed, bh) & 0xFFFFFFFF)) & 0xFFFFFFFF)
    return (((h >> (8 * (q % 4))) & 0xFF) < keep8), 256.0 / keep8


def _oracle(q, k, v, do, B, NH, SQ, SK, HD, causal, lens, p, seed, bias):
    out = [torch.zeros(t.shape, dtype=torch.float64, device=t.device) for t in (q, q, k, v)]
    o, dq, dk, dv = out
    dbias = torch.zeros_like(bias) if bias is not None else None
    i, j = torch.arange(SQ, device=q.device)[:, None], torch.arange(SK, device=q.device)[None, :]
    for b in range(B):
        rq, rk = slice(b * SQ, (b + 1) * SQ), slice(b * SK, (b + 1) * SK)
        n = SK if lens is None else int(lens[b])
        for h in range(NH):
            c = slice(h * HD, (h + 1) * HD)
            t = [x.double().requires_grad_(True) for x in (q[rq, c], k[rk, c], v[rk, c])]
            s = t[0] @ t[1].t() / math.sqrt(HD)
            leaves = list(t)
            if bias is not None:
                bt = bias[h].double().requires_grad_(True)
                s = s + bt[j - i + SQ - 1]
                leaves.append(bt)
            hidden = j >= n
            if causal:
                hidden = hidden | (j > i)
            if n > 0:
                pr = torch.softmax(s.masked_fill(hidden, -math.inf), -1)
            else:
                pr = s * 0.0
            if p > 0:
                m, sc = _keep_mask(seed, b * NH + h, SQ, SK, p)
                pr = pr * m.to(q.device) * sc
            y = pr @ t[2]
            o[rq, c] = y.detach()
            g = torch.autograd.grad(y, leaves, do[rq, c].double())
            dq[rq, c], dk[rk, c], dv[rk, c] = g[:3]
            if bias is not None:
                dbias[h] += g[3].float()
    return o, dq, dk, dv, dbias


@pytest.mark.parametrize("SQ,SK,HD,causal,lens,p,bias", [
    (1, 1, 128, True, None, 0.0, False),
    (127, 127, 64, True, None, 0.1, False),
    (129, 129, 128, True, None, 0.1, False),
    (257, 257, 128, True, None, 0.0, False),
    (513, 513, 64, True, None, 0.3, False),
    (1000, 1000, 128, True, None, 0.1, False),
    (64, 384, 128, False, (384, 0, 257), 0.0, False),     # one sample without any visible key
    (255, 130, 64, False, (1, 128, 130), 0.1, False),
    (384, 96, 128, False, None, 0.5, False),
    (256, 256, 64, False, (256, 129, 100), 0.1, True),
    (200, 200, 128, True, None, 0.0, True),
    (131, 131, 64, False, None, 0.1, True),
])
def test_attention_tile_edges(SQ, SK, HD, causal, lens, p, bias):
    _check(3, 2, SQ, SK, HD, causal, lens, p, bias)


@pytest.mark.parametrize("B,NH,S,HD,causal,lens,p,bias", [
    (5, 60, 300, 128, True, None, 0.1, False),            # 900 key blocks and 600 query pairs of unequal length
    (4, 50, 260, 64, False, (260, 0, 129, 1), 0.0, False),  # blocks and samples without a visible key in between
    (4, 40, 250, 64, False, (250, 128, 129, 3), 0.1, True),
    (3, 50, 129, 128, False, None, 0.0, False),
])
def test_attention_with_more_work_items_than_sms(B, NH, S, HD, causal, lens, p, bias):
    """CTAs that go on with further work items: backward key blocks, forward pairs of query tiles."""
    _check(B, NH, S, S, HD, causal, lens, p, bias)


@pytest.mark.parametrize("SQ,SK,HD,causal,lens,p,bias", [
    (128, 128, 128, False, None, 0.0, False),             # one key block: the second slot stays empty
    (100, 1000, 64, False, (129, 1000, 0), 0.1, False),   # the second slot empty for one sample, both for another
    (70, 640, 128, False, (640, 300, 257), 0.1, False),
    (2048, 2048, 128, True, None, 0.1, False),
    (96, 385, 64, False, (385, 128, 256), 0.0, True),
])
def test_attention_with_few_query_tiles(SQ, SK, HD, causal, lens, p, bias):
    """Forward with the key blocks of a tile dealt to two slots whose sums and accumulators are brought together."""
    _check(3, 2, SQ, SK, HD, causal, lens, p, bias)


@pytest.mark.parametrize("HD", [64, 128])
@pytest.mark.parametrize("S,lens,p,bias", [(100, True, 0.1, False), (128, False, 0.0, True), (33, True, 0.0, False)])
@pytest.mark.parametrize("extra", [0, 1])
def test_attention_backward_with_a_key_block_per_sm(HD, S, lens, p, bias, extra):
    """As many key blocks as SMs: every CTA has one and its math warps write dV and dK; with one more, CTAs go on and the drain
    warps write them."""
    heads = torch.cuda.get_device_properties(0).multi_processor_count + extra
    B = next(b for b in (4, 3, 2, 1) if heads % b == 0)
    _check(B, heads // B, S, S, HD, False, ((S, 0, S - 32, 1)[:B] if lens else None), p, bias)


def _check(B, NH, SQ, SK, HD, causal, lens, p, bias):
    seed = 77
    g = torch.Generator(device="cuda").manual_seed(SQ * 1000 + SK)
    w = NH * HD
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    q, k, v, do = (r(B * n, w).bfloat16() for n in (SQ, SK, SK, SQ))
    for t in (q, k, v):
        t.requires_grad_(True)
    bt = r(NH, SQ + SK - 1).requires_grad_(True) if bias else None
    ln = torch.tensor(lens, dtype=torch.int32, device="cuda") if lens else None
    y = F.flash_attention(q, k, v, B, NH, SQ, SK, HD, causal=causal, kv_lens=ln, dropout_p=p, seed=seed, bias_table=bt)
    y.backward(do)
    want = _oracle(q.detach(), k.detach(), v.detach(), do, B, NH, SQ, SK, HD, causal, lens, p, seed,
                   bt.detach() if bias else None)
    got = [y.detach(), q.grad, k.grad, v.grad] + ([bt.grad] if bias else [])
    for a, e in zip(got, want):
        e = e.double()
        assert torch.isfinite(a).all()
        assert float((a.double() - e).norm()) <= TOL * float(e.norm()) + HD * 2.0 ** -24 * float(do.double().norm())
