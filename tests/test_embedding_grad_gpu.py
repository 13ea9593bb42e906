"""The grouped embedding gradient (csrc/embedding_grad.cu) against the sort-based kernel, bit for bit: both sum a row's tokens
in order.  Sizes around the limits of the kernel: one token, a token more than the threads of a cluster, the largest batch; runs
around the length up to which tokens are ranked one by one; ids outside the table."""
import pytest
import torch

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def sorted_grad(keys_t, dst, k0, g, p, seed):
    keys, order = torch.sort(keys_t, stable=True)
    native.ext().embedding_bwd_sorted(keys, order, g, dst, k0, p, seed)
    return dst


@pytest.mark.parametrize("tokens,V,S,H", [(1, 5, 1, 8), (33, 7, 16, 64), (1024, 50, 128, 520), (8193, 51200, 1024, 64),
                                          (16384, 300, 2048, 2048), (65536, 65600, 512, 32)])
@pytest.mark.parametrize("p", [0.0, 0.1])
def test_grouped_embedding_gradient_equals_the_sorted_one(tokens, V, S, H, p):
    torch.manual_seed(tokens + H)
    k0 = 11
    ids = torch.randint(k0 - 5, k0 + V + 5, (tokens,), device=DEV)     # some outside the table
    pos = torch.arange(tokens, device=DEV) % S
    g = torch.randn(tokens, H, device=DEV).bfloat16()
    start_w, start_p = torch.randn(V, H, device=DEV), torch.randn(S, H, device=DEV)
    dW, dP = start_w.clone(), start_p.clone()
    native.ext().embedding_bwd_grouped(ids, pos, g, dW, dP, k0, p, 5)
    assert torch.equal(dW, sorted_grad(ids, start_w.clone(), k0, g, p, 5))
    assert torch.equal(dP, sorted_grad(pos, start_p.clone(), 0, g, p, 5))
    alone = start_w.clone()
    native.ext().embedding_bwd_grouped(ids, None, g, alone, None, k0, p, 5)
    assert torch.equal(alone, dW)


@pytest.mark.parametrize("run", [2, 5, 255, 256, 257, 4000])
def test_runs_of_one_row(run):
    torch.manual_seed(run)
    tokens, V, H = 4000, 900, 136
    ids = torch.randint(0, V, (tokens,), device=DEV)
    ids[ids == 3] = 4
    ids[torch.randperm(tokens, device=DEV)[:run]] = 3
    g = torch.randn(tokens, H, device=DEV).bfloat16()
    dW = torch.zeros(V, H, device=DEV)
    native.ext().embedding_bwd_grouped(ids, None, g, dW, None, 0, 0.0, 0)
    assert torch.equal(dW, sorted_grad(ids, torch.zeros(V, H, device=DEV), 0, g, 0.0, 0))


def test_no_row_of_the_table_occurs():
    ids, g = torch.full((100,), 9, device=DEV), torch.randn(100, 64, device=DEV).bfloat16()
    dW = torch.ones(9, 64, device=DEV)
    native.ext().embedding_bwd_grouped(ids, None, g, dW, None, 0, 0.0, 0)
    assert torch.equal(dW, torch.ones(9, 64, device=DEV))
    with pytest.raises(RuntimeError):
        native.ext().embedding_bwd_grouped(ids[:0], None, g[:0], dW, None, 0, 0.0, 0)


@pytest.mark.parametrize("H", [8, 16, 64, 120, 200, 264, 2040, 2048, 2056, 2560, 4104])   # 1 to 256 threads a token, two, three passes
@pytest.mark.parametrize("tokens", [1, 887, 889, 2500])                         # around a token for every block; further rounds
@pytest.mark.parametrize("places", [False, True])
def test_lookup(H, tokens, places):
    """Ids outside [v0, v1) give no word; a sum of two bf16 values rounds once."""
    torch.manual_seed(H + tokens)
    V, v0 = 300, 50
    W, P = torch.randn(V, H, device=DEV).bfloat16(), torch.randn(77, H, device=DEV).bfloat16()
    ids = torch.randint(0, v0 + V + 40, (tokens,), device=DEV)
    pos = torch.randint(0, 77, (tokens,), device=DEV)
    y = native.ext().embedding_fwd(ids, pos if places else None, W, P if places else None, v0, 0.0, 1)
    here = ((ids >= v0) & (ids < v0 + V))[:, None]
    want = torch.where(here, W[(ids - v0).clamp(0, V - 1)].float(), torch.zeros((), device=DEV))
    if places:
        want = want + P[pos].float()
    assert torch.equal(y, want.bfloat16())


@pytest.mark.parametrize("places", [False, True])
def test_tables_of_no_columns(places):
    """Accepted: no values, no gradients, no division by the length of a row."""
    ids = torch.tensor([[1, 7, 2]], device=DEV)
    W, P = (torch.nn.Parameter(torch.empty(n, 0, device=DEV, dtype=torch.bfloat16)) for n in (5, 3))
    args = (ids, torch.arange(3, device=DEV) if places else None, W, P if places else None, 0, 0.1, 7)
    for call in (F.embedding, F.EmbeddingFn.apply):
        y = call(*args)
        assert y.shape == (3, 0)
        y.backward(torch.empty_like(y))
        assert W.grad.shape == W.shape and (not places or P.grad.shape == P.shape)
    assert native.check_status() == 0


@pytest.mark.parametrize("H", [8, 64, 264, 2048, 2056, 4104])                   # several tokens a block, one pass, two, three
@pytest.mark.parametrize("tokens", [1, 889, 2500])
@pytest.mark.parametrize("p", [0.1, 0.996])
def test_lookup_dropout(H, tokens, p):
    """The mask is the element-wise kernel's for the same seed and flat index; sum and scale are fp32, rounded once; every gradient
    kernel drops what the forward dropped."""
    torch.manual_seed(H + tokens)
    ext = native.ext()
    W, P = torch.randn(3000, H, device=DEV).bfloat16(), torch.randn(77, H, device=DEV).bfloat16()
    ids, pos = torch.randperm(3000, device=DEV)[:tokens], torch.randint(0, 77, (tokens,), device=DEV)
    ones = torch.ones(tokens, H, device=DEV).bfloat16()
    kept = ext.elementwise(F.EW_DROPOUT, ones, None, None, p, 9) != 0
    scale = torch.tensor(256.0 / max(1, int((1 - p) * 256 + 0.5)), device=DEV)
    zero = torch.zeros((), device=DEV)
    y = ext.embedding_fwd(ids, pos, W, P, 0, p, 9)
    assert torch.equal(y, torch.where(kept, (W[ids].float() + P[pos].float()) * scale, zero).bfloat16())
    want = torch.zeros(3000, H, device=DEV)
    want[ids] = torch.where(kept, scale, zero)
    grouped, atomic = torch.zeros_like(want), torch.zeros_like(want)
    ext.embedding_bwd_grouped(ids, None, ones, grouped, None, 0, p, 9)
    ext.embedding_bwd(ids, None, ones, atomic, None, 0, p, 9)
    for dW in (grouped, atomic, sorted_grad(ids, torch.zeros_like(want), 0, ones, p, 9)):
        assert torch.equal(dW, want)
