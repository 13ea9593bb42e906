"""Edges of the streamed support kernels: LayerNorm rows of any length, the one-read cross entropy, the vectorised Adam and
the narrow sort keys of the embedding gradient, each against the same formula in 64 bits."""
import pytest
import torch
import torch.nn.functional as TF

from superscaler_b200.ops import functional as F
from superscaler_b200.ops import native

pytestmark = pytest.mark.gpu


def _rel(a, e):
    return float((a.detach().double() - e).norm() / e.norm().clamp_min(1e-30))


@pytest.mark.parametrize("rows", [1, 7, 301])
@pytest.mark.parametrize("H", [8, 64, 504, 520, 1096, 2048, 2056, 4096, 4104])
@pytest.mark.parametrize("shift", [0, 1])        # 1: gamma / beta start 4 bytes off a 16-byte boundary
def test_layernorm_rows(rows, H, shift):
    g = torch.Generator(device="cuda").manual_seed(H + rows)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, dy, dres = (r(rows, H).bfloat16() for _ in range(3))
    x.requires_grad_(True)
    par = [torch.nn.Parameter((r(H + 4) + 1.0)[shift:shift + H]) for _ in range(2)]
    for p in par:
        p.main_grad = torch.zeros(H, device="cuda")
    y, keep = F.layernorm_keep_input(x, *par, 1e-5)
    torch.autograd.backward([y, keep], [dy, dres])
    t = [v.detach().double().requires_grad_(True) for v in (x, *par)]
    want = TF.layer_norm(t[0], (H,), t[1], t[2], 1e-5)
    dx, dg, db = torch.autograd.grad(want, t, dy.double())
    # one bf16 rounding of y and dx; fp32 sums over the rows
    assert _rel(y, want.detach()) < 2.0 ** -8
    assert _rel(x.grad, dx + dres.double()) < 2.0 ** -8
    assert _rel(par[0].main_grad, dg) < 1e-5 and _rel(par[1].main_grad, db) < 1e-5


@pytest.mark.parametrize("V,ld", [(8, 8), (1000, 1000), (1003, 1008), (51200, 51200), (57344, 57344), (57352, 57352)])
def test_cross_entropy_rows(V, ld):
    rows = 5
    g = torch.Generator(device="cuda").manual_seed(V)
    buf = (torch.randn(rows, ld, generator=g, device="cuda") * 4).bfloat16()
    buf[1, : V // 2] = float("-inf")                      # half a row masked out
    t = torch.randint(V // 2, V, (rows,), generator=g, device="cuda")
    t[2] = V + 3                                          # another rank's target: no entry of this row
    w = torch.rand(rows, generator=g, device="cuda")
    x = buf[:, :V].double()
    work = buf.clone()
    loss = native.ext().ce_loss_grad(work[:, :V], t, w, 0, 0.5)
    lse = torch.logsumexp(x, -1)
    own = t < V
    hit = torch.zeros(rows, dtype=torch.float64, device="cuda")
    hit[own] = x[own, t[own]]
    assert torch.allclose(loss.double(), (lse - hit) * w.double(), rtol=1e-5, atol=1e-5)
    grad = torch.softmax(x, -1)
    grad[own, t[own]] -= 1.0
    grad = grad * w.double()[:, None] * 0.5
    assert _rel(work[:, :V], grad) < 2.0 ** -8
    assert torch.equal(work[:, V:], buf[:, V:])


@pytest.mark.parametrize("n,start", [(1, 0), (5, 0), (4096, 0), (4099, 0), (300001, 0), (4096, 1), (4096, 2)])
def test_adam_vector_and_scalar_parts(n, start):
    g = torch.Generator(device="cuda").manual_seed(n)
    r = lambda: torch.randn(n + 8, generator=g, device="cuda")[start:start + n]
    p, m, grad, v = r(), r(), r(), r().square()
    p16 = torch.zeros(n + 8, dtype=torch.bfloat16, device="cuda")[start:start + n]
    wd_end = max(0, n - 3)                                # the decayed part ends inside a vector
    skipped = torch.zeros(1, dtype=torch.int32, device="cuda")
    ss = grad.square().sum().reshape(1)
    args = [t.double() for t in (p, m, v, grad)]
    native.ext().adam_step(p, m, v, grad, p16, ss, skipped, 1e-2, 0.9, 0.999, 1e-8, 0.1, 7, 1.0, 1.0, wd_end, True)
    pd, md, vd, gd = args
    gd = gd * min(1.0, 1.0 / (float(ss.sqrt()) + 1e-6))
    md, vd = 0.9 * md + 0.1 * gd, 0.999 * vd + 0.001 * gd * gd
    decay = torch.zeros(n, dtype=torch.float64, device="cuda")
    decay[:wd_end] = 0.1
    pd = pd - 1e-2 * ((md / (1 - 0.9 ** 7)) / ((vd / (1 - 0.999 ** 7)).sqrt() + 1e-8) + decay * pd)
    assert _rel(m, md) < 1e-6 and _rel(v, vd) < 1e-6 and _rel(p, pd) < 1e-5
    assert torch.equal(p16, p.bfloat16()) and not grad.any()


@pytest.mark.parametrize("n", [300, 4096])
@pytest.mark.parametrize("V", [3, 32766, 32767, 40000])
def test_embedding_gradient_keys(V, n, H=64):
    """Two sequences of n tokens: grouped by row up to 65536 tokens, sorted beyond."""
    v0 = 5
    g = torch.Generator(device="cuda").manual_seed(V)
    ids = torch.randint(v0, v0 + V, (2, n), generator=g, device="cuda")
    ids[0, :4] = torch.tensor([0, v0 - 1, v0 + V, 2 ** 40], device="cuda")    # outside the table, one past 32 bits
    ids[1, 10:60] = v0 + V - 1                                               # a long run
    W = torch.nn.Parameter(torch.randn(V, H, generator=g, device="cuda").bfloat16())
    W.main_grad = torch.zeros(V, H, device="cuda")
    y = F.embedding(ids, None, W, None, v0)
    dy = torch.randn(2 * n, H, generator=g, device="cuda").bfloat16()
    y.backward(dy)
    want = torch.zeros(V, H, dtype=torch.float64, device="cuda")
    flat = ids.view(-1) - v0
    ok = (flat >= 0) & (flat < V)
    want.index_add_(0, flat[ok], dy.double()[ok])
    assert _rel(W.main_grad, want) < 1e-6


@pytest.mark.parametrize("H", [512, 520, 2048, 4104])
def test_layernorm_refuses_misaligned_rows(H):
    """The kernels move 16 bytes a lane: contiguous matrices that start elsewhere are an error on the host."""
    rows, ext = 9, native.ext()
    even = torch.zeros(rows, H, dtype=torch.bfloat16, device="cuda")
    odd = torch.zeros(rows * H + 8, dtype=torch.bfloat16, device="cuda")[1:rows * H + 1].view(rows, H)
    gamma, stat = torch.ones(H, device="cuda"), torch.ones(rows, device="cuda")
    dg, db = torch.zeros(H, device="cuda"), torch.zeros(H, device="cuda")
    for x, res in ((odd, None), (even, odd)):
        with pytest.raises(RuntimeError, match="layernorm_fwd"):
            ext.layernorm_fwd(x, res, gamma, gamma, 1e-5)
    for dy, x, dres in ((odd, even, None), (even, odd, None), (even, even, odd)):
        with pytest.raises(RuntimeError, match="layernorm_bwd"):
            ext.layernorm_bwd(dy, x, gamma, stat, stat, dres, dg, db, False)


@pytest.mark.parametrize("rows,H", [(16603, 504), (8317, 1000), (4157, 2048), (2083, 4096)])
@pytest.mark.parametrize("residual", [False, True])
def test_layernorm_backward_wraps_its_ring(rows, H, residual):
    """Rows enough for every block (two per SM at most) to reuse each of the three stages of its ring at least once, the last
    chunk ragged: one to eight warps per row."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, dy, dres = (r(rows, H).bfloat16() for _ in range(3))
    gamma, beta = r(H) + 1.0, r(H)
    y, mean, rstd = native.ext().layernorm_fwd(x, None, gamma, beta, 1e-5)
    dg, db = torch.zeros(H, device="cuda"), torch.zeros(H, device="cuda")
    dx = native.ext().layernorm_bwd(dy, x, gamma, mean, rstd, dres if residual else None, dg, db, True)
    t = [v.double().requires_grad_(True) for v in (x, gamma, beta)]
    want = torch.autograd.grad(TF.layer_norm(t[0], (H,), t[1], t[2], 1e-5), t, dy.double())
    assert _rel(dx, want[0] + (dres.double() if residual else 0.0)) < 2.0 ** -8
    assert _rel(dg, want[1]) < 1e-5 and _rel(db, want[2]) < 1e-5
    assert native.check_status() == 0


@pytest.mark.parametrize("two_pass", [False, True])       # the form of one rank alone, the one of a vocabulary over several
def test_cross_entropy_at_the_benchmark_vocabulary(two_pass):
    """4096 rows of 51200 bf16 logits, every entry: fp32 sums of 51200 exponentials, each off by a few units in the last
    place (1e-5 of the loss); the gradient carries one bf16 rounding (2^-9) on top of that, so 2^-8 of each entry."""
    T, V = 4096, 51200
    g = torch.Generator(device="cuda").manual_seed(45)
    logits = (torch.randn(T, V, generator=g, device="cuda") * 2).bfloat16()
    t = torch.randint(0, V, (T,), generator=g, device="cuda")
    work, ext = logits.clone(), native.ext()
    if two_pass:
        loss = ext.ce_finalize(work, t, ext.ce_stats(work, t, 0), None, 0, 0.25, True)
    else:
        loss = ext.ce_loss_grad(work, t, None, 0, 0.25)
    for r in range(0, T, 512):
        x, tt = logits[r:r + 512].double(), t[r:r + 512]
        assert torch.allclose(loss[r:r + 512].double(), TF.cross_entropy(x, tt, reduction="none"), rtol=1e-5, atol=1e-5)
        grad = torch.softmax(x, -1)
        grad[torch.arange(512, device="cuda"), tt] -= 1.0
        off = (work[r:r + 512].double() - 0.25 * grad).abs() - 2.0 ** -8 * 0.25 * grad.abs()
        assert float(off.max()) <= 2.0 ** -126                # below the smallest normal number bf16 may round to zero


@pytest.mark.parametrize("V", [8, 1003, 2048, 14336, 14344, 36864, 36872])     # 128, 256 and 512 threads a row
def test_cross_entropy_of_many_rows(V):
    """More rows than fit on the chip at once, where the width of the row chooses the number of threads."""
    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 5
    g = torch.Generator(device="cuda").manual_seed(V)
    buf = (torch.randn(rows, (V + 7) // 8 * 8, generator=g, device="cuda") * 4).bfloat16()
    t = torch.randint(0, V, (rows,), generator=g, device="cuda")
    x = buf[:, :V].double()
    work = buf.clone()
    loss = native.ext().ce_loss_grad(work[:, :V], t, None, 0, 0.5)
    assert torch.allclose(loss.double(), TF.cross_entropy(x, t, reduction="none"), rtol=1e-5, atol=1e-5)
    grad = torch.softmax(x, -1)
    grad[torch.arange(rows, device="cuda"), t] -= 1.0
    assert _rel(work[:, :V], 0.5 * grad) < 2.0 ** -8
    assert torch.equal(work[:, V:], buf[:, V:])


@pytest.mark.parametrize("per_sm,extra,start", [(1024, 0, 0), (1024, 1, 0), (1024, 7, 1), (8 * 2048, 4099, 0)])
def test_adam_at_the_edges_of_its_forms(per_sm, extra, start):
    """An element a thread up to 1024 elements an SM, then vectors; from 8 x 2048 an SM on every block takes several passes."""
    test_adam_vector_and_scalar_parts(torch.cuda.get_device_properties(0).multi_processor_count * per_sm + extra, start)


@pytest.mark.parametrize("V", [40, 1003, 2048, 40000])
@pytest.mark.parametrize("rows", [9, 900])
def test_cross_entropy_of_rows_that_are_not_finite(V, rows):
    """Rows of -inf alone, with +inf or NaN in a vector or in the ragged end, targets in and outside the row: the one-pass form
    gives what the two-pass form gives, NaN where that gives NaN."""
    g = torch.Generator(device="cuda").manual_seed(V)
    buf = torch.randn(rows, (V + 7) // 8 * 8, generator=g, device="cuda").bfloat16()
    inf, nan = float("inf"), float("nan")
    buf[0], buf[1], buf[2, :V // 2], buf[3, V // 2:] = -inf, -inf, -inf, -inf
    buf[4, 3], buf[5, V - 1], buf[6, 3], buf[7, V - 1] = inf, inf, nan, nan
    buf[8, :8] = nan
    t = torch.randint(0, V, (rows,), generator=g, device="cuda")
    t[1] = t[7] = V + 1                                   # another rank's target
    one, two, ext = buf.clone(), buf.clone(), native.ext()
    a = ext.ce_loss_grad(one[:, :V], t, None, 0, 0.5)
    b = ext.ce_finalize(two[:, :V], t, ext.ce_stats(two[:, :V], t, 0), None, 0, 0.5, True)
    assert torch.allclose(a, b, rtol=1e-5, atol=1e-5, equal_nan=True)
    assert torch.allclose(one.float(), two.float(), rtol=2.0 ** -7, atol=0.0, equal_nan=True)   # one unit of bf16


@pytest.mark.parametrize("V", [3, 32766, 32767, 40000])   # sort keys of 16 bits up to 32766 rows, of 32 beyond
@pytest.mark.parametrize("n", [32768, 32769, 40000])      # two sequences: the last token count that is grouped, then sorted ones
def test_embedding_gradient_of_many_tokens(V, n):
    test_embedding_gradient_keys(V, n, H=8)


@pytest.mark.parametrize("V", [1, 32766, 32767, 40000])
@pytest.mark.parametrize("n", [1, 257, 5000])
def test_sorted_embedding_gradient_with_narrow_keys(V, n):
    """The sorted form itself, with the keys it is given above 65536 tokens: every row summed in token order."""
    H, k0, ext = 24, 7, native.ext()
    g = torch.Generator(device="cuda").manual_seed(V + n)
    ids = torch.randint(k0 - 3, k0 + V + 3, (n,), generator=g, device="cuda")
    ids[0] = 2 ** 40 + k0                                 # one past 32 bits
    if n > 100:
        ids[10:90] = k0 + V - 1                           # a run at the last row
    dy, start = torch.randn(n, H, generator=g, device="cuda").bfloat16(), torch.randn(V, H, generator=g, device="cuda")
    keys = ext.embedding_keys(ids, k0, V)
    assert keys.dtype == (torch.int16 if V <= 32766 else torch.int32)
    inside = (ids >= k0) & (ids < k0 + V)
    assert torch.equal(keys.long(), torch.where(inside, ids - k0, V))
    keys, order = torch.sort(keys, stable=True)
    dst = start.clone()
    ext.embedding_bwd_sorted(keys, order, dy, dst, 0, 0.0, 0)
    want = start.double().index_add_(0, (ids - k0)[inside], dy.double()[inside])
    assert _rel(dst, want) < 1e-6
    again = start.clone()
    ext.embedding_bwd_sorted(keys, order, dy, again, 0, 0.0, 0)
    assert torch.equal(dst, again)


@pytest.mark.parametrize("V", [40, 1003, 40000, 60000])   # the one-pass form at each number of threads, the two-pass form
def test_cross_entropy_keeps_probabilities_below_the_normal_range(V):
    """Probabilities of 1e-39 to 1e-42 times a large gradient scale (a loss scale) are ordinary gradients: exp is good to 2^-16
    there (the exponent is near 140, in fp32), a subnormal of 5e-42 holds eleven bits, and bf16 rounds by 2^-9: below 2^-8."""
    rows, scale = 6, 2.0 ** 100
    buf = torch.zeros(rows, (V + 7) // 8 * 8, device="cuda", dtype=torch.bfloat16)
    for r, low in enumerate((-80.0, -86.0, -88.0, -90.0, -92.0, -95.0)):
        buf[r] = low
    t = torch.tensor([0, 1, V // 2, V - 1, V - 2, 7], device="cuda")
    buf[torch.arange(rows, device="cuda"), t] = 0.0
    work = buf.clone()
    native.ext().ce_loss_grad(work[:, :V], t, None, 0, scale)
    x = buf[:, :V].double()
    grad = torch.softmax(x, -1) * scale
    grad[torch.arange(rows, device="cuda"), t] = 0.0     # p - 1 of the target rounds to nothing
    work[torch.arange(rows, device="cuda"), t] = 0.0
    off = (work[:, :V].double() - grad).abs() - 2.0 ** -8 * grad
    assert float(off.max()) <= 0.0


@pytest.mark.parametrize("rows,H", [(1, 1032), (7, 1536), (1777, 1288), (2500, 1536), (1200, 1544), (2401, 1800)])
@pytest.mark.parametrize("residual", [False, True])
def test_layernorm_backward_with_three_and_four_warps_a_row(rows, H, residual):
    torch.manual_seed(rows + H)
    x, dy = (torch.randn(rows, H, device="cuda") * 2 + 1).bfloat16(), torch.randn(rows, H, device="cuda").bfloat16()
    g, b = torch.randn(H, device="cuda"), torch.randn(H, device="cuda")
    dres = torch.randn(rows, H, device="cuda").bfloat16() if residual else None
    _, mean, rstd = native.ext().layernorm_fwd(x, None, g, b, 1e-5)[:3]
    dg, db = torch.ones(H, device="cuda"), torch.ones(H, device="cuda")
    dx = native.ext().layernorm_bwd(dy, x, g, mean, rstd, dres, dg, db, True)
    t = [v.double().requires_grad_(True) for v in (x, g, b)]
    want = torch.autograd.grad(torch.nn.functional.layer_norm(t[0], (H,), t[1], t[2], 1e-5), t, dy.double())
    assert _rel(dx, want[0] + (dres.double() if residual else 0)) < 2.0 ** -8       # one rounding to bf16
    assert _rel(dg - 1, want[1]) < 1e-5 and _rel(db - 1, want[2]) < 1e-5            # fp32 sums
    assert native.check_status() == 0


@pytest.mark.parametrize("rows,N", [(1, 8), (63, 264), (64, 256), (65, 2048), (129, 520), (1000, 1000), (8192, 72), (8193, 640), (20000, 8192)])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("off", [0, 2])                  # columns in front: rows that do not start on 16 bytes take the two-pass kernel
def test_column_sums(rows, N, accumulate, off):
    """One slice of rows, a few, as many as there may be.  Whole numbers: every sum is exact in fp32, a row lost or added twice shows."""
    torch.manual_seed(rows + N)
    a = torch.randint(-4, 5, (rows, N + 8), device="cuda").bfloat16()[:, off:off + N]
    out = torch.randint(-1000, 1001, (N,), device="cuda").float()
    want = a.double().sum(0) + (out.double() if accumulate else 0)
    for _ in range(2):                                   # the counters are as they were after a call
        got = out.clone()
        native.ext().colsum(a, got, accumulate)
        assert torch.equal(got.double(), want)


@pytest.mark.parametrize("V,rows,fewer", [(14336, 200, 147), (15001, 296, 1), (16392, 296, 148),           # one row an SM, two
                                          (16392, 3080, 3060), (24584, 860, 850), (40000, 530, 520)])       # loads ahead and not
def test_cross_entropy_of_a_row_does_not_depend_on_a_few_more(V, rows, fewer):
    """The same threads add the same values, whether their loads run ahead (from 96 MiB of logits on, from 40 MiB of rows of more than
    24576) or not."""
    torch.manual_seed(V)
    x = torch.randn(rows, (V + 7) // 8 * 8, device="cuda").bfloat16()
    t = torch.randint(0, V, (rows,), device="cuda")
    whole, part = x.clone(), x[:fewer].clone()
    want = native.ext().ce_loss_grad(whole[:, :V], t, None, 0, 0.5)
    loss = native.ext().ce_loss_grad(part[:, :V], t[:fewer], None, 0, 0.5)
    assert torch.equal(loss, want[:fewer]) and torch.equal(part[:, :V], whole[:fewer, :V])
    some = slice(0, rows, 7)
    exact = torch.nn.functional.cross_entropy(x[some, :V].double(), t[some], reduction="none")
    assert torch.allclose(want[some].double(), exact, rtol=1e-5, atol=1e-5)
