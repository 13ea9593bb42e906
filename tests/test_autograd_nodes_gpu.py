"""The native autograd nodes of linear, MLP, LayerNorm, attention, embedding and the head with its loss (csrc/autograd_nodes.h)."""
import subprocess
import sys
import warnings
from pathlib import Path

import pytest
import torch
import torch.utils.checkpoint

from superscaler_b200.ops import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def _parameters(op):
    """{name: parameter} and the call of an op with two or more parameters, on inputs that are always the same."""
    torch.manual_seed(11)
    bf = lambda *s: torch.randn(*s, device=DEV).bfloat16()
    x = bf(192, 256).requires_grad_(True)
    if op == "linear":
        p = {"w": bf(128, 256) * 0.05, "b": bf(128)}
        call = lambda: F.linear(x, p["w"], p["b"], act=F.ACT_GELU)
    elif op == "mlp":
        p = {"w1": bf(512, 256) * 0.05, "b1": bf(512), "w2": bf(256, 512) * 0.05, "b2": bf(256)}
        call = lambda: F.mlp(x, p["w1"], p["b1"], p["w2"], p["b2"])
    else:
        p = {"g": torch.randn(256, device=DEV), "b": torch.randn(256, device=DEV)}
        if op == "layernorm":
            call = lambda: F.layernorm(x, p["g"], p["b"])
        else:
            call = lambda: sum(F.layernorm_keep_input(x, p["g"], p["b"]))
    for k in p:
        p[k] = torch.nn.Parameter(p[k])
    return p, call


@pytest.mark.parametrize("op", ["linear", "mlp", "layernorm", "layernorm_keep_input"])
@pytest.mark.parametrize("change", ["attach", "replace", "remove"])
def test_the_gradient_buffer_is_the_one_of_the_backward(op, change):
    """`main_grad` is looked up when the backward runs: one that comes, changes or goes after the forward counts."""
    params, call = _parameters(op)
    call().float().square().mean().backward()
    want = {k: p.grad.clone() for k, p in params.items()}
    for p in params.values():
        p.grad = None
        if change != "attach":
            p.main_grad = torch.zeros(p.shape, device=DEV)
    first = {k: getattr(p, "main_grad", None) for k, p in params.items()}
    y = call()
    for p in params.values():
        p.main_grad = None if change == "remove" else torch.zeros(p.shape, device=DEV)
    y.float().square().mean().backward()
    for k, p in params.items():
        if change != "attach":
            assert not first[k].any()
        if change == "remove":
            assert torch.equal(p.grad, want[k])
        else:
            # the same sums, rounded to the parameter's type (bf16: 2^-9) in `want` only
            assert p.grad is None and rel(p.main_grad, want[k]) < 2.0 ** -8


def test_first_use_of_the_device_values_in_a_backward():
    """The status word is made by whichever thread comes first: here Python threads and the backward's, each on a stream of its
    own, in a fresh process.  (Products only: column sums share their ticket counters between the streams of a device.)"""
    code = """
import threading, torch
from superscaler_b200.ops import functional as F, native
x = torch.randn(256, 512, device="cuda").bfloat16().requires_grad_(True)
w = torch.nn.Parameter(torch.randn(256, 512, device="cuda").bfloat16() * 0.05)
torch.cuda.synchronize()
out = {}
def work(i):
    with torch.cuda.stream(torch.cuda.Stream()):
        g = torch.autograd.grad(F.linear(x, w, act=F.ACT_GELU).float().sum(), [x, w])
        torch.cuda.current_stream().synchronize()
        out[i] = g
threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
[t.start() for t in threads]
[t.join() for t in threads]
assert len(out) == 4 and all(torch.equal(a, e) for o in out.values() for a, e in zip(o, out[0]))
assert native.check_status() == 0
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=Path(__file__).parent.parent)


# ---------------------------------- the nodes against the Python functions of the same ops ----------------------------------
# Same kernels in the same order: results are compared bit for bit.
def _bf(*s, scale=1.0):
    return (torch.randn(*s, device=DEV) * scale).bfloat16()


def _linear(act, bias, residual, p):
    t = {"x": _bf(136, 192), "w": _bf(264, 192, scale=0.1)}
    if bias:
        t["b"] = _bf(264)
    if residual:
        t["r"] = _bf(136, 264)
    args = lambda t: (t["x"], t["w"], t.get("b"), t.get("r"), act, p, 7)
    return t, ("w", "b"), lambda t: F.linear(*args(t)), lambda t: F.LinearFn.apply(*args(t))


def _mlp(act, bias, residual, p):
    t = {"x": _bf(136, 192), "w1": _bf(264, 192, scale=0.1), "w2": _bf(192, 264, scale=0.1)}
    if bias:
        t["b1"], t["b2"] = _bf(264), _bf(192)
    if residual:
        t["r"] = _bf(136, 192)
    args = lambda t: (t["x"], t["w1"], t.get("b1"), t["w2"], t.get("b2"), t.get("r"), act, p, 7)
    return t, ("w1", "b1", "w2", "b2"), lambda t: F.mlp(*args(t)), lambda t: F.MLPFn.apply(*args(t))


def _layernorm(keep):
    t = {"x": _bf(136, 264), "g": torch.randn(264, device=DEV), "b": torch.randn(264, device=DEV)}
    node = F.layernorm_keep_input if keep else F.layernorm
    return t, ("g", "b"), lambda t: node(t["x"], t["g"], t["b"]), lambda t: F.LayerNormFn.apply(t["x"], t["g"], t["b"], 1e-5, keep)


def _attention(form, causal, lens, p, table):
    """One block of keys: dQ has one contribution, so it does not depend on an order of arrival."""
    B, NH, HD, S = 3, 2, 64, 120
    w = NH * HD
    if form == "qkv":
        t = {"q": _bf(B * S, 3 * w)}
        operands = lambda t: (t["q"], t["q"], t["q"])
        cols = (0, w, 2 * w)
    elif form == "kv":
        t = {"q": _bf(B * S, w), "k": _bf(B * S, 2 * w + 8)}        # (a carrier wider than its heads)
        operands = lambda t: (t["q"], t["k"], t["k"])
        cols = (0, 0, w)
    else:
        t = {"q": _bf(B * S, w), "k": _bf(B * S, w), "v": _bf(B * S, w)}
        operands = lambda t: (t["q"], t["k"], t["v"])
        cols = (0, 0, 0)
    if table:
        t["table"] = torch.randn(NH, 2 * S - 1, device=DEV)
    kv_lens = torch.tensor([S, 0, 77], dtype=torch.int32, device=DEV) if lens else None
    tail = lambda t: (B, NH, S, S, HD, cols, HD ** -0.5, causal, kv_lens, p, 7, t.get("table"))
    return t, (), lambda t: F.flash_attention(*operands(t), *tail(t)), lambda t: F.FlashAttnFn.apply(*operands(t), *tail(t))


def _embedding(places, v0, p):
    ids = torch.randint(v0 - 4, v0 + 54, (5, 24), device=DEV)           # some outside the table
    pos = torch.arange(24, device=DEV).repeat(5)
    t = {"W": _bf(50, 264)}
    if places:
        t["P"] = _bf(24, 264)
    args = lambda t: (ids, pos if places else None, t["W"], t.get("P"), v0, p, 7)
    return t, ("W", "P"), lambda t: F.embedding(*args(t)), lambda t: F.EmbeddingFn.apply(*args(t))


def _head(mask, v0):
    t = {"x": _bf(136, 192), "W": _bf(264, 192, scale=0.1)}
    targets = torch.randint(v0, v0 + 264, (8, 17), device=DEV)
    weights = torch.rand(136, device=DEV) if mask else None
    args = lambda t: (t["x"], t["W"], targets, weights, v0, 1.0 / 136, None)
    return t, ("W",), lambda t: F.lm_head_cross_entropy(*args(t)), lambda t: F.LMHeadCrossEntropyFn.apply(*args(t))


CASES = {
    "embedding": (_embedding, False, 11, 0.0),
    "embedding_places_dropout": (_embedding, True, 0, 0.1),
    "head_loss": (_head, False, 0),
    "head_loss_mask": (_head, True, 5),
    "linear": (_linear, F.ACT_NONE, True, True, 0.0),
    "linear_gelu_dropout": (_linear, F.ACT_GELU, True, True, 0.1),
    "linear_relu": (_linear, F.ACT_RELU, True, False, 0.0),
    "linear_no_bias": (_linear, F.ACT_NONE, False, False, 0.1),
    "mlp": (_mlp, F.ACT_GELU, True, True, 0.1),
    "mlp_relu_no_bias": (_mlp, F.ACT_RELU, False, False, 0.0),
    "layernorm": (_layernorm, False),
    "layernorm_keep_input": (_layernorm, True),
    "attention_qkv": (_attention, "qkv", True, False, 0.1, False),
    "attention_kv": (_attention, "kv", False, True, 0.0, False),
    "attention_table": (_attention, "separate", False, True, 0.1, True),
}


def _outcome(tensors, params, call, frozen=(), buffers=(), used=None, backwards=1):
    """Outputs, gradients and buffers of a call on fresh copies of the tensors; `used`: the outputs that reach the loss."""
    t = {k: (torch.nn.Parameter(v.clone()) if k in params else v.clone()).requires_grad_(k not in frozen) for k, v in tensors.items()}
    for k in buffers:
        if k in t:
            t[k].main_grad = torch.full(t[k].shape, 0.5, device=DEV)
    y = call(t)
    outs = y if isinstance(y, tuple) else (y,)
    got = {f"out{i}": o.detach().clone() for i, o in enumerate(outs)}
    loss = sum((o.float() * (1 + i + torch.arange(o.numel(), device=DEV).view(o.shape) % 5)).mean()
               for i, o in enumerate(outs) if used is None or i in used)
    if loss.requires_grad:
        for i in range(backwards):
            loss.backward(retain_graph=i + 1 < backwards)
    for k, v in t.items():
        got[k] = v.grad
        got[k + ".main_grad"] = getattr(v, "main_grad", None)
    return got


def _same(a, b):
    assert a.keys() == b.keys()
    for k in a:
        assert (a[k] is None) == (b[k] is None), k
        if a[k] is None:
            continue
        if k == "table":     # atomic additions: an order of fp32 sums
            assert torch.allclose(a[k], b[k], rtol=1e-4, atol=1e-5 * float(b[k].abs().max())), k
        else:
            assert torch.equal(a[k], b[k]), k


@pytest.mark.parametrize("name", CASES)
def test_node_equals_the_function(name):
    torch.manual_seed(5)
    make, *how = CASES[name]
    tensors, params, node, function = make(*how)
    names = list(tensors)
    runs = [{}, dict(backwards=2), dict(buffers=params), dict(buffers=params, backwards=2), dict(frozen=names)]
    runs += [dict(buffers=(k,)) for k in params]
    runs += [dict(frozen=(k,)) for k in names] + [dict(frozen=tuple(n for n in names if n != k)) for k in names]
    runs += [dict(frozen=(k,), buffers=params) for k in names]
    if name == "layernorm_keep_input":
        runs += [dict(used=(0,)), dict(used=(1,)), dict(used=(0,), buffers=params), dict(used=(1,), buffers=params)]
    for run in runs:
        _same(_outcome(tensors, params, node, **run), _outcome(tensors, params, function, **run))
    with torch.no_grad():
        _same(_outcome(tensors, params, node), _outcome(tensors, params, function))


@pytest.mark.parametrize("name", CASES)
def test_node_under_hooks_and_recompute(name):
    """Saved tensors that come back as others (moved to the host and back, recomputed); the buffer is still the parameter's."""
    torch.manual_seed(6)
    make, *how = CASES[name]
    tensors, params, node, _ = make(*how)
    plain = {b: _outcome(tensors, params, node, buffers=b) for b in ((), params)}

    def offloaded(t):
        with torch.autograd.graph.save_on_cpu():
            return node(t)

    def recomputed(t):
        return torch.utils.checkpoint.checkpoint(node, t, use_reentrant=False)

    for call in (offloaded, recomputed):
        for b in ((), params):
            _same(_outcome(tensors, params, call, buffers=b), plain[b])


@pytest.mark.parametrize("name", ["linear_gelu_dropout", "mlp", "layernorm", "attention_qkv"])
def test_backward_of_a_freed_graph_is_refused(name):
    torch.manual_seed(7)
    make, *how = CASES[name]
    tensors, _, node, function = make(*how)
    for call in (node, function):
        y = call({k: v.clone().requires_grad_(True) for k, v in tensors.items()}).float().sum()
        y.backward()
        with pytest.raises(RuntimeError, match="second time"):
            y.backward()


@pytest.mark.parametrize("name", CASES)
def test_transformed_calls_get_the_answer_of_the_function(name):
    """Compiled calls run; forward-mode differentiation and functorch transforms are refused as an autograd function without
    support for them is."""
    torch.manual_seed(8)
    make, *how = CASES[name]
    tensors, params, node, function = make(*how)
    first = next(iter(tensors))

    def dual(call):
        with torch.autograd.forward_ad.dual_level():
            call({**tensors, first: torch.autograd.forward_ad.make_dual(tensors[first], torch.ones_like(tensors[first]))})

    def transformed(call):
        total = lambda y: sum(o.float().sum() for o in y) if isinstance(y, tuple) else y.float().sum()
        torch.func.grad(lambda x: total(call({**tensors, first: x})))(tensors[first])

    for use in (dual, transformed):
        refused = []
        for call in (node, function):
            with pytest.raises(RuntimeError) as e:
                use(call)
            refused.append(e.type)
        assert refused[0] is refused[1]


@pytest.mark.parametrize("name", ["linear_gelu_dropout", "mlp", "layernorm_keep_input", "attention_qkv"])
def test_compiled_calls(name):
    torch.manual_seed(9)
    make, *how = CASES[name]
    tensors, params, node, _ = make(*how)
    torch._dynamo.reset()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")                  # the graph breaks at the kernels' bindings
        compiled = _outcome(tensors, params, torch.compile(node, backend="eager"), buffers=params)
    _same(compiled, _outcome(tensors, params, node, buffers=params))


@pytest.mark.parametrize("in_order,tokens", [(True, 70000), (False, 120)])      # sorted above 65536 tokens; float atomics
def test_embedding_node_takes_the_other_gradient_kernels(in_order, tokens):
    torch.manual_seed(3)
    ids, pos = torch.randint(0, 300, (tokens,), device=DEV), torch.arange(tokens, device=DEV) % 64
    g = torch.randn(tokens, 64, device=DEV).bfloat16()
    grads = []
    for call in (F.embedding, F.EmbeddingFn.apply):
        W, P = (torch.nn.Parameter(torch.zeros(n, 64, device=DEV).bfloat16()) for n in (300, 64))
        P.main_grad = torch.ones(64, 64, device=DEV)
        y = call(ids, pos, W, P, 0, 0.0, 0)
        F.set_deterministic_embedding_grad(in_order)                            # what counts is the switch at the backward
        try:
            y.backward(g)
        finally:
            F.set_deterministic_embedding_grad(True)
        assert P.grad is None
        grads.append((W.grad, P.main_grad))
    for a, b in zip(*grads):
        if in_order:
            assert torch.equal(a, b)
        else:
            assert rel(a, b) < 2.0 ** -8
