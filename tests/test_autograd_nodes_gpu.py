"""The native autograd nodes of linear, MLP, LayerNorm and attention (csrc/autograd_nodes.h)."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch

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
