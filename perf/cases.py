"""Performance cases: the pieces of work a training or scoring program has this framework do, each through the public
entry point such a program calls (`ops.functional`, `ops.conv`, `StageOptimizer`, `Trainer`).

A case is a dict of plain values.  `prepare` makes what the program holds before the call (activations, parameters with
their fp32 `main_grad`, a trainer), `run` is one pass and returns its outputs whole, `exact` restates the same pass in
64-bit torch, `work` counts the bytes and operations the pass cannot do without.  Sizes are those of the model tables
(GPT-3 1.3B, T5 770M, BERT, Wide-ResNet 1B) and of the tests; `draw` spreads over the ranges between them.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as TF

from superscaler_b200.ops import conv as C
from superscaler_b200.ops import functional as F

_SEED = 0x5EED


def listed():
    return [
        # self-attention of a GPT-3 1.3B layer in training: the plan's micro-batch of 16, dropout 0.1
        dict(name="gpt_attention_train", kind="attention", B=16, NH=16, SQ=2048, SK=2048, HD=128, causal=True,
             cross=False, lens=False, bias=False, dropout=0.1, train=True),
        # the same layer scoring one prompt (text generation re-runs the causal forward over its window)
        dict(name="gpt_attention_prefill", kind="attention", B=1, NH=16, SQ=2048, SK=2048, HD=128, causal=True,
             cross=False, lens=False, bias=False, dropout=0.0, train=False),
        # encoder self-attention of T5 770M: relative-position bias, padded batch
        dict(name="t5_attention_train", kind="attention", B=32, NH=16, SQ=512, SK=512, HD=64, causal=False,
             cross=False, lens=True, bias=True, dropout=0.1, train=True),
        # decoder-to-encoder attention with ragged lengths on both sides
        dict(name="cross_attention_ragged_train", kind="attention", B=8, NH=16, SQ=123, SK=477, HD=64, causal=False,
             cross=True, lens=True, bias=False, dropout=0.0, train=True),
        # feed-forward block of a GPT-3 1.3B layer, four sequences
        dict(name="gpt_mlp_train", kind="mlp", rows=8192, H=2048, F=8192, dropout=0.1),
        # LayerNorm in front of a sub-layer, with the residual branch, the plan's micro-batch
        dict(name="layernorm_train", kind="layernorm", rows=32768, H=2048),
        # word + position embedding of eight sequences
        dict(name="embedding_train", kind="embedding", B=8, S=2048, V=51200, H=2048, dropout=0.1),
        # tied language-model head and its loss, two sequences
        dict(name="lm_head_loss_train", kind="head", rows=4096, V=51200, H=2048),
        # 3 x 3 convolution + BatchNorm + ReLU of Wide-ResNet 1B's second group
        dict(name="resnet_conv_train", kind="conv", N=16, HW=28, C=640, K=640, k=3, stride=1),
        # optimizer step of a stage with 400 M parameters: norm, clip, Adam, bf16 copy
        dict(name="adam_step", kind="adam", matrices=24, rows=8192, cols=2048),
        # a whole training step of a small GPT (launch- and latency-bound)
        dict(name="small_gpt_train_step", kind="step", layers=2, B=4, mbs=2, S=256, H=512, NH=4, V=2048),
        # scoring: logits of one prompt through a four-layer GPT
        dict(name="gpt_logits", kind="logits", layers=4, B=1, S=512, H=1024, NH=8, V=51200),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "attention", "mlp", "layernorm", "embedding", "head",
                       "conv", "adam", "step", "logits"])
    if kind == "attention":
        HD, NH = rng.choice([64, 128]), rng.choice([4, 8, 12, 16, 20])
        form = rng.choice(["causal", "causal", "full", "cross"])
        SQ = _log_int(rng, 64, 2048)
        SK = _log_int(rng, 64, 2048) if form == "cross" else SQ
        B = max(1, min(32, _log_int(rng, 1, 32), int(16 * 16 * 2048 ** 2 * 128 * 0.5 / (NH * SQ * SK * HD))))
        return dict(kind=kind, B=B, NH=NH, SQ=SQ, SK=SK, HD=HD, causal=form == "causal", cross=form == "cross",
                    lens=form != "causal" and rng.random() < 0.6, bias=form == "full" and rng.random() < 0.4,
                    dropout=rng.choice([0.0, 0.1]), train=rng.random() < 0.75)
    if kind == "mlp":
        H = 64 * _log_int(rng, 8, 32)
        return dict(kind=kind, rows=_log_int(rng, 64, 8192), H=H, F=4 * H, dropout=rng.choice([0.0, 0.1]))
    if kind == "layernorm":
        return dict(kind=kind, rows=_log_int(rng, 64, 32768), H=64 * _log_int(rng, 8, 32))
    if kind == "embedding":
        return dict(kind=kind, B=rng.randint(1, 8), S=_log_int(rng, 64, 2048), V=1024 * _log_int(rng, 2, 50),
                    H=64 * _log_int(rng, 8, 32), dropout=rng.choice([0.0, 0.1]))
    if kind == "head":
        return dict(kind=kind, rows=_log_int(rng, 64, 4096), V=1024 * _log_int(rng, 2, 50), H=64 * _log_int(rng, 8, 32))
    if kind == "conv":
        HW = rng.choice([7, 14, 28, 56])
        ch = 8 * _log_int(rng, 8, 80)
        return dict(kind=kind, N=_log_int(rng, 1, max(1, min(64, 16 * (28 * 640) ** 2 // (HW * ch) ** 2))), HW=HW, C=ch,
                    K=ch, k=rng.choice([3, 3, 1]), stride=rng.choice([1, 1, 2]))
    if kind == "adam":
        return dict(kind=kind, matrices=rng.randint(1, 24), rows=_log_int(rng, 64, 8192), cols=64 * _log_int(rng, 2, 32))
    NH = rng.choice([2, 4, 8])
    if kind == "step":
        return dict(kind=kind, layers=rng.randint(1, 3), B=4, mbs=rng.choice([1, 2, 4]), S=_log_int(rng, 64, 512),
                    H=NH * 128, NH=NH, V=1024 * rng.randint(1, 8))
    return dict(kind=kind, layers=rng.randint(1, 4), B=rng.randint(1, 2), S=_log_int(rng, 64, 512), H=NH * 128, NH=NH,
                V=1024 * _log_int(rng, 2, 50))


# ------------------------------------------------- inputs -------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def _param(t):
    """A parameter as the framework's store holds it: the tensor and its fp32 gradient buffer."""
    p = torch.nn.Parameter(t)
    p.main_grad = torch.zeros(t.shape, dtype=torch.float32, device=t.device)
    return p


def _attention_inputs(c, g):
    w = c["NH"] * c["HD"]
    if c["cross"]:
        q, kv = _randn(g, c["B"] * c["SQ"], w), _randn(g, c["B"] * c["SK"], 2 * w)
    else:
        q, kv = _randn(g, c["B"] * c["SQ"], 3 * w), None
    do = _randn(g, c["B"] * c["SQ"], w)
    lens = None
    if c["lens"]:
        lens = torch.randint(max(1, c["SK"] // 2), c["SK"] + 1, (c["B"],), generator=g, device="cuda", dtype=torch.int32)
    bias = _randn(g, c["NH"], c["SQ"] + c["SK"] - 1, dtype=torch.float32) if c["bias"] else None
    return dict(q=q, kv=kv, do=do, lens=lens, bias=bias)


def _mlp_inputs(c, g):
    return dict(x=_randn(g, c["rows"], c["H"]), w1=_randn(g, c["F"], c["H"], std=0.02), b1=_randn(g, c["F"], std=0.02),
                w2=_randn(g, c["H"], c["F"], std=0.02), b2=_randn(g, c["H"], std=0.02), res=_randn(g, c["rows"], c["H"]),
                dy=_randn(g, c["rows"], c["H"]))


def _layernorm_inputs(c, g):
    return dict(x=_randn(g, c["rows"], c["H"]), gamma=1 + _randn(g, c["H"], std=0.1, dtype=torch.float32),
                beta=_randn(g, c["H"], std=0.1, dtype=torch.float32), dy=_randn(g, c["rows"], c["H"]),
                dres=_randn(g, c["rows"], c["H"]))


def _embedding_inputs(c, g):
    ids = torch.randint(0, c["V"], (c["B"], c["S"]), generator=g, device="cuda")
    return dict(ids=ids, pos=torch.arange(c["S"], device="cuda").repeat(c["B"]), W=_randn(g, c["V"], c["H"], std=0.02),
                P=_randn(g, c["S"], c["H"], std=0.02), dy=_randn(g, c["B"] * c["S"], c["H"]))


def _head_inputs(c, g):
    return dict(x=_randn(g, c["rows"], c["H"]), W=_randn(g, c["V"], c["H"], std=0.02),
                targets=torch.randint(0, c["V"], (c["rows"],), generator=g, device="cuda"))


def _conv_out(c):
    return (c["HW"] + 2 * (c["k"] // 2) - c["k"]) // c["stride"] + 1


def _conv_inputs(c, g):
    kk, o = c["k"] * c["k"] * c["C"], _conv_out(c)
    return dict(x=_randn(g, c["N"], c["HW"], c["HW"], c["C"]).relu(), w=_randn(g, c["K"], kk, std=(2.0 / kk) ** 0.5),
                gamma=1 + _randn(g, c["K"], std=0.1, dtype=torch.float32),
                beta=_randn(g, c["K"], std=0.1, dtype=torch.float32), dy=_randn(g, c["N"], o, o, c["K"]))


def _adam_inputs(c, g):
    n = c["matrices"] * c["rows"] * c["cols"]
    return dict(w=_randn(g, n, std=0.02), grad=_randn(g, n, std=1e-3, dtype=torch.float32),
                m=_randn(g, n, std=1e-3, dtype=torch.float32), v=_randn(g, n, std=1e-3, dtype=torch.float32).square())


def _gpt_weights(c, g):
    """Parameters of the GPT op list by name (the word embeddings are tied to the head)."""
    H, L = c["H"], c["layers"]
    out_std = 0.02 / math.sqrt(2.0 * L)
    w = {"ops.0.word_embeddings.weight": _randn(g, c["V"], H, std=0.02).float(),
         "ops.0.position_embeddings.weight": _randn(g, c["S"], H, std=0.02).float()}
    for i in range(L):
        b = 1 + 13 * i
        for k, name, shape, std in ((1, "query_key_value", (3, H, H), 0.02), (6, "dense", (H, H), out_std),
                                    (9, "dense_h_to_4h", (4 * H, H), 0.02), (11, "dense_4h_to_h", (H, 4 * H), out_std)):
            w[f"ops.{b + k}.{name}.weight"] = _randn(g, *shape, std=std).float()
            w[f"ops.{b + k}.{name}.bias"] = _randn(g, *shape[:-1], std=0.02).float()
        for k in (0, 8):
            w[f"ops.{b + k}.layernorm.weight"] = 1 + _randn(g, H, std=0.1, dtype=torch.float32)
            w[f"ops.{b + k}.layernorm.bias"] = _randn(g, H, std=0.02, dtype=torch.float32)
    b = 1 + 13 * L
    w[f"ops.{b}.layernorm.weight"] = 1 + _randn(g, H, std=0.1, dtype=torch.float32)
    w[f"ops.{b}.layernorm.bias"] = _randn(g, H, std=0.02, dtype=torch.float32)
    return w


def _gpt_inputs(c, g):
    t = torch.randint(0, c["V"], (c["B"], c["S"] + 1), generator=g, device="cuda")
    return dict(ids=t[:, :-1].contiguous(), labels=t[:, 1:].contiguous(), weights=_gpt_weights(c, g))


_INPUTS = dict(attention=_attention_inputs, mlp=_mlp_inputs, layernorm=_layernorm_inputs, embedding=_embedding_inputs,
               head=_head_inputs, conv=_conv_inputs, adam=_adam_inputs, step=_gpt_inputs, logits=_gpt_inputs)

_LR, _BETAS, _EPS, _WD, _CLIP = 1.5e-4, (0.9, 0.999), 1e-8, 0.01, 1.0


def _adam_state(c, d):
    from superscaler_b200.parallel.state import ParallelState
    from superscaler_b200.runtime.optimizer import StageOptimizer
    from superscaler_b200.runtime.params import ParamSpec, ParamStore
    store = ParamStore(torch.device("cuda", torch.cuda.current_device()))
    for i in range(c["matrices"]):
        store.declare(ParamSpec(name=f"w{i}", shape=(c["rows"], c["cols"]), init="zeros"))
    store.materialize()
    store.master.copy_(d["w"].float())
    store.model16.copy_(d["w"])
    store.grad.copy_(d["grad"])
    store.exp_avg.copy_(d["m"])
    store.exp_avg_sq.copy_(d["v"])
    opt = StageOptimizer(store, ParallelState([1]), lr=_LR, betas=_BETAS, eps=_EPS, weight_decay=_WD, clip_grad=_CLIP)
    opt.step_count = 99
    return dict(store=store, opt=opt)


def _trainer(c, weights, training):
    from superscaler_b200.models.gpt import gpt_op_names
    from superscaler_b200.runtime.trainer import Trainer
    n = len(gpt_op_names(c["layers"]))
    plan = dict(model_name="gpt", model_size="small", num_layers=c["layers"], seq_length=c["S"],
                max_position_embeddings=c["S"], num_attention_heads=c["NH"], hidden_size=c["H"], kv_channels=128,
                vocab_size=c["V"], global_batch_size=c["B"], micro_batch_size=c.get("mbs", c["B"]), num_stages=1,
                num_gpus=[1], checkpoint_activations=[False], resharding_stages=[False], num_ops_in_each_stage=[n],
                model_parallel_size_of_each_op=[[1] * n], data_parallel_size_of_each_op=[[1] * n],
                recompute_ops=[[0] * n], algo_of_each_op=[[0] * n])
    t = Trainer(plan, lr=_LR, min_lr=_LR, weight_decay=_WD, clip_grad=_CLIP, lr_warmup_steps=0, training=training,
                model_overrides=dict(hidden_dropout=0.0, attention_dropout=0.0))
    t.store.load_state_dict(weights)
    return t


def prepare(case, seed):
    kind = case["kind"]
    d = _INPUTS[kind](case, _gen(seed))
    s = dict(case=case, d=d)
    if kind == "attention" and case["train"]:
        for k in ("q", "kv", "bias"):
            if d[k] is not None:
                d[k].requires_grad_(True)
    elif kind in ("mlp", "layernorm", "embedding", "head", "conv"):
        if "x" in d:
            d["x"].requires_grad_(True)
        if "res" in d:
            d["res"].requires_grad_(True)
        for k in ("w1", "b1", "w2", "b2", "gamma", "beta", "W", "P", "w"):
            if k in d:
                d[k] = _param(d[k])
        if kind == "conv":
            s["run_mean"] = torch.zeros(case["K"], device="cuda")
            s["run_var"] = torch.ones(case["K"], device="cuda")
    elif kind == "adam":
        s.update(_adam_state(case, d))
        del s["d"]
    elif kind in ("step", "logits"):
        s["trainer"] = _trainer(case, d["weights"], kind == "step")
        del d["weights"]
        if kind == "step":   # a data loader's batch: pinned host memory
            s["batch"] = {k: d[k].cpu().pin_memory() for k in ("ids", "labels")}
    return s


# --------------------------------------------------- one pass ---------------------------------------------------
def run(state):
    return _RUN[state["case"]["kind"]](state, state["case"], state.get("d"))


def _attend(c, d):
    w, q, kv = c["NH"] * c["HD"], d["q"], d["kv"]
    k, cols = (kv, (0, 0, w)) if c["cross"] else (q, (0, w, 2 * w))
    return F.flash_attention(q, k, k, c["B"], c["NH"], c["SQ"], c["SK"], c["HD"], cols=cols, causal=c["causal"],
                             kv_lens=d["lens"], dropout_p=c["dropout"], seed=_SEED, bias_table=d["bias"])


def _run_attention(s, c, d):
    if not c["train"]:
        with torch.no_grad():
            return {"o": _attend(c, d)}
    ins = {k: d[k] for k in ("q", "kv", "bias") if d[k] is not None}
    for t in ins.values():
        t.grad = None
    o = _attend(c, d)
    o.backward(d["do"])
    return {"o": o.detach(), **{"d" + k: t.grad for k, t in ins.items()}}


def _zero(d, names):
    for k in names:
        d[k].main_grad.zero_()


def _run_mlp(s, c, d):
    names = ("w1", "b1", "w2", "b2")
    _zero(d, names)
    d["x"].grad = d["res"].grad = None
    y = F.mlp(d["x"], d["w1"], d["b1"], d["w2"], d["b2"], residual=d["res"], act=F.ACT_GELU, dropout_p=c["dropout"],
              seed=_SEED)
    y.backward(d["dy"])
    return {"y": y.detach(), "dx": d["x"].grad, "dres": d["res"].grad, **{"d" + k: d[k].main_grad for k in names}}


def _run_layernorm(s, c, d):
    _zero(d, ("gamma", "beta"))
    d["x"].grad = None
    y, keep = F.layernorm_keep_input(d["x"], d["gamma"], d["beta"], 1e-5)
    torch.autograd.backward([y, keep], [d["dy"], d["dres"]])
    return {"y": y.detach(), "dx": d["x"].grad, "dgamma": d["gamma"].main_grad, "dbeta": d["beta"].main_grad}


def _run_embedding(s, c, d):
    _zero(d, ("W", "P"))
    y = F.embedding(d["ids"], d["pos"], d["W"], d["P"], 0, c["dropout"], _SEED)
    y.backward(d["dy"])
    return {"y": y.detach(), "dW": d["W"].main_grad, "dP": d["P"].main_grad}


def _run_head(s, c, d):
    _zero(d, ("W",))
    d["x"].grad = None
    loss = F.lm_head_cross_entropy(d["x"], d["W"], d["targets"], None, 0, 1.0 / c["rows"])
    loss.backward()
    return {"loss": loss.detach(), "dx": d["x"].grad, "dW": d["W"].main_grad}


def _run_conv(s, c, d):
    _zero(d, ("w", "gamma", "beta"))
    d["x"].grad = None
    y = C.conv2d(d["x"], d["w"], c["k"], c["k"], c["stride"], c["k"] // 2)
    y = C.batch_norm(y, d["gamma"], d["beta"], None, s["run_mean"], s["run_var"], 1e-5, 0.1, True)
    y.backward(d["dy"])
    return {"y": y.detach(), "dx": d["x"].grad, "dw": d["w"].main_grad, "dgamma": d["gamma"].main_grad,
            "dbeta": d["beta"].main_grad}


def _run_adam(s, c, d):
    s["opt"].step(zero_grad=False)
    st = s["store"]
    return {"master": st.master, "exp_avg": st.exp_avg, "exp_avg_sq": st.exp_avg_sq, "model16": st.model16}


def _moments(store, flat):
    return {k: flat[o:o + n].view(store.params[k].shape) for k, (o, n) in store.offsets.items()}


def _run_step(s, c, d):
    t = s["trainer"]
    stats = t.train_step(s["batch"])
    return {"loss": stats["loss_tensor"], "master": t.store.master, "exp_avg": _moments(t.store, t.store.exp_avg)}


def _run_logits(s, c, d):
    return {"logits": s["trainer"].logits(d["ids"])}


_RUN = dict(attention=_run_attention, mlp=_run_mlp, layernorm=_run_layernorm, embedding=_run_embedding, head=_run_head,
            conv=_run_conv, adam=_run_adam, step=_run_step, logits=_run_logits)


# ------------------------------------------ what a pass cannot do without ------------------------------------------
def _gpt_matrix_params(c):
    return c["layers"] * 12 * c["H"] ** 2


def work(case):
    c, kind = case, case["kind"]
    if kind == "attention":
        w = c["NH"] * c["HD"]
        pairs = c["B"] * c["NH"] * c["SQ"] * c["SK"] * (0.5 if c["causal"] else 0.75 if c["lens"] else 1.0)
        io = 2 * c["B"] * (2 * c["SQ"] + 2 * c["SK"]) * w
        table = 4 * c["NH"] * (c["SQ"] + c["SK"] - 1) if c["bias"] else 0
        if not c["train"]:
            return {"bytes": io + table, "flops": 4 * pairs * c["HD"]}
        grads = 2 * c["B"] * (2 * c["SQ"] + 2 * c["SK"]) * w
        return {"bytes": io + grads + 2 * table, "flops": 14 * pairs * c["HD"]}
    if kind == "mlp":
        r, H, Fd = c["rows"], c["H"], c["F"]
        return {"bytes": 2 * r * H * 6 + 2 * H * Fd * (2 + 4), "flops": 12 * r * H * Fd}
    if kind == "layernorm":
        return {"bytes": 2 * c["rows"] * c["H"] * 5 + 16 * c["H"], "flops": 12 * c["rows"] * c["H"]}
    if kind == "embedding":
        n = c["B"] * c["S"]
        return {"bytes": n * 8 + 2 * min(n, c["V"]) * c["H"] + 2 * c["S"] * c["H"] + 4 * n * c["H"]
                + 4 * (c["V"] + c["S"]) * c["H"], "flops": 4 * n * c["H"]}
    if kind == "head":
        return {"bytes": 4 * c["rows"] * c["H"] + (2 + 4) * c["V"] * c["H"], "flops": 6 * c["rows"] * c["V"] * c["H"]}
    if kind == "conv":
        rows, wn = c["N"] * _conv_out(c) ** 2, c["K"] * c["C"] * c["k"] ** 2
        return {"bytes": 2 * (2 * c["N"] * c["HW"] ** 2 * c["C"] + 2 * rows * c["K"]) + 6 * wn,
                "flops": 6 * rows * wn}
    n = c["matrices"] * c["rows"] * c["cols"] if kind == "adam" else 0
    if kind == "adam":
        return {"bytes": n * (4 * 4 + 3 * 4 + 2), "flops": 14 * n}
    tokens, mats = c["B"] * c["S"], _gpt_matrix_params(c)
    att = c["layers"] * 4 * 0.5 * tokens * c["S"] * c["H"]
    if kind == "logits":
        return {"bytes": 2 * (mats + c["V"] * c["H"]) + 2 * tokens * c["V"],
                "flops": 2 * tokens * (mats + c["V"] * c["H"]) + att}
    n = mats + (c["V"] + c["S"]) * c["H"]
    return {"bytes": n * (2 + 7 * 4 + 2), "flops": 6 * tokens * (mats + c["V"] * c["H"]) + 3.5 * att}


def tolerance(case):
    # bf16 operands and results (8 significant bits) and fp32 sums everywhere but the optimizer; in the whole-model cases
    # the rounding of a layer travels through those that follow
    return {"adam": {"rel": 1e-4}, "step": {"rel": 4e-2}, "logits": {"rel": 3e-2}, "layernorm": {"rel": 5e-3},
            "embedding": {"rel": 5e-3}}.get(case["kind"], {"rel": 1.5e-2})


# --------------------------------------------- the same pass in 64 bits ---------------------------------------------
def exact(case, seed):
    if case.get("dropout"):
        return None     # the mask is the framework's own counter-based stream
    return _EXACT[case["kind"]](case, _INPUTS[case["kind"]](case, _gen(seed)))


def _attention64(c, q, k, v, lens, bias, b, h):
    """One head of one sample: [SQ, HD] from [SQ, HD], [SK, HD], [SK, HD]."""
    s = q @ k.t() / math.sqrt(c["HD"])
    i, j = torch.arange(c["SQ"], device="cuda")[:, None], torch.arange(c["SK"], device="cuda")[None, :]
    if bias is not None:
        s = s + bias[h][j - i + c["SQ"] - 1]
    if c["causal"]:
        s = s.masked_fill(j > i, -math.inf)
    if lens is not None:
        s = s.masked_fill(j >= lens[b], -math.inf)
    return torch.softmax(s, -1) @ v


def _exact_attention(c, d):
    w, hd, train = c["NH"] * c["HD"], c["HD"], c["train"]
    q, kv = d["q"].double(), d["kv"].double() if c["cross"] else None
    bias = d["bias"].double() if c["bias"] else None
    do = d["do"].double()
    o = torch.empty_like(do)
    dq, dkv = torch.zeros_like(q), torch.zeros_like(kv) if kv is not None else None
    dbias = torch.zeros_like(bias) if bias is not None else None
    for b in range(c["B"]):
        rq, rk = slice(b * c["SQ"], (b + 1) * c["SQ"]), slice(b * c["SK"], (b + 1) * c["SK"])
        src, gsrc, k0 = (kv, dkv, 0) if c["cross"] else (q, dq, w)
        for h in range(c["NH"]):
            a, e = h * hd, (h + 1) * hd
            parts = [q[rq, a:e], src[rk, k0 + a:k0 + e], src[rk, k0 + w + a:k0 + w + e]]
            parts = [p.detach().clone().requires_grad_(train) for p in parts]
            bb = bias.detach().clone().requires_grad_(train) if bias is not None else None
            y = _attention64(c, *parts, d["lens"], bb, b, h)
            o[rq, a:e] = y.detach()
            if train:
                g = torch.autograd.grad(y, parts + ([bb] if bb is not None else []), do[rq, a:e])
                dq[rq, a:e] = g[0]
                gsrc[rk, k0 + a:k0 + e] = g[1]
                gsrc[rk, k0 + w + a:k0 + w + e] = g[2]
                if bb is not None:
                    dbias += g[3]
    if not train:
        return {"o": o}
    return {"o": o, "dq": dq, **({"dkv": dkv} if c["cross"] else {}), **({"dbias": dbias} if c["bias"] else {})}


def _grads(y, dy, leaves):
    return dict(zip(("d" + k for k in leaves), torch.autograd.grad(y, list(leaves.values()), dy)))


def _leaf64(d, names):
    return {k: d[k].double().requires_grad_(True) for k in names}


def _exact_mlp(c, d):
    t = _leaf64(d, ("x", "res", "w1", "b1", "w2", "b2"))
    y = t["res"] + TF.gelu(t["x"] @ t["w1"].t() + t["b1"], approximate="tanh") @ t["w2"].t() + t["b2"]
    return {"y": y.detach(), **_grads(y, d["dy"].double(), t)}


def _exact_layernorm(c, d):
    t = _leaf64(d, ("x", "gamma", "beta"))
    y = TF.layer_norm(t["x"], (c["H"],), t["gamma"], t["beta"], 1e-5)
    out = {"y": y.detach(), **_grads(y, d["dy"].double(), t)}
    out["dx"] = out["dx"] + d["dres"].double()
    return out


def _exact_embedding(c, d):
    t = _leaf64(d, ("W", "P"))
    y = t["W"][d["ids"].reshape(-1)] + t["P"][d["pos"]]
    return {"y": y.detach(), **_grads(y, d["dy"].double(), t)}


def _exact_head(c, d):
    t = _leaf64(d, ("x", "W"))
    loss = TF.cross_entropy(t["x"] @ t["W"].t(), d["targets"])
    return {"loss": loss.detach(), **_grads(loss, None, t)}


def _exact_conv(c, d):
    t = _leaf64(d, ("x", "w", "gamma", "beta"))
    w = t["w"].view(c["K"], c["k"], c["k"], c["C"])
    p, o, st = c["k"] // 2, _conv_out(c), c["stride"]
    x = TF.pad(t["x"], (0, 0, p, p, p, p))
    y = 0
    for i in range(c["k"]):
        for j in range(c["k"]):
            y = y + x[:, i:i + st * (o - 1) + 1:st, j:j + st * (o - 1) + 1:st] @ w[:, i, j].t()
    m, v = y.mean((0, 1, 2)), y.var((0, 1, 2), unbiased=False)
    y = torch.relu((y - m) / torch.sqrt(v + 1e-5) * t["gamma"] + t["beta"])
    return {"y": y.detach(), **_grads(y, d["dy"].double(), t)}


def _exact_adam(c, d):
    w, g, m, v = (d[k].double() for k in ("w", "grad", "m", "v"))
    g = g * min(1.0, _CLIP / (float(g.square().sum().sqrt()) + 1e-6))
    m = _BETAS[0] * m + (1 - _BETAS[0]) * g
    v = _BETAS[1] * v + (1 - _BETAS[1]) * g * g
    step = (m / (1 - _BETAS[0] ** 100)) / ((v / (1 - _BETAS[1] ** 100)).sqrt() + _EPS)
    w = w - _LR * (step + _WD * w)
    return {"master": w, "exp_avg": m, "exp_avg_sq": v, "model16": w}


def _gpt64(c, w, ids):
    B, S, H, NH = ids.shape[0], c["S"], c["H"], c["NH"]
    x = w["ops.0.word_embeddings.weight"][ids] + w["ops.0.position_embeddings.weight"][None]

    def ln(x, i):
        return TF.layer_norm(x, (H,), w[f"ops.{i}.layernorm.weight"], w[f"ops.{i}.layernorm.bias"], 1e-5)

    def lin(x, name):
        k = w[name + ".weight"].reshape(-1, w[name + ".weight"].shape[-1])
        return x @ k.t() + w[name + ".bias"].reshape(-1)

    for i in range(c["layers"]):
        b = 1 + 13 * i
        q, k, v = (t.view(B, S, NH, -1).transpose(1, 2) for t in
                   lin(ln(x, b), f"ops.{b + 1}.query_key_value").chunk(3, -1))
        s = (q @ k.transpose(-1, -2)) / math.sqrt(H // NH)
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), -math.inf)
        x = x + lin((torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, S, H), f"ops.{b + 6}.dense")
        h = TF.gelu(lin(ln(x, b + 8), f"ops.{b + 9}.dense_h_to_4h"), approximate="tanh")
        x = x + lin(h, f"ops.{b + 11}.dense_4h_to_h")
    return ln(x, 1 + 13 * c["layers"]) @ w["ops.0.word_embeddings.weight"].t()


def _exact_logits(c, d):
    with torch.no_grad():
        return {"logits": _gpt64(c, {k: v.double() for k, v in d["weights"].items()}, d["ids"])}


def _exact_step(c, d):
    w = {k: v.double().requires_grad_(True) for k, v in d["weights"].items()}
    loss = TF.cross_entropy(_gpt64(c, w, d["ids"]).view(-1, c["V"]), d["labels"].reshape(-1))
    g = dict(zip(w, torch.autograd.grad(loss, list(w.values()))))
    clip = min(1.0, _CLIP / (float(sum(t.square().sum() for t in g.values())) ** 0.5 + 1e-6))
    return {"loss": loss.detach().reshape(1), "master": None,
            "exp_avg": {k: (1 - _BETAS[0]) * clip * t for k, t in g.items()}}


_EXACT = dict(attention=_exact_attention, mlp=_exact_mlp, layernorm=_exact_layernorm, embedding=_exact_embedding,
              head=_exact_head, conv=_exact_conv, adam=_exact_adam, step=_exact_step, logits=_exact_logits)
