# SPDX-License-Identifier: Apache-2.0
"""What the performance of this framework is measured on: the layers, the optimizer and the training step of GPT-2 as a
user's program calls them, over sizes from one short sequence to the full micro-batch of the training benchmark.

A case is a dict of plain values. Its "kind" names the public entry points that one pass goes through:

  attention  ops.Attention.forward_packed + backward_packed on the packed qkv projection (head dimension 64, bf16)
  mlp        the feed-forward half of a block, forward + backward with weight gradients: linear with the GELU epilogue,
             GELU-linear with the residual added, and their four backward products
  linear     one projection, forward + backward with the weight gradient (and the bias gradient where it has a bias)
  head       classifier and cross-entropy in one op, forward + backward
  norm       LayerNorm forward, and backward with the residual gradient added
  embed      token + position embedding, forward + backward
  adamw      one AdamW step of fp32 master weights with a bf16 working copy
  logits     the forward pass of a whole GPT-2 to its logits
  train      one training step of a whole GPT-2: forward, backward, AdamW

Weights and activations are drawn as bf16 values, so a 64-bit computation of the same pass starts from exactly the same
numbers; gradients that come into a layer are scaled like those of a mean loss over its rows.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import core_scheduler_b200 as cs
from core_scheduler_b200 import ops
from core_scheduler_b200.models import PRESETS, gpt2_config
from core_scheduler_b200.parallel import GPT2Trainer

C = cs._C
BF = torch.bfloat16
DEV = "cuda"
_scheduler = None


def _s():
    """One scheduler for the process, as a training program has."""
    global _scheduler
    if _scheduler is None:
        _scheduler = cs.DynamicScheduler(0, device=DEV)
    return _scheduler


def listed():
    return [
        # attention of the 124M model at the training benchmark's micro-batch
        dict(name="attention_train", kind="attention", batch=16, seq=1024, heads=12, causal=True),
        # long context, few sequences, the head count of the 774M model
        dict(name="attention_long", kind="attention", batch=2, seq=4096, heads=20, causal=True),
        # a short sequence without a causal mask: an encoder or a small fine-tuning batch
        dict(name="attention_short", kind="attention", batch=4, seq=256, heads=12, causal=False),
        # feed-forward of the 124M model at the training benchmark's micro-batch
        dict(name="mlp_train", kind="mlp", rows=16384, width=768, bias=False),
        # feed-forward of the 774M width on a ragged number of tokens, with biases
        dict(name="mlp_ragged", kind="mlp", rows=3000, width=1280, bias=True),
        # the qkv projection of the 350M width on one short sequence: launches and latency count
        dict(name="linear_small", kind="linear", rows=128, inp=1024, out=3072, bias=False),
        # classifier + loss of the 124M model at the training benchmark's micro-batch
        dict(name="head_train", kind="head", rows=16384, width=768, vocab=50257, padded=50304),
        # LayerNorm of the 774M width on 32 sequences of 1024
        dict(name="norm_large", kind="norm", rows=32768, width=1280),
        # embedding tables of the 124M model at the training benchmark's micro-batch
        dict(name="embed_train", kind="embed", batch=16, seq=1024, width=768, vocab=50304, positions=1024),
        # all parameters of the 124M model (untied classifier) in one optimizer step
        dict(name="adamw_model", kind="adamw", n=162_991_104),
        # evaluation of a batch of prompts with the 124M model
        dict(name="logits_eval", kind="logits", model="124M", batch=4, seq=384),
        # the training step of the 124M model, micro-batch 8
        dict(name="train_step", kind="train", model="124M", batch=8, seq=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "mlp", "mlp", "linear", "linear", "head", "norm", "embed",
                       "adamw", "logits"])
    if kind == "attention":
        heads = rng.choice([4, 8, 12, 16, 20])
        seq = 128 * _log(rng, 1, 32)
        if rng.random() < 0.2:  # a sequence that is no multiple of a tile
            seq = max(8, seq - rng.randrange(1, 127))
        batch = _log(rng, 1, max(1, min(64, 16 * 1024 * 12 // (seq * heads))))
        return dict(kind=kind, batch=batch, seq=seq, heads=heads, causal=rng.random() < 0.75)
    if kind == "mlp":
        width = rng.choice([256, 512, 768, 1000, 1024, 1280, 1600])
        return dict(kind=kind, rows=_log(rng, 16, 16384 * 768 * 768 // (width * width)), width=width, bias=rng.random() < 0.4)
    if kind == "linear":
        inp, out = rng.choice([(768, 768), (768, 2304), (1024, 1024), (1024, 3072), (1280, 1280), (1280, 3840), (520, 1000), (768, 3072)])
        return dict(kind=kind, rows=_log(rng, 1, 16384), inp=inp, out=out, bias=rng.random() < 0.4)
    if kind == "head":
        vocab, padded = rng.choice([(50257, 50304), (32000, 32000), (512, 512), (10000, 10112)])
        width = rng.choice([256, 768, 1024, 1280])
        return dict(kind=kind, rows=_log(rng, 64, 16384 * 768 // max(768, width)), width=width, vocab=vocab, padded=padded)
    if kind == "norm":
        return dict(kind=kind, rows=_log(rng, 64, 32768), width=rng.choice([256, 768, 1000, 1024, 1280, 1600, 2048]))
    if kind == "embed":
        seq = _log(rng, 16, 1024)
        return dict(kind=kind, batch=_log(rng, 1, 16), seq=seq, width=rng.choice([256, 768, 1024, 1280]), vocab=rng.choice([10000, 50304]),
                    positions=1024)
    if kind == "adamw":
        return dict(kind=kind, n=_log(rng, 10_000, 162_991_104))
    return dict(kind=kind, model=rng.choice(["124M", "350M"]), batch=_log(rng, 1, 4), seq=128 * rng.randint(1, 4))


# ------------------------------------------------------------------------------------ inputs ----
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, *shape, std=1.0):
    """Normal values that bf16 holds exactly, as bf16."""
    return torch.empty(shape, device=DEV).normal_(0.0, std, generator=g).to(BF)


def _ids(g, vocab, *shape):
    """Token ids with the skew of text: a few ids make up much of a batch, most of the vocabulary is rare."""
    u = torch.empty(shape, device=DEV).uniform_(0.0, 1.0, generator=g)
    return (torch.exp(u * math.log(vocab)) - 1.0).to(torch.int64).clamp_(0, vocab - 1)


def _inputs(case, seed):
    """Every tensor of a case, from the seed alone."""
    g = _gen(seed)
    k = case["kind"]
    if k == "attention":
        b, t, w = case["batch"], case["seq"], case["heads"] * 64
        return dict(qkv=_normal(g, b, t, 3 * w), dout=_normal(g, b, t, w, std=1e-2))
    if k == "mlp":
        r, w = case["rows"], case["width"]
        return dict(x=_normal(g, r, w), res=_normal(g, r, w), dy=_normal(g, r, w, std=1e-2), w1=_normal(g, 4 * w, w, std=0.5 / math.sqrt(w)),
                    w2=_normal(g, w, 4 * w, std=0.5 / math.sqrt(w)), b1=_normal(g, 4 * w, std=0.1), b2=_normal(g, w, std=0.1))
    if k == "linear":
        r, i, o = case["rows"], case["inp"], case["out"]
        return dict(x=_normal(g, r, i), dy=_normal(g, r, o, std=1e-2), w=_normal(g, o, i, std=1.0 / math.sqrt(i)), b=_normal(g, o, std=0.1))
    if k == "head":
        return dict(x=_normal(g, case["rows"], case["width"]), w=_normal(g, case["padded"], case["width"], std=1.0 / math.sqrt(case["width"])),
                    target=_ids(g, case["vocab"], case["rows"]))
    if k == "norm":
        r, w = case["rows"], case["width"]
        return dict(x=_normal(g, r, w, std=2.0), dy=_normal(g, r, w, std=1e-2), res=_normal(g, r, w, std=1e-2),
                    gamma=_normal(g, w, std=0.2) + 1, beta=_normal(g, w, std=0.2))
    if k == "embed":
        w = case["width"]
        return dict(ids=_ids(g, case["vocab"], case["batch"], case["seq"]), wte=_normal(g, case["vocab"], w, std=0.02),
                    wpe=_normal(g, case["positions"], w, std=0.02), dy=_normal(g, case["batch"], case["seq"], w, std=1e-3))
    if k == "adamw":
        n = case["n"]
        f = lambda std: torch.empty(n, device=DEV).normal_(0.0, std, generator=g)  # noqa: E731
        return dict(w=f(0.02), g=f(1e-3), m=f(1e-4), v=f(1e-3).square_())
    _, _, d, _, vocab, _ = PRESETS[case["model"]]
    ids = _ids(g, vocab, case["batch"], case["seq"] + 1)
    return dict(ids=ids[:, :-1].contiguous(), labels=ids[:, 1:].contiguous())


def _model_shapes(name):
    n_layer, _, d, block, _, padded = PRESETS[name]
    shapes = {"wte.weight": (padded, d), "wpe.weight": (block, d)}
    for l in range(n_layer):
        shapes.update({f"{l}.ln1.weight": (d,), f"{l}.ln1.bias": (d,), f"{l}.attn.c_attn.weight": (3 * d, d), f"{l}.attn.c_proj.weight": (d, d),
                       f"{l}.ln2.weight": (d,), f"{l}.ln2.bias": (d,), f"{l}.mlp.fc1.weight": (4 * d, d), f"{l}.mlp.fc2.weight": (d, 4 * d)})
    shapes.update({"lnf.weight": (d,), "lnf.bias": (d,), "lm_head.weight": (padded, d)})
    return shapes


def _model_weights(name, seed):
    """Weights of a model part of the way through training rather than at its start: gains that differ from one."""
    g = _gen(seed + 7919)
    out = {}
    for key, shape in _model_shapes(name).items():
        if len(shape) == 1:
            out[key] = _normal(g, *shape, std=0.1) + (1 if key.endswith("weight") else 0)
        else:
            out[key] = _normal(g, *shape, std=0.02)
    return out


def _set(handle, value):
    """Gives a parameter its value: the handle's own storage, in its own type."""
    handle.raw().copy_(value.to(handle.raw().dtype).view(handle.raw().shape))


def prepare(case, seed):
    s, k, x = _s(), case["kind"], _inputs(case, seed)
    st = dict(kind=k)
    if k == "attention":
        st.update(op=ops.Attention(s, is_causal=case["causal"]), heads=case["heads"])
    elif k == "mlp":
        w = case["width"]
        fc1 = C.linear_init(s, w, 4 * w, bias=case["bias"], gelu_epilogue=True)
        fc2 = C.gelu_linear_init(s, 4 * w, w, bias=case["bias"])
        torch.cuda.synchronize()
        _set(fc1.weight, x.pop("w1"))
        _set(fc2.weight, x.pop("w2"))
        b1, b2 = x.pop("b1"), x.pop("b2")
        if case["bias"]:
            _set(fc1.bias, b1)
            _set(fc2.bias, b2)
        st.update(fc1=fc1, fc2=fc2, bias=case["bias"])
    elif k == "linear":
        op = ops.Linear(s, case["inp"], case["out"], bias=case["bias"])
        torch.cuda.synchronize()
        _set(op.weight, x.pop("w"))
        b = x.pop("b")
        if case["bias"]:
            _set(op.bias, b)
        st.update(op=op, bias=case["bias"])
    elif k == "head":
        linear = ops.Linear(s, case["width"], case["padded"], bias=False)
        torch.cuda.synchronize()
        _set(linear.weight, x.pop("w"))
        st.update(linear=linear, op=ops.LinearCrossEntropy(s, linear, valid_classes=case["vocab"]))
    elif k == "norm":
        op = ops.LayerNorm(s, case["width"])
        torch.cuda.synchronize()
        _set(op.weight, x.pop("gamma"))
        _set(op.bias, x.pop("beta"))
        st.update(op=op)
    elif k == "embed":
        wte, wpe = ops.Embedding(s, case["vocab"], case["width"]), ops.Embedding(s, case["positions"], case["width"])
        torch.cuda.synchronize()
        _set(wte.weight, x.pop("wte"))
        _set(wpe.weight, x.pop("wpe"))
        st.update(wte=wte, wpe=wpe)
    elif k == "adamw":
        weight = cs.from_torch(x.pop("w"))
        C.working_copy(s, weight, BF)
        op = ops.AdamW(s, weight, lr=3e-4, beta1=0.9, beta2=0.95, weight_decay=0.1)
        torch.cuda.synchronize()
        op.state.m.raw().copy_(x.pop("m"))
        op.state.v.raw().copy_(x.pop("v"))
        st.update(op=op, weight=weight)
    else:
        config = gpt2_config(case["model"])
        if k == "train":
            trainer = GPT2Trainer(config, device=DEV, scheduler=s, lr=3e-4)
            model = trainer.model
            st.update(trainer=trainer)
        else:
            x.pop("labels")
            model = cs.GPT2(s, config)
            st.update(flat=C.flatten_parameters(s, model, lp_dtype=BF))
        torch.cuda.synchronize()
        named = model.named_parameters()
        for key, value in _model_weights(case["model"], seed).items():
            _set(named[key], value)
            lp = named[key].lp()
            if lp is not None:
                lp.copy_(value.view(lp.shape))
        st.update(model=model)
    torch.cuda.synchronize()
    # the tensors stay with the state; the handles are what the calls take
    st.update(tensors=x, handles={name: cs.from_torch(t) for name, t in x.items()})
    return st


def run(state):
    s, k, h = _s(), state["kind"], state["handles"]
    if k == "attention":
        out = state["op"].forward_packed(h["qkv"], state["heads"])
        dqkv = state["op"].backward_packed(h["dout"])
        return dict(out=out.raw(), dqkv=dqkv.raw())
    if k == "mlp":
        fc1, fc2 = state["fc1"], state["fc2"]
        with cs.autocast(s, BF):
            pre = C.linear_forward(s, fc1, h["x"])
            y = C.gelu_linear_forward(s, fc2, pre, h["res"])
        dpre = C.gelu_linear_backward_input(s, fc2, h["dy"])
        C.gelu_linear_backward_parameter(s, fc2, h["dy"])
        dx = C.linear_backward_input(s, fc1, dpre)
        C.linear_backward_parameter(s, fc1, dpre)
        out = dict(y=y.raw(), dx=dx.raw(), dw1=fc1.grad_weight.raw(), dw2=fc2.grad_weight.raw())
        if state["bias"]:
            out.update(db1=fc1.grad_bias.raw(), db2=fc2.grad_bias.raw())
        fc1.zero_grad()
        fc2.zero_grad()
        return out
    if k == "linear":
        op = state["op"]
        with cs.autocast(s, BF):
            y = op.forward(h["x"])
        dx = op.backward(h["dy"])
        out = dict(y=y.raw(), dx=dx.raw(), dw=op.grad_weight.raw())
        if state["bias"]:
            out.update(db=op.grad_bias.raw())
        op.zero_grad()
        return out
    if k == "head":
        with cs.autocast(s, BF):
            loss = state["op"].forward(h["x"], h["target"])
        dx = state["op"].backward()
        out = dict(loss=loss.raw(), dx=dx.raw(), dw=state["linear"].grad_weight.raw())
        state["linear"].zero_grad()
        return out
    if k == "norm":
        op = state["op"]
        with cs.autocast(s, BF):
            y = op.forward(h["x"])
        dx = op.backward(h["dy"], h["res"])
        out = dict(y=y.raw(), dx=dx.raw(), dgamma=op.grad_weight.raw(), dbeta=op.state.grad_bias.raw())
        op.zero_grad()
        return out
    if k == "embed":
        wte, wpe = state["wte"], state["wpe"]
        with cs.autocast(s, BF):
            y = C.embedding_forward_token_position(s, wte.state, wpe.state, h["ids"])
        C.embedding_backward_token_position(s, wte.state, wpe.state, h["dy"])
        out = dict(y=y.raw(), dwte=wte.grad_weight.raw(), dwpe=wpe.grad_weight.raw())
        wte.zero_grad()
        wpe.zero_grad()
        return out
    if k == "adamw":
        op, w = state["op"], state["weight"]
        op.step(w, h["g"])
        return dict(w=w.raw(), m=op.state.m.raw(), v=op.state.v.raw(), copy=w.lp())
    if k == "logits":
        with cs.autocast(s, BF):
            return state["model"].forward(s, h["ids"]).raw()
    loss = state["trainer"].step(h["ids"], h["labels"])
    return dict(loss=loss.raw(), weights=state["trainer"].flat.params.raw())


# ------------------------------------------------------------------------------- what it costs ----
def work(case):
    k = case["kind"]
    if k == "attention":
        b, t, w = case["batch"], case["seq"], case["heads"] * 64
        pairs = t * (t + 1) / 2 if case["causal"] else t * t
        # forward 2 products, backward 5; qkv read twice, out and its gradient, dqkv
        return dict(bytes=b * t * w * 2 * (3 + 1 + 3 + 1 + 1 + 3), flops=7 * 2.0 * b * pairs * w)
    if k == "mlp":
        r, w = case["rows"], case["width"]
        return dict(bytes=r * w * 2 * (1 + 1 + 1 + 1 + 1) + 8 * w * w * (2 + 4), flops=6 * 2.0 * r * 4 * w * w)
    if k == "linear":
        r, i, o = case["rows"], case["inp"], case["out"]
        return dict(bytes=r * (2 * i + 2 * o) * 2 + i * o * (2 + 4), flops=3 * 2.0 * r * i * o)
    if k == "head":
        r, w, v = case["rows"], case["width"], case["padded"]
        return dict(bytes=r * w * 4 + v * w * (2 + 4) + r * 8, flops=3 * 2.0 * r * w * v)
    if k == "norm":
        r, w = case["rows"], case["width"]
        return dict(bytes=r * w * 2 * (2 + 4), flops=0)
    if k == "embed":
        r, w = case["batch"] * case["seq"], case["width"]
        return dict(bytes=r * w * 2 * 2 + r * 8 + min(r, case["vocab"]) * w * 4 + (case["vocab"] + case["positions"]) * w * 4, flops=0)
    if k == "adamw":
        return dict(bytes=case["n"] * (4 * 4 + 3 * 4 + 2), flops=0)
    n_layer, _, d, _, _, padded = PRESETS[case["model"]]
    tokens, t = case["batch"] * case["seq"], case["seq"]
    matmul = 2.0 * tokens * (12 * n_layer * d * d + padded * d)
    attention = 2 * 2.0 * n_layer * case["batch"] * t * (t + 1) / 2 * d
    params = sum(math.prod(shape) for shape in _model_shapes(case["model"]).values())
    if k == "logits":
        return dict(bytes=(params - padded * d) * 2 + tokens * padded * 2, flops=matmul + attention)
    return dict(bytes=params * (2 + 2 + 4 + 4 * 4 + 3 * 4 + 2), flops=3 * matmul + 3.5 * attention)


def tolerance(case):
    # relative errors against 64 bits, measured: bf16 results of one layer 2e-3 to 4e-3; a whole forward pass 1e-2
    k = case["kind"]
    if k == "adamw":
        return dict(rel=4e-3, max=2e-2)  # the bf16 copy may round the other way; the fp32 state is far closer
    if k == "logits":
        return dict(rel=2.5e-2, max=0.3)
    if k == "train":
        return dict(rel=1e-2, max=0.5)
    return dict(rel=1e-2, max=0.3)


# ---------------------------------------------------------------------------- the same in 64 bits ----
def _exact_attention(qkv, dout, heads, causal):
    """[t, 3w], [t, w] -> out [t, w], dqkv [t, 3w]; one sequence, in blocks of heads."""
    t, w = dout.shape
    out, dqkv = torch.empty(t, w, device=DEV, dtype=torch.float64), torch.empty(t, 3 * w, device=DEV, dtype=torch.float64)
    mask = torch.ones(t, t, device=DEV, dtype=torch.bool).tril() if causal else None
    q, k, v = (x.reshape(t, heads, 64).transpose(0, 1) for x in qkv.split(w, dim=1))
    do = dout.reshape(t, heads, 64).transpose(0, 1)
    for h in range(heads):
        s = (q[h] @ k[h].t()) * 0.125
        if causal:
            s.masked_fill_(~mask, float("-inf"))
        p = torch.softmax(s, -1)
        o = p @ v[h]
        dp = do[h] @ v[h].t()
        ds = p * (dp - (do[h] * o).sum(-1, keepdim=True)) * 0.125
        cols = slice(h * 64, (h + 1) * 64)
        out[:, cols] = o
        dqkv[:, cols] = ds @ k[h]
        dqkv[:, w + h * 64:w + (h + 1) * 64] = ds.t() @ q[h]
        dqkv[:, 2 * w + h * 64:2 * w + (h + 1) * 64] = p.t() @ do[h]
    return out, dqkv


class _Attention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, heads):
        w = qkv.shape[1] // 3
        ctx.save_for_backward(qkv)
        ctx.heads = heads
        return _exact_attention(qkv, torch.zeros(qkv.shape[0], w, device=DEV, dtype=torch.float64), heads, True)[0]

    @staticmethod
    def backward(ctx, dout):
        return _exact_attention(ctx.saved_tensors[0], dout, ctx.heads, True)[1], None


def _gelu_grad(x):
    return 0.5 * (1 + torch.erf(x / math.sqrt(2))) + x * torch.exp(-0.5 * x * x) / math.sqrt(2 * math.pi)


def _exact_logits(case, weights, ids):
    """[t] ids of one sequence -> [t, padded]"""
    n_layer, heads, d, _, _, _ = PRESETS[case["model"]]
    x = weights["wte.weight"][ids] + weights["wpe.weight"][:ids.shape[0]]
    for l in range(n_layer):
        a = F.layer_norm(x, (d,), weights[f"{l}.ln1.weight"], weights[f"{l}.ln1.bias"])
        x = x + _Attention.apply(a @ weights[f"{l}.attn.c_attn.weight"].t(), heads) @ weights[f"{l}.attn.c_proj.weight"].t()
        b = F.layer_norm(x, (d,), weights[f"{l}.ln2.weight"], weights[f"{l}.ln2.bias"])
        x = x + F.gelu(b @ weights[f"{l}.mlp.fc1.weight"].t()) @ weights[f"{l}.mlp.fc2.weight"].t()
    x = F.layer_norm(x, (d,), weights["lnf.weight"], weights["lnf.bias"])
    return x @ weights["lm_head.weight"].t()


def exact(case, seed):
    k = case["kind"]
    x = {name: t.double() if t.is_floating_point() else t for name, t in _inputs(case, seed).items()}
    if k == "attention":
        parts = [_exact_attention(q, d, case["heads"], case["causal"]) for q, d in zip(x["qkv"], x["dout"])]
        return dict(out=torch.stack([p[0] for p in parts]), dqkv=torch.stack([p[1] for p in parts]))
    if k == "mlp":
        pre = x["x"] @ x["w1"].t()
        if case["bias"]:
            pre = pre + x["b1"]
        act = F.gelu(pre)
        y = act @ x["w2"].t() + x["res"]
        if case["bias"]:
            y = y + x["b2"]
        dpre = (x["dy"] @ x["w2"]) * _gelu_grad(pre)
        out = dict(y=y, dx=dpre @ x["w1"], dw1=dpre.t() @ x["x"], dw2=x["dy"].t() @ act)
        if case["bias"]:
            out.update(db1=dpre.sum(0), db2=x["dy"].sum(0))
        return out
    if k == "linear":
        y = x["x"] @ x["w"].t()
        out = dict(y=y + x["b"] if case["bias"] else y, dx=x["dy"] @ x["w"], dw=x["dy"].t() @ x["x"])
        if case["bias"]:
            out.update(db=x["dy"].sum(0))
        return out
    if k == "head":
        rows, v = case["rows"], case["vocab"]
        loss, dx, dw = 0.0, torch.empty_like(x["x"]), torch.zeros_like(x["w"])
        for at in range(0, rows, 2048):
            xs, ts = x["x"][at:at + 2048], x["target"][at:at + 2048]
            logp = torch.log_softmax(xs @ x["w"][:v].t(), -1)
            loss = loss - logp.gather(1, ts[:, None]).sum() / rows
            dl = logp.exp_()
            dl[torch.arange(ts.shape[0], device=DEV), ts] -= 1
            dl /= rows
            dx[at:at + 2048] = dl @ x["w"][:v]
            dw[:v] += dl.t() @ xs
        return dict(loss=loss, dx=dx, dw=dw)
    if k == "norm":
        mean, var = x["x"].mean(-1, keepdim=True), x["x"].var(-1, unbiased=False, keepdim=True)
        rstd = 1 / torch.sqrt(var + 1e-5)
        xh = (x["x"] - mean) * rstd
        dyg = x["dy"] * x["gamma"]
        dx = rstd * (dyg - dyg.mean(-1, keepdim=True) - xh * (dyg * xh).mean(-1, keepdim=True)) + x["res"]
        return dict(y=xh * x["gamma"] + x["beta"], dx=dx, dgamma=(x["dy"] * xh).sum(0), dbeta=x["dy"].sum(0))
    if k == "embed":
        w, t = case["width"], case["seq"]
        dwte = torch.zeros(case["vocab"], w, device=DEV, dtype=torch.float64).index_add_(0, x["ids"].reshape(-1), x["dy"].reshape(-1, w))
        dwpe = torch.zeros(case["positions"], w, device=DEV, dtype=torch.float64)
        dwpe[:t] = x["dy"].sum(0)
        return dict(y=x["wte"][x["ids"]] + x["wpe"][:t], dwte=dwte, dwpe=dwpe)
    if k == "adamw":
        m = 0.9 * x["m"] + 0.1 * x["g"]
        v = 0.95 * x["v"] + 0.05 * x["g"] ** 2
        w = x["w"] * (1 - 3e-4 * 0.1) - 3e-4 * (m / (1 - 0.9)) / (torch.sqrt(v / (1 - 0.95)) + 1e-8)
        return dict(w=w, m=m, v=v, copy=w)
    weights = {name: t.double() for name, t in _model_weights(case["model"], seed).items()}
    if k == "logits":
        with torch.no_grad():
            return torch.stack([_exact_logits(case, weights, ids) for ids in x["ids"]])
    vocab = PRESETS[case["model"]][4]
    weights = {name: t.requires_grad_(True) for name, t in weights.items()}
    total = 0.0
    for ids, labels in zip(x["ids"], x["labels"]):
        loss = F.cross_entropy(_exact_logits(case, weights, ids)[:, :vocab], labels) / case["batch"]
        loss.backward()
        total = total + loss.detach()
    with torch.no_grad():
        new = [t * (1 - 3e-4 * 0.1) - 3e-4 * t.grad / (t.grad.abs() + 1e-8) for t in weights.values()]
    return dict(loss=total, weights=torch.cat([t.reshape(-1) for t in new]))
