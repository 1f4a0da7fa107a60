"""The work this framework is measured on: its layers and operators through their public entry points, from the sizes
where launches count up to one layer of the large language models it trains.

``listed()`` names the cases, ``draw`` gives more of the same ranges, ``prepare`` makes what a program holds before the
call (inputs, weights, a cell or an optimizer), ``run`` is one pass, ``exact`` the same in 64-bit torch.

Kinds of a case (what they stand for):

* ``llama``   : a whole decoder, logits, mean loss and every weight gradient: the smoke-test network, launch-bound.
* ``attn``    : one attention layer of a decoder (fused QKV projection, rotary embedding, causal attention, output
                projection), forward and backward.
* ``flash``   : ``FlashAttentionScore`` by itself: grouped key / value heads in training, full attention as a prefill or an
                encoder runs it.
* ``mlp``     : the SwiGLU feed-forward layer of a decoder, forward and backward.
* ``dense``   : ``nn.Dense``: a projection of a few tokens as decoding runs it, or of many, with and without backward.
* ``norm``    : residual add + RMSNorm, or LayerNorm, forward and backward.
* ``ce``      : the loss over a vocabulary, forward and backward, some labels ignored.
* ``adamw``   : one optimizer step over the flat arena with gradient clipping.
* ``conv``    : a ResNet-50 bottleneck in training (convolutions, BatchNorm, ReLU, shortcut), forward and backward.
* ``moe``     : a mixture-of-experts feed-forward layer, router included, forward and backward.
"""
import math

import torch
import torch.nn.functional as F

import mindspore_b200 as ms
from mindspore_b200 import nn, ops
from mindspore_b200.models.llama import LlamaAttention, LlamaConfig, LlamaForCausalLM, LlamaMLP
from mindspore_b200.models.resnet import Bottleneck
from mindspore_b200.ops import fused
from mindspore_b200.parallel.moe import MoE, MoEConfig, calculate_expert_capacity

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
NORM_EPS = 1e-5
ADAMW = dict(learning_rate=3e-4, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, max_grad_norm=1.0)


def listed():
    return [
        # the network of the framework's smoke test: every kernel is short, launches and host time count
        dict(name="llama-tiny", kind="llama", vocab=2048, hidden=512, layers=2, heads=4, kv_heads=4, ffn=1408, seq=256,
             batch=2),
        # the attention layer of the benchmark's 7B decoder, one micro-batch
        dict(name="attn-7b", kind="attn", hidden=4096, heads=32, kv_heads=32, seq=4096, batch=1),
        # grouped key / value heads in training
        dict(name="flash-gqa-train", kind="flash", heads=32, kv_heads=8, seq=2048, batch=2, causal=True, dtype="bf16",
             backward=True),
        # full attention without gradients: prefill of an encoder, fp16
        dict(name="flash-full-fp16", kind="flash", heads=16, kv_heads=16, seq=1024, batch=4, causal=False, dtype="fp16",
             backward=False),
        # the feed-forward layer of the 7B decoder, one micro-batch
        dict(name="mlp-7b", kind="mlp", tokens=4096, hidden=4096, ffn=11008),
        # one projection of a few tokens, as a decoding step runs it
        dict(name="dense-decode", kind="dense", tokens=24, cin=4096, cout=4096, bias=True, dtype="bf16", backward=False),
        # residual add + RMSNorm of the 7B decoder
        dict(name="norm-7b", kind="norm", op="add_rms", rows=4096, hidden=4096, dtype="bf16"),
        # LayerNorm of the GPT 2.6B network on a ragged number of rows
        dict(name="layernorm-gpt", kind="norm", op="layer", rows=8191, hidden=2560, dtype="bf16"),
        # the loss of the 7B decoder, one micro-batch
        dict(name="ce-32000", kind="ce", rows=4096, vocab=32000, dtype="bf16"),
        # one optimizer step over the weights of one 7B decoder layer
        dict(name="adamw-layer", kind="adamw", hidden=4096, ffn=11008),
        # an identity bottleneck of the first ResNet-50 stage
        dict(name="bottleneck-56", kind="conv", batch=64, cin=256, width=64, stride=1, size=56),
        # one expert layer of the 8-expert network, one sequence
        dict(name="moe-8x", kind="moe", tokens=2048, hidden=4096, ffn=14336, experts=8, choices=2),
    ]


def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def _seq(rng, lo, hi):
    """Whole blocks of 128 tokens mostly, an arbitrary length sometimes."""
    return _log(rng, lo, hi) if rng.random() < 0.2 else _log(rng, lo, hi, 128)


def draw(rng):
    kind = rng.choice(["llama", "attn", "flash", "flash", "mlp", "dense", "dense", "norm", "norm", "ce", "adamw", "conv",
                       "moe"])
    if kind == "llama":
        heads = rng.choice([2, 4, 8])
        return dict(kind=kind, vocab=_log(rng, 512, 8192, 8), hidden=heads * 128, layers=rng.randint(1, 4), heads=heads,
                    kv_heads=heads, ffn=_log(rng, 512, 2816, 8), seq=_seq(rng, 128, 1024), batch=rng.randint(1, 4))
    if kind == "attn":
        heads = rng.choice([4, 8, 16, 32])
        return dict(kind=kind, hidden=heads * 128, heads=heads, kv_heads=heads if rng.random() < 0.6 else heads // 4,
                    seq=_seq(rng, 128, 4096), batch=1)
    if kind == "flash":
        heads, backward = rng.choice([4, 8, 16, 32]), rng.random() < 0.6
        seq = _seq(rng, 128, 4096)
        return dict(kind=kind, heads=heads, kv_heads=heads if rng.random() < 0.5 else heads // 4, seq=seq,
                    batch=rng.randint(1, max(1, min(4, 8192 // seq))), causal=rng.random() < 0.7,
                    dtype=rng.choice(["bf16", "bf16", "fp16"]), backward=backward)
    if kind == "mlp":
        return dict(kind=kind, tokens=_log(rng, 64, 4096), hidden=_log(rng, 512, 4096, 128),
                    ffn=_log(rng, 1408, 11008, 128))
    if kind == "dense":
        backward = rng.random() < 0.5
        return dict(kind=kind, tokens=_log(rng, 1, 8192), cin=_log(rng, 256, 8192, 8), cout=_log(rng, 256, 8192, 8),
                    bias=rng.random() < 0.5, dtype=rng.choice(["bf16", "bf16", "fp16"]), backward=backward)
    if kind == "norm":
        return dict(kind=kind, op=rng.choice(["add_rms", "layer"]), rows=_log(rng, 1, 16384),
                    hidden=_log(rng, 256, 8192, 8), dtype=rng.choice(["bf16", "bf16", "fp16"]))
    if kind == "ce":
        return dict(kind=kind, rows=_log(rng, 64, 8192), vocab=_log(rng, 1000, 50000),
                    dtype=rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "adamw":
        return dict(kind=kind, hidden=_log(rng, 256, 4096, 8), ffn=_log(rng, 704, 11008, 8))
    if kind == "conv":
        i = rng.randint(0, 3)
        first = rng.random() < 0.4
        width, size = 64 << i, 56 >> i
        stride = 2 if first and i else 1
        return dict(kind=kind, batch=_log(rng, 1, 64), cin=(width * 2 if stride == 2 else width * 4), width=width,
                    stride=stride, size=size * stride)
    return dict(kind=kind, tokens=_log(rng, 128, 2048), hidden=_log(rng, 512, 4096, 128), ffn=_log(rng, 1024, 7168, 128),
                experts=rng.choice([4, 8]), choices=rng.choice([1, 2]))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, dtype=torch.bfloat16, std=1.0, mean=0.0):
    t = torch.empty(shape, device="cuda", dtype=torch.float32).normal_(mean, std, generator=g)
    return t.to(dtype)


def _fill(p, g, std, mean=0.0):
    """Gives the parameter ``p`` seeded normal values."""
    with torch.no_grad():
        p.data.normal_(mean, std, generator=g)


def _context():
    ms.set_context(mode=ms.PYNATIVE_MODE, device_target="GPU", device_id=0)


def _leaf(t):
    return ms.Tensor(t).requires_grad_(True)


def _llama_config(c):
    return LlamaConfig(vocab_size=c["vocab"], hidden_size=c["hidden"], num_layers=c["layers"], num_heads=c["heads"],
                       num_kv_heads=c["kv_heads"], ffn_hidden_size=c["ffn"], seq_length=c["seq"])


def prepare(case, seed):
    _context()
    c, g = case, _gen(seed)
    s = {"case": c}
    kind = c["kind"]
    if kind == "llama":
        net = LlamaForCausalLM(_llama_config(c))
        for p in net.trainable_params():
            _fill(p, g, 0.1 if p.dim() == 1 else 0.03, 1.0 if p.dim() == 1 else 0.0)
        net.set_train()
        tok = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=g, device="cuda", dtype=torch.int32)
        s.update(net=net, loss=ops.SparseSoftmaxCrossEntropyWithLogits(), weights=net.trainable_params(),
                 tokens=ms.Tensor(tok[:, :-1].contiguous()), labels=ms.Tensor(tok[:, 1:].reshape(-1).contiguous()))
    elif kind in ("attn", "mlp"):
        cfg = LlamaConfig(hidden_size=c["hidden"], num_heads=c.get("heads", 4), num_kv_heads=c.get("kv_heads", 4),
                          ffn_hidden_size=c.get("ffn", 512), seq_length=c.get("seq", 128))
        tokens = c["tokens"] if kind == "mlp" else c["batch"] * c["seq"]
        net = LlamaMLP(cfg) if kind == "mlp" else LlamaAttention(cfg)
        for p in net.trainable_params():
            _fill(p, g, 1.0 / math.sqrt(p.shape[1]))
        x = _randn(g, (tokens, c["hidden"]))
        s.update(net=net, x=_leaf(x), weights=net.trainable_params(), dy=_randn(g, (tokens, c["hidden"]), std=0.1))
        if kind == "attn":
            s["rope"] = fused.rope_tables(c["seq"], cfg.head_dim, device="cuda")
    elif kind == "flash":
        dt, d = DTYPES[c["dtype"]], 128
        q, k, v = (_randn(g, (c["batch"], c["seq"], h * d), dt) for h in (c["heads"], c["kv_heads"], c["kv_heads"]))
        op = ops.FlashAttentionScore(head_num=c["heads"], scale_value=1.0 / math.sqrt(d), input_layout="BSH",
                                     next_tokens=0 if c["causal"] else 2147483647)
        if c["backward"]:
            s.update(op=op, qkv=tuple(_leaf(t) for t in (q, k, v)), dy=_randn(g, q.shape, dt, 0.1))
        else:
            s.update(op=op, qkv=tuple(ms.Tensor(t) for t in (q, k, v)))
    elif kind == "dense":
        dt = DTYPES[c["dtype"]]
        net = nn.Dense(c["cin"], c["cout"], has_bias=c["bias"], dtype=dt)
        for p in net.trainable_params():
            _fill(p, g, 1.0 / math.sqrt(c["cin"]))
        x = _randn(g, (c["tokens"], c["cin"]), dt)
        s.update(net=net, weights=net.trainable_params(), x=_leaf(x) if c["backward"] else ms.Tensor(x))
        if c["backward"]:
            s["dy"] = _randn(g, (c["tokens"], c["cout"]), dt, 0.1)
    elif kind == "norm":
        dt, shape = DTYPES[c["dtype"]], (c["rows"], c["hidden"])
        s.update(x=_leaf(_randn(g, shape, dt)), dy=_randn(g, shape, dt, 0.1))
        if c["op"] == "layer":
            net = nn.LayerNorm((c["hidden"],), epsilon=NORM_EPS, dtype=dt)
            _fill(net.gamma, g, 0.1, 1.0)
            _fill(net.beta, g, 0.1)
            s["net"] = net
        else:
            s.update(op=ops.AddRmsNorm(NORM_EPS), res=_leaf(_randn(g, shape, dt)), dstream=_randn(g, shape, dt, 0.1),
                     gamma=ms.Parameter(ms.Tensor(_randn(g, (c["hidden"],), dt, 0.1, 1.0)), name="gamma"))
    elif kind == "ce":
        labels = torch.randint(0, c["vocab"], (c["rows"],), generator=g, device="cuda", dtype=torch.int32)
        labels[torch.rand(c["rows"], generator=g, device="cuda") < 0.05] = -100
        s.update(op=ops.SparseSoftmaxCrossEntropyWithLogits(), labels=ms.Tensor(labels),
                 logits=_leaf(_randn(g, (c["rows"], c["vocab"]), DTYPES[c["dtype"]], 2.0)))
    elif kind == "adamw":
        params = [ms.Parameter(ms.Tensor(_randn(g, shape, std=0.02, mean=1.0 if len(shape) == 1 else 0.0)), name=name)
                  for name, shape in _layer_shapes(c)]
        opt = nn.AdamWeightDecay(params, **ADAMW)
        for p in params:
            p.main_grad.normal_(0.0, 1e-3, generator=g)
        s.update(opt=opt, params=params)
    elif kind == "conv":
        net = Bottleneck(c["cin"], c["width"], c["stride"], torch.bfloat16)
        for p in net.trainable_params():
            if p.dim() == 4:
                _fill(p, g, math.sqrt(2.0 / (p.shape[0] * p.shape[2] * p.shape[3])))
            else:
                _fill(p, g, 0.1, 1.0 if p.name.endswith("gamma") else 0.0)
        net.set_train()
        shape = (c["batch"], c["size"], c["size"], c["cin"])
        out = (c["batch"], c["size"] // c["stride"], c["size"] // c["stride"], c["width"] * 4)
        x = _randn(g, shape).relu_().permute(0, 3, 1, 2)                    # channels-last, after a ReLU
        s.update(net=net, weights=net.trainable_params(), x=_leaf(x), dy=_randn(g, out, std=0.1).permute(0, 3, 1, 2))
    elif kind == "moe":
        net = MoE(c["hidden"], c["ffn"], hidden_act="swiglu", param_init_type=torch.bfloat16, has_bias=False,
                  moe_config=MoEConfig(expert_num=c["experts"], capacity_factor=1.25, num_experts_chosen=c["choices"]))
        _fill(net.router_weight, g, 1.0 / math.sqrt(c["hidden"]))
        _fill(net.w1, g, 1.0 / math.sqrt(c["hidden"]))
        _fill(net.w2, g, 1.0 / math.sqrt(c["ffn"]))
        shape = (c["tokens"], c["hidden"])
        s.update(net=net, weights=(net.router_weight, net.w1, net.w2), x=_leaf(_randn(g, shape)),
                 dy=_randn(g, shape, std=0.1), daux=torch.ones((), device="cuda"))
    else:
        raise ValueError("unknown kind %r" % kind)
    return s


def _layer_shapes(c):
    """The weights of one decoder layer."""
    h, f = c["hidden"], c["ffn"]
    return [("attention_norm", (h,)), ("ffn_norm", (h,)), ("wqkv", (3 * h, h)), ("wo", (h, h)), ("w_gate_up", (2 * f, h)),
            ("w_down", (h, f))]


# ------------------------------------------------------------------------------------------------ one pass
def _grads(outs, wrt, douts=None):
    return list(torch.autograd.grad(outs, list(wrt), douts))


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "llama":
        logits = s["net"].logits(s["tokens"])
        loss = s["loss"](logits, s["labels"])
        return {"logits": logits, "loss": loss, "grads": _grads(loss, s["weights"])}
    if kind in ("attn", "mlp"):
        y = s["net"](s["x"], *s["rope"]) if kind == "attn" else s["net"](s["x"])
        return {"y": y, "grads": _grads(y, [s["x"], *s["weights"]], s["dy"])}
    if kind == "flash":
        o = s["op"](*s["qkv"])[3]
        return {"o": o, "grads": _grads(o, s["qkv"], s["dy"])} if c["backward"] else {"o": o}
    if kind == "dense":
        if not c["backward"]:
            with torch.no_grad():
                return {"y": s["net"](s["x"])}
        y = s["net"](s["x"])
        return {"y": y, "grads": _grads(y, [s["x"], *s["weights"]], s["dy"])}
    if kind == "norm":
        if c["op"] == "layer":
            y = s["net"](s["x"])
            return {"y": y, "grads": _grads(y, [s["x"], s["net"].gamma, s["net"].beta], s["dy"])}
        y, stream = s["op"](s["x"], s["res"], s["gamma"])
        return {"y": y, "stream": stream,
                "grads": _grads([y, stream], [s["x"], s["res"], s["gamma"]], [s["dy"], s["dstream"]])}
    if kind == "ce":
        loss = s["op"](s["logits"], s["labels"])
        return {"loss": loss, "grads": _grads(loss, [s["logits"]])}
    if kind == "adamw":
        s["opt"]()
        return {"weights": [p.data for p in s["params"]], "m": [p.data for p in s["opt"].moment1],
                "v": [p.data for p in s["opt"].moment2]}
    if kind == "conv":
        y = s["net"](s["x"])
        return {"y": y, "grads": _grads(y, [s["x"], *s["weights"]], s["dy"])}
    y, aux = s["net"](s["x"])
    return {"y": y, "aux": aux, "grads": _grads([y, aux], [s["x"], *s["weights"]], [s["dy"], s["daux"]])}


# ------------------------------------------------------------------------------------------------ work of one pass
def _attention_work(batch, seq, heads, kv_heads, causal, backward):
    flops = 4.0 * batch * heads * seq * seq * 128 * (0.5 if causal else 1.0)
    moved = 2.0 * batch * seq * 128 * (2 * heads + 2 * kv_heads)
    return flops * (3.5 if backward else 1.0), moved * (3 if backward else 1)


def work(case):
    c, kind = case, case["kind"]
    if kind == "llama":
        h, f, v, t = c["hidden"], c["ffn"], c["vocab"], c["batch"] * c["seq"]
        gemm = c["layers"] * (h * 3 * h + h * h + 3 * h * f) + v * h
        fa, _ = _attention_work(c["batch"], c["seq"], c["heads"], c["kv_heads"], True, True)
        return {"flops": 6.0 * gemm * t + c["layers"] * fa,
                "bytes": 2.0 * 2 * (gemm + v * h) + 2.0 * t * v + 2.0 * c["layers"] * t * (10 * h + 6 * f)}
    if kind == "attn":
        h, t, kv = c["hidden"], c["batch"] * c["seq"], c["kv_heads"] * 128
        w = h * (h + 2 * kv) + h * h
        fa, _ = _attention_work(c["batch"], c["seq"], c["heads"], c["kv_heads"], True, True)
        return {"flops": 6.0 * w * t + fa, "bytes": 2.0 * (2 * w + 4 * t * h)}
    if kind == "flash":
        fl, by = _attention_work(c["batch"], c["seq"], c["heads"], c["kv_heads"], c["causal"], c["backward"])
        return {"flops": fl, "bytes": by}
    if kind == "mlp":
        w, t = 3 * c["hidden"] * c["ffn"], c["tokens"]
        return {"flops": 6.0 * w * t, "bytes": 2.0 * (2 * w + 4 * t * c["hidden"])}
    if kind == "dense":
        w, t = c["cin"] * c["cout"], c["tokens"]
        if not c["backward"]:
            return {"flops": 2.0 * w * t, "bytes": 2.0 * (w + t * (c["cin"] + c["cout"]))}
        return {"flops": 6.0 * w * t, "bytes": 2.0 * (2 * w + 2 * t * (c["cin"] + c["cout"]))}
    if kind == "norm":
        n = c["rows"] * c["hidden"]
        return {"flops": 20.0 * n, "bytes": 2.0 * n * (8 if c["op"] == "add_rms" else 4)}
    if kind == "ce":
        n = c["rows"] * c["vocab"]
        return {"flops": 8.0 * n, "bytes": (4.0 if c["dtype"] == "fp32" else 2.0) * 2 * n}
    if kind == "adamw":
        n = sum(math.prod(sh) for _, sh in _layer_shapes(c))
        return {"flops": 16.0 * n, "bytes": 30.0 * n}
    if kind == "conv":
        b, w, cin, si, st = c["batch"], c["width"], c["cin"], c["size"], c["stride"]
        so = si // st
        macs = si * si * cin * w + so * so * w * w * 9 + so * so * w * w * 4
        down = st != 1 or cin != 4 * w
        macs += so * so * cin * 4 * w if down else 0
        return {"flops": 6.0 * b * macs, "bytes": 2.0 * b * (2 * si * si * cin + 2 * so * so * 4 * w)}
    w = 3 * c["hidden"] * c["ffn"]
    rows = c["choices"] * c["tokens"]
    return {"flops": 6.0 * w * rows, "bytes": 2.0 * (2 * w * c["experts"] + 4 * c["tokens"] * c["hidden"])}


def tolerance(case):
    """About four times the relative error against ``exact`` that the operators showed when this was written: 9e-4 (loss
    gradient), 1.7e-3 to 3.5e-3 (one or two bf16 roundings: norms, GEMMs, attention), 5e-3 (attention layer, experts),
    1.1e-2 (decoder of bf16 layers), an eighth of the bf16 figures in fp16, and about 8e-2 for the bottleneck, where a
    16-bit rounding in front of a ReLU flips some of its signs and each flip passes or drops a whole gradient value."""
    kind, dt = case["kind"], case.get("dtype", "bf16")
    if dt == "fp16":
        return {"rel": 1.5e-3}
    if dt == "fp32":
        return {"rel": 1e-5}
    return {"rel": {"llama": 4e-2, "conv": 2e-1, "moe": 2e-2, "attn": 2e-2, "mlp": 1.4e-2, "ce": 4e-3,
                    "adamw": 7e-3}.get(kind, 1.2e-2)}


# ------------------------------------------------------------------------------------------------ 64-bit results
def _d(t, grad=False):
    return t.detach().as_subclass(torch.Tensor).double().requires_grad_(grad)


def _rms(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + NORM_EPS) * w


def _rotate(x, cos, sin):
    """x [batch, seq, heads, d], rotate-half."""
    a, b = x.chunk(2, -1)
    cos, sin = cos[None, :, None, :], sin[None, :, None, :]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, causal):
    """[batch, seq, heads, 128] each, one head at a time."""
    mask = torch.ones(q.shape[1], q.shape[1], device=q.device, dtype=torch.bool).triu(1) if causal else None
    group = q.shape[2] // k.shape[2]

    def one(b, h):
        p = q[b, :, h] @ k[b, :, h // group].t() / math.sqrt(128)
        p = p.masked_fill(mask, -math.inf) if causal else p
        return torch.softmax(p, -1) @ v[b, :, h // group]

    return torch.stack([torch.stack([torch.utils.checkpoint.checkpoint(one, b, h, use_reentrant=False)
                                     for h in range(q.shape[2])], 1) for b in range(q.shape[0])], 0)


def _rotary_attention(qkv, batch, seq, heads, kv_heads):
    inv = 1.0 / (10000.0 ** (torch.arange(0, 128, 2, device=qkv.device, dtype=torch.float64) / 128))
    ang = torch.outer(torch.arange(seq, device=qkv.device, dtype=torch.float64), inv)
    q, k, v = (t.reshape(batch, seq, -1, 128) for t in qkv.split([heads * 128, kv_heads * 128, kv_heads * 128], -1))
    o = _attend(_rotate(q, ang.cos(), ang.sin()), _rotate(k, ang.cos(), ang.sin()), v, True)
    return o.reshape(batch * seq, heads * 128)


def _swiglu(gu):
    gate, up = gu.chunk(2, -1)
    return F.silu(gate) * up


def _exact_llama(s, c):
    names = [p.name for p in s["weights"]]
    w = {n: _d(p, True) for n, p in zip(names, s["weights"])}

    def find(layer, name):
        want = "layers.%d." % layer
        return next(w[n] for n in names if want in n and n.endswith("." + name))

    def top(name):
        return next(w[n] for n in names if n.split(".")[-1] == name)

    x = F.embedding(s["tokens"].as_subclass(torch.Tensor).reshape(-1).long(), top("tok_embeddings"))
    for i in range(c["layers"]):
        a = _rotary_attention(_rms(x, find(i, "attention_norm")) @ find(i, "wqkv").t(), c["batch"], c["seq"], c["heads"],
                              c["kv_heads"])
        x = x + a @ find(i, "wo").t()
        x = x + _swiglu(_rms(x, find(i, "ffn_norm")) @ find(i, "w_gate_up").t()) @ find(i, "w_down").t()
    logits = _rms(x, top("norm_out")) @ top("lm_head").t()
    loss = F.cross_entropy(logits, s["labels"].as_subclass(torch.Tensor).long())
    return {"logits": logits, "loss": loss, "grads": _grads(loss, [w[n] for n in names])}


def _exact_conv(s, c):
    w = {p.name: _d(p, True) for p in s["weights"]}
    x = _d(s["x"], True)

    def unit(name, t, stride, pad):
        get = lambda part: next(w[n] for n in w if name + "." in n and n.endswith(part))  # noqa: E731
        y = F.conv2d(t, get("conv.weight"), None, stride, pad)
        return F.batch_norm(y, None, None, get("gamma"), get("beta"), True, 0.0, 1e-5)

    short = unit("down", x, c["stride"], 0) if any("down." in n for n in w) else x
    y = torch.relu(unit("conv1", x, 1, 0))
    y = torch.relu(unit("conv2", y, c["stride"], 1))
    y = torch.relu(unit("conv3", y, 1, 0) + short)
    return {"y": y, "grads": _grads(y, [x, *w.values()], _d(s["dy"]))}


def _exact_moe(s, c):
    x, (rw, w1, w2) = _d(s["x"], True), (_d(p, True) for p in s["weights"])
    T, E, K = c["tokens"], c["experts"], c["choices"]
    cap = (calculate_expert_capacity(K, T, 1.25, E) + 7) // 8 * 8
    prob, taken = torch.softmax(x @ rw.t(), -1), torch.zeros(T, E, device=x.device, dtype=torch.float64)
    fill, aux, gates, picks = torch.zeros(E, device=x.device, dtype=torch.long), 0.0, [], []
    for _ in range(K):
        left = prob * (1 - taken)
        gate, idx = left.max(-1)
        mask = F.one_hot(idx, E).double()
        aux = aux + (mask.mean(0) * (left / (left.sum(-1, keepdim=True) + 1e-9)).mean(0)).mean() * E * E
        pos = ((torch.cumsum(mask, 0) - mask).long() + fill).gather(1, idx[:, None])[:, 0]
        kept = mask * (pos < cap)[:, None]
        taken, fill = taken + kept, fill + kept.sum(0).long()
        gates.append(gate * (pos < cap))
        picks.append((idx, pos < cap))
    gate = torch.stack(gates, 1)
    weight = gate / (gate.sum(-1, keepdim=True) + 1e-9) if K > 1 else gate
    y = torch.zeros_like(x)
    for e in range(E):
        for j, (idx, keep) in enumerate(picks):
            rows = torch.nonzero((idx == e) & keep)[:, 0]
            y = y.index_add(0, rows, _swiglu(x[rows] @ w1[e]) @ w2[e] * weight[rows, j:j + 1])
    aux = aux * 0.05
    return {"y": y, "aux": aux, "grads": _grads([y, aux], [x, rw, w1, w2], [_d(s["dy"]), _d(s["daux"])])}


def _exact_adamw(s):
    lr, b1, b2 = ADAMW["learning_rate"], ADAMW["beta1"], ADAMW["beta2"]
    gr = [_d(p.main_grad) for p in s["params"]]
    norm = math.sqrt(sum(float(g.pow(2).sum()) for g in gr))
    scale = min(1.0, ADAMW["max_grad_norm"] / (norm + 1e-6))
    weights, ms_, vs = {}, {}, {}
    for p, g in zip(s["params"], gr):
        w, g = _d(p), g * scale
        m, v = (1 - b1) * g, (1 - b2) * g * g
        w = w * (1 - lr * ADAMW["weight_decay"] * (p.dim() > 1))
        weights[p.name] = w - lr * (m / (1 - b1)) / ((v / (1 - b2)).sqrt() + ADAMW["eps"])
        ms_[p.name], vs[p.name] = m, v
    order = lambda ps, d: [d[next(n for n in d if p.name.endswith(n))] for p in ps]  # noqa: E731
    return {"weights": order(s["params"], weights), "m": order(s["opt"].moment1, ms_), "v": order(s["opt"].moment2, vs)}


def exact(case, seed):
    import torch.utils.checkpoint  # noqa: F401
    s, c = prepare(case, seed), case
    kind = c["kind"]
    if kind == "llama":
        return _exact_llama(s, c)
    if kind == "conv":
        return _exact_conv(s, c)
    if kind == "moe":
        return _exact_moe(s, c)
    if kind == "adamw":
        return _exact_adamw(s)
    if kind == "flash":
        q, k, v = (_d(t, True) for t in s["qkv"])
        o = _attend(*(t.reshape(c["batch"], c["seq"], -1, 128) for t in (q, k, v)), c["causal"]).reshape(q.shape)
        return {"o": o, "grads": _grads(o, [q, k, v], _d(s["dy"]))} if c["backward"] else {"o": o.detach()}
    if kind == "ce":
        logits = _d(s["logits"], True)
        loss = F.cross_entropy(logits, s["labels"].as_subclass(torch.Tensor).long())
        return {"loss": loss, "grads": _grads(loss, [logits])}
    x = _d(s["x"], True)
    if kind == "norm" and c["op"] == "add_rms":
        res, gamma = _d(s["res"], True), _d(s["gamma"], True)
        stream = x + res
        y = _rms(stream, gamma)
        return {"y": y, "stream": stream, "grads": _grads([y, stream], [x, res, gamma], [_d(s["dy"]), _d(s["dstream"])])}
    if kind == "norm":
        w = [_d(s["net"].gamma, True), _d(s["net"].beta, True)]
        y = F.layer_norm(x, (c["hidden"],), *w, NORM_EPS)
    else:
        w = [_d(p, True) for p in s["weights"]]
        named = {p.name.split(".")[-1]: t for p, t in zip(s["weights"], w)}
        if kind == "attn":
            y = _rotary_attention(x @ named["wqkv"].t(), c["batch"], c["seq"], c["heads"], c["kv_heads"]) @ named["wo"].t()
        elif kind == "mlp":
            y = _swiglu(x @ named["w_gate_up"].t()) @ named["w_down"].t()
        else:
            y = F.linear(x, named["weight"], named.get("bias"))
            if not c["backward"]:
                return {"y": y}
    return {"y": y, "grads": _grads(y, [x, *w], _d(s["dy"]))}
