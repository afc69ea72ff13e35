"""Performance cases of the framework: its layers, blocks and whole calls over the sizes that they are used at.

Every case is a dict of plain values. ``prepare`` makes what a program holds before the call (inputs, weights, a trainer),
``run`` is one pass through the public entry points, ``work`` the bytes and operations that no implementation can avoid,
``exact`` the same outputs in 64-bit arithmetic with plain PyTorch.

Kinds:

* ``logits``       a whole GPT-2 forward pass without gradients (scoring, one step of ``generate``)
* ``mlp``          the GELU MLP of a GPT-2 block, inference (few rows) or training (forward and backward)
* ``attention``    flash attention on the packed QKV projection (GPT-2) or on separate q, k, v (Llama)
* ``llama_block``  one Llama decoder block, forward and backward: RMSNorm, rotary positions, attention, SwiGLU
* ``norm``         LayerNorm / RMSNorm, forward and backward
* ``head``         LM head and fused cross-entropy with the vocabulary padded to 64, forward and backward
* ``bottleneck``   one ResNet bottleneck in training: 1x1, 3x3, 1x1 convolutions with BatchNorm, forward and backward
* ``train_step``   a GPT-2 training step through ``CausalLMTrainer``, the batch coming from pinned host memory
"""
import math

import torch

from torsh_b200 import nn
from torsh_b200.engine import CausalLMTrainer
from torsh_b200.models.gpt2 import GPT2Config, GPTForCausalLM
from torsh_b200.models.llama import LlamaBlock, LlamaConfig
from torsh_b200.models.resnet import BottleneckBlock
from torsh_b200.ops.attention import flash_attention, flash_attention_qkvpacked
from torsh_b200.ops.linear import linear, mlp_gelu
from torsh_b200.ops.norm import layer_norm, rms_norm
from torsh_b200.ops.softmax import cross_entropy

DEV = "cuda"
BF16 = torch.bfloat16
STEPS_BEFORE = 10
NO_DROPOUT = dict(embd_pdrop=0.0, attn_pdrop=0.0, resid_pdrop=0.0)


def listed():
    return [
        # scoring one short prompt with the 4-layer smoke configuration: all launch latency
        dict(name="logits_tiny", kind="logits", model="tiny", batch=1, seq=33),
        # a handful of rows through one GPT-2-medium MLP: weight streaming, the shape of batched token-by-token work
        dict(name="mlp_rows13", kind="mlp", rows=13, embd=1024, train=False),
        # the same MLP in the training step of the benchmark (batch 8 x 1024 tokens)
        dict(name="mlp_train", kind="mlp", rows=8192, embd=1024, train=True),
        # attention of the benchmark's training step
        dict(name="attn_train_d64", kind="attention", batch=8, seq=1024, heads=16, dim=64, causal=True, packed=True, train=True),
        # encoder-style inference on a ragged length, no mask
        dict(name="attn_infer_ragged", kind="attention", batch=3, seq=1531, heads=12, dim=64, causal=False, packed=False, train=False),
        # long-context training with Llama's head size
        dict(name="attn_train_d128", kind="attention", batch=2, seq=4096, heads=16, dim=128, causal=True, packed=False, train=True),
        # one Llama-7B block in training
        dict(name="llama_block", kind="llama_block", batch=1, seq=2048, embd=4096, ffn=11008, heads=32),
        # a LayerNorm of a large batch in training
        dict(name="layernorm_train", kind="norm", rows=32768, embd=1024, dtype="bf16", rms=False),
        # a full-precision RMSNorm with an odd row count
        dict(name="rmsnorm_fp32", kind="norm", rows=1999, embd=4096, dtype="fp32", rms=True),
        # LM head and loss over GPT-2's vocabulary
        dict(name="head_train", kind="head", rows=4096, embd=1024, vocab=50257),
        # a stage-1 bottleneck of ResNet-50 in training
        dict(name="bottleneck_train", kind="bottleneck", batch=64, hw=56, planes=64),
        # the benchmark: a GPT-2-medium training step
        dict(name="train_step", kind="train_step", model="medium", batch=8, seq=1024),
    ]


def _log(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["logits", "mlp", "mlp", "attention", "attention", "llama_block", "norm", "norm", "head", "bottleneck", "train_step"])
    if kind == "logits":
        if rng.random() < 0.5:
            return dict(kind=kind, model="tiny", batch=rng.randint(1, 8), seq=_log(rng, 2, 128))
        return dict(kind=kind, model="small", batch=rng.randint(1, 4), seq=_log(rng, 8, 1024))
    if kind == "mlp":
        train = rng.random() < 0.6
        return dict(kind=kind, rows=_log(rng, 64, 8192) if train else _log(rng, 1, 4096), embd=rng.choice([256, 768, 1024, 1280, 1600]),
                    train=train)
    if kind == "attention":
        dim = rng.choice([64, 128])
        seq = _log(rng, 16, 4096)
        heads = rng.choice([4, 12, 16, 25, 32])
        # at most the tokens x keys x channels of the largest listed case, and 16 sequences
        most = max(1, (2 * 4096 * 4096 * 16 * 128) // (seq * seq * heads * dim))
        return dict(kind=kind, batch=rng.randint(1, min(16, most)), seq=seq, heads=heads, dim=dim, causal=rng.random() < 0.7,
                    packed=rng.random() < 0.5, train=rng.random() < 0.6)
    if kind == "llama_block":
        heads = rng.choice([4, 8, 16, 32])
        embd = heads * 128
        return dict(kind=kind, batch=rng.randint(1, 2), seq=_log(rng, 32, 1024), embd=embd, ffn=(embd * 43 // 16 + 63) // 64 * 64, heads=heads)
    if kind == "norm":
        embd = rng.choice([256, 768, 1024, 1280, 1600, 2048, 4096])
        return dict(kind=kind, rows=_log(rng, 16, 32 * 1024 * 1024 // embd), embd=embd, dtype=rng.choice(["bf16", "bf16", "fp32"]),
                    rms=rng.random() < 0.5)
    if kind == "head":
        return dict(kind=kind, rows=_log(rng, 64, 4096), embd=rng.choice([256, 768, 1024]), vocab=rng.choice([1000, 1024, 32000, 50257]))
    if kind == "bottleneck":
        planes, hw = rng.choice([(64, 56), (128, 28), (256, 14), (512, 7)])
        return dict(kind=kind, batch=_log(rng, 1, 64), hw=hw, planes=planes)
    if rng.random() < 0.5:
        return dict(kind="train_step", model="tiny", batch=rng.randint(1, 16), seq=rng.choice([32, 64, 100, 128]))
    return dict(kind="train_step", model="small", batch=rng.randint(1, 8), seq=rng.choice([128, 250, 512, 1024]))


# ---- preparation ----------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, device=DEV, generator=g) * std).to(dtype)


def _leaf(t):
    return t.requires_grad_(True)


def _gpt2(case, seed):
    cfg = getattr(GPT2Config, case["model"])(**NO_DROPOUT)
    torch.manual_seed(seed)
    with torch.device(DEV):
        return cfg, GPTForCausalLM(cfg)


def _mlp_inputs(case, seed):
    g, e = _gen(seed), case["embd"]
    f = 4 * e
    x = _randn(g, case["rows"], e)
    w1, b1 = _randn(g, f, e, std=0.02), _randn(g, f, std=0.02)
    w2, b2 = _randn(g, e, f, std=0.02), _randn(g, e, std=0.02)
    return x, w1, b1, w2, b2, _randn(g, case["rows"], e), _randn(g, case["rows"], e)


def _attention_inputs(case, seed):
    g = _gen(seed)
    b, s, h, d = case["batch"], case["seq"], case["heads"], case["dim"]
    if case["packed"]:
        return (_randn(g, b * s, 3 * h * d),), _randn(g, b * s, h * d)
    return tuple(_randn(g, b, s, h, d) for _ in range(3)), _randn(g, b, s, h, d)


def _llama(case, seed):
    cfg = LlamaConfig(hidden_size=case["embd"], intermediate_size=case["ffn"], num_layers=32, num_heads=case["heads"])
    torch.manual_seed(seed)
    with torch.device(DEV):
        blk = LlamaBlock(cfg).to(BF16)
    g = _gen(seed)
    rows = case["batch"] * case["seq"]
    return cfg, blk, _randn(g, rows, case["embd"]), _randn(g, rows, case["embd"])


def _norm_inputs(case, seed):
    g, e = _gen(seed), case["embd"]
    dt = BF16 if case["dtype"] == "bf16" else torch.float32
    x = _randn(g, case["rows"], e, std=2.0, dtype=dt)
    w = (1.0 + _randn(g, e, std=0.1, dtype=torch.float32)).to(dt)
    b = None if case["rms"] else _randn(g, e, std=0.1, dtype=dt)
    return x, w, b, _randn(g, case["rows"], e, dtype=dt)


def _head_inputs(case, seed):
    g, v = _gen(seed), case["vocab"]
    w = torch.zeros((v + 63) // 64 * 64, case["embd"], device=DEV, dtype=BF16)
    w[:v] = _randn(g, v, case["embd"], std=0.02)
    targets = torch.randint(0, v, (case["rows"],), device=DEV, generator=g)
    return _randn(g, case["rows"], case["embd"]), w, targets


def _bottleneck(case, seed):
    p = case["planes"]
    torch.manual_seed(seed)
    with torch.device(DEV):
        blk = BottleneckBlock(4 * p, p)
        for m in blk.modules():
            if isinstance(m, torch.nn.Conv2d):
                torch.nn.init.kaiming_normal_(m.weight, mode="fan_out", nonlinearity="relu")
            elif isinstance(m, torch.nn.BatchNorm2d):
                torch.nn.init.uniform_(m.weight, 0.5, 1.5)
                torch.nn.init.normal_(m.bias, 0.0, 0.1)
    g = _gen(seed)
    shape = (case["batch"], case["hw"], case["hw"], 4 * p)
    # a gradient as it comes back through the pooling at the end: most of it is shared by the pixels of a channel
    dy = _randn(g, shape[0], 1, 1, shape[3]) + _randn(g, *shape, std=0.25)
    return blk.train(), torch.relu(_randn(g, *shape)), dy


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "logits":
        cfg, model = _gpt2(case, seed)
        st["model"] = model.to(BF16).eval()
        st["ids"] = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"]), device=DEV, generator=_gen(seed))
    elif kind == "mlp":
        x, w1, b1, w2, b2, res, dy = _mlp_inputs(case, seed)
        st["args"], st["dy"] = (x, w1, b1, w2, b2, res), dy
        if case["train"]:
            for t in st["args"]:
                _leaf(t)
    elif kind == "attention":
        st["args"], st["dy"] = _attention_inputs(case, seed)
        if case["train"]:
            for t in st["args"]:
                _leaf(t)
    elif kind == "llama_block":
        _, st["block"], x, st["dy"] = _llama(case, seed)
        st["args"] = (_leaf(x), *st["block"].parameters())
    elif kind == "norm":
        x, w, b, st["dy"] = _norm_inputs(case, seed)
        st["args"] = tuple(_leaf(t) for t in (x, w, b) if t is not None)
    elif kind == "head":
        h, w, st["targets"] = _head_inputs(case, seed)
        st["args"] = (_leaf(h), _leaf(w))
    elif kind == "bottleneck":
        st["block"], x, st["dy"] = _bottleneck(case, seed)
        with torch.no_grad():
            for _ in range(STEPS_BEFORE):  # a block in the midst of training: its running statistics have settled
                st["block"].forward_nhwc(x)
        st["args"] = (_leaf(x), *st["block"].parameters())
    else:
        cfg, model = _gpt2(case, seed)
        st["trainer"] = CausalLMTrainer(model, batch_size=case["batch"], seq_len=case["seq"])
        data = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"] + 1), generator=torch.Generator().manual_seed(seed))
        st["ids"], st["targets"] = data[:, :-1].contiguous().pin_memory(), data[:, 1:].contiguous().pin_memory()
        for _ in range(3):  # two eager steps, then the one that captures the graph
            st["trainer"].step(st["ids"], st["targets"])
    return st


# ---- one pass -------------------------------------------------------------------------------------------------------
def _attend(case, args):
    if case["packed"]:
        return flash_attention_qkvpacked(args[0], case["batch"], case["seq"], case["heads"], case["dim"], causal=case["causal"])
    return flash_attention(*args, causal=case["causal"])


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "logits":
        with torch.no_grad():
            return st["model"](st["ids"])
    if kind in ("mlp", "attention"):
        forward = (lambda: mlp_gelu(*st["args"])) if kind == "mlp" else (lambda: _attend(case, st["args"]))
        if not case["train"]:
            with torch.no_grad():
                return forward()
        y = forward()
        return [y, *torch.autograd.grad(y, st["args"], st["dy"])]
    if kind == "llama_block":
        y = st["block"](st["args"][0], case["batch"], case["seq"])
        return [y, *torch.autograd.grad(y, st["args"], st["dy"])]
    if kind == "norm":
        y = rms_norm(*st["args"]) if case["rms"] else layer_norm(*st["args"])
        return [y, *torch.autograd.grad(y, st["args"], st["dy"])]
    if kind == "head":
        h, w = st["args"]
        loss = cross_entropy(linear(h, w), st["targets"], num_classes=case["vocab"], inplace_grad=True, root_scale=1.0)
        return [loss, *torch.autograd.grad(loss, st["args"])]
    if kind == "bottleneck":
        y = st["block"].forward_nhwc(st["args"][0])
        grads = torch.autograd.grad(y, st["args"], st["dy"])
        bns = (st["block"].bn1, st["block"].bn2, st["block"].bn3)
        return [y, *grads, *(t for bn in bns for t in (bn.running_mean, bn.running_var))]
    loss = st["trainer"].step(st["ids"], st["targets"])
    return [loss, st["trainer"].flat.master, st["trainer"].flat.lowp]


# ---- bytes and operations -------------------------------------------------------------------------------------------
def _gpt2_sizes(case):
    cfg = getattr(GPT2Config, case["model"])()
    e, layers, v = cfg.n_embd, cfg.n_layer, cfg.padded_vocab
    per_layer = 4 * e * e + 2 * e * cfg.inner
    small = layers * (9 * e + cfg.inner + 4 * e) + 2 * e + cfg.n_positions * e
    return cfg, layers * per_layer, v * e, small


def work(case):
    kind = case["kind"]
    if kind == "logits":
        cfg, mat, emb, small = _gpt2_sizes(case)
        t = case["batch"] * case["seq"]
        attn = 4 * t * case["seq"] * cfg.n_embd * cfg.n_layer / 2
        return dict(bytes=2 * (mat + emb + small) + 2 * t * cfg.vocab_size + 8 * t, flops=2 * t * (mat + emb) + attn)
    if kind == "mlp":
        r, e = case["rows"], case["embd"]
        w, flops = 8 * e * e, 16 * r * e * e
        if not case["train"]:
            return dict(bytes=2 * (w + 5 * e + 3 * r * e), flops=flops)
        # in: x, weights, residual, dy; out: y, dx and the weights' gradients (the residual's gradient is dy)
        return dict(bytes=2 * (2 * w + 10 * e + 5 * r * e), flops=3 * flops)
    if kind == "attention":
        n = case["batch"] * case["seq"] * case["heads"] * case["dim"]
        pairs = case["batch"] * case["heads"] * case["seq"] * case["seq"] * (0.5 if case["causal"] else 1.0)
        fwd = 4 * pairs * case["dim"]
        return dict(bytes=2 * n * (8 if case["train"] else 4), flops=fwd * (3.5 if case["train"] else 1.0))
    if kind == "llama_block":
        t, e, f = case["batch"] * case["seq"], case["embd"], case["ffn"]
        mat = 4 * e * e + 3 * e * f
        return dict(bytes=2 * (2 * mat + 4 * e + 4 * t * e), flops=6 * t * mat + 3.5 * 4 * t * case["seq"] * e / 2)
    if kind == "norm":
        n, size = case["rows"] * case["embd"], 2 if case["dtype"] == "bf16" else 4
        return dict(bytes=size * (4 * n + (2 if case["rms"] else 4) * case["embd"]), flops=14 * n)
    if kind == "head":
        r, e, v = case["rows"], case["embd"], case["vocab"]
        return dict(bytes=2 * (2 * r * e + 2 * v * e) + 8 * r, flops=6 * r * e * v)
    if kind == "bottleneck":
        p, px = case["planes"], case["batch"] * case["hw"] * case["hw"]
        mat = 17 * p * p
        # in: x, dy; out: y, dx in bf16; BatchNorm needs each convolution's whole output before its apply pass
        return dict(bytes=2 * 4 * px * 4 * p + 8 * mat, flops=6 * px * mat)
    cfg, mat, emb, small = _gpt2_sizes(case)
    t = case["batch"] * case["seq"]
    # AdamW: master, both moments read and written, the bf16 copy written and read once by the forward pass
    return dict(bytes=28 * (mat + emb + small) + 16 * t, flops=6 * t * (mat + emb) + 3.5 * 4 * t * case["seq"] * cfg.n_embd * cfg.n_layer / 2)


def tolerance(case):
    """About four times the largest relative error against :func:`exact` over the listed and 24 drawn cases: 2.5e-3 for the
    bf16 MLP and attention, 1.7e-3 for the bf16 norms and the head, 1.5e-7 for the fp32 norms, 9e-3 for whole forward
    passes. Two kinds are wider by their nature and get less than four times: the Llama block (3.3e-2 at 2048 tokens, where
    the fp32 rotary angles are largest) and the bottleneck (9e-2 in its gradients: an activation within a bf16 rounding of
    zero switches its ReLU). Two runs of the same training steps differ by 8e-4 (the order of the fp32 atomic sums)."""
    kind = case["kind"]
    if kind == "norm":
        return {"rel": 2e-6 if case["dtype"] == "fp32" else 7e-3}
    return {"rel": {"logits": 4e-2, "mlp": 1e-2, "attention": 1e-2, "llama_block": 5e-2, "head": 7e-3, "bottleneck": 0.2,
                    "train_step": 1e-2}[kind]}


# ---- 64-bit references ----------------------------------------------------------------------------------------------
def _gelu64(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _ln64(x, w, b, eps=1e-5):
    c = x - x.mean(-1, keepdim=True)
    y = c * torch.rsqrt(c.square().mean(-1, keepdim=True) + eps) * w
    return y if b is None else y + b


def _rms64(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _attention64(q, k, v, causal):
    """``[B, H, S, D]`` in, the same out."""
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if causal:
        n = q.shape[-2]
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=q.device).triu(1), float("-inf"))
    return torch.softmax(s, -1) @ v


def _attention_grads64(q, k, v, dy, causal, train):
    """One sequence and head group at a time, so that the scores of long sequences fit."""
    outs = [torch.empty_like(q) for _ in range(4 if train else 1)]
    step = max(1, 2 ** 27 // (q.shape[2] * q.shape[2]))
    for b in range(q.shape[0]):
        for h in range(0, q.shape[1], step):
            at = (slice(b, b + 1), slice(h, h + step))
            part = [t[at].detach().requires_grad_(train) for t in (q, k, v)]
            o = _attention64(*part, causal)
            outs[0][at] = o.detach()
            if train:
                for dst, g in zip(outs[1:], torch.autograd.grad(o, part, dy[at])):
                    dst[at] = g
    return outs


def _d(t):
    return t.detach().double()


def _rope64(x, base):
    s, d = x.shape[1], x.shape[-1]
    freq = base ** (-torch.arange(0, d, 2, device=x.device, dtype=torch.float64) / d)
    ang = torch.arange(s, device=x.device, dtype=torch.float64)[:, None] * freq
    c, n = ang.cos()[None, :, None], ang.sin()[None, :, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * c - b * n, a * n + b * c), -1).flatten(-2)


def _llama64(case, cfg, names, x):
    b, s, h, d = case["batch"], case["seq"], case["heads"], cfg.head_dim
    e = case["embd"]
    qkv = _rms64(x, names["input_norm.weight"], cfg.rms_eps) @ names["qkv.weight"].t()
    q, k, v = (qkv[:, i * e:(i + 1) * e].reshape(b, s, h, d) for i in range(3))
    q, k = _rope64(q, cfg.rope_theta), _rope64(k, cfg.rope_theta)
    ctx = _attention64(*(t.transpose(1, 2) for t in (q, k, v)), True).transpose(1, 2).reshape(b * s, e)
    x = x + ctx @ names["o.weight"].t()
    u = _rms64(x, names["post_attn_norm.weight"], cfg.rms_eps) @ names["gate_up.weight"].t()
    up, gate = u[:, :case["ffn"]], u[:, case["ffn"]:]
    return x + (up * gate * torch.sigmoid(gate)) @ names["down.weight"].t()


def _bottleneck64(names, x):
    y, stats = x.permute(0, 3, 1, 2), []
    for i in (1, 2, 3):
        y = torch.nn.functional.conv2d(y, names[f"conv{i}.weight"], padding=1 if i == 2 else 0)
        n = y.numel() / y.shape[1]
        mean, var = y.mean((0, 2, 3)), y.var((0, 2, 3), unbiased=False)
        old = 0.9 ** (STEPS_BEFORE + 1)
        stats += [(1 - old) * mean.detach(), old + (1 - old) * var.detach() * n / (n - 1)]
        y = (y - mean[:, None, None]) * torch.rsqrt(var[:, None, None] + 1e-5)
        y = y * names[f"bn{i}.weight"][:, None, None] + names[f"bn{i}.bias"][:, None, None]
        y = torch.relu(y) if i < 3 else torch.relu(y + x.permute(0, 3, 1, 2))
    return y.permute(0, 2, 3, 1), stats


def _block_grads64(module, x, dy, forward):
    """Output and gradients of ``forward(parameters by name, x)`` for the module's parameters in 64 bits."""
    names = {n: _d(p).requires_grad_(True) for n, p in module.named_parameters()}
    x = _d(x).requires_grad_(True)
    y = forward(names, x)
    y, more = y if isinstance(y, tuple) else (y, [])
    return [y.detach(), *torch.autograd.grad(y, (x, *names.values()), _d(dy)), *more]


def exact(case, seed):
    kind = case["kind"]
    if kind == "logits":
        cfg, model = _gpt2(case, seed)
        names = {n: _d(p.to(BF16)) for n, p in model.named_parameters()}
        b, s = case["batch"], case["seq"]
        ids = torch.randint(0, cfg.vocab_size, (b, s), device=DEV, generator=_gen(seed))
        x = names["transformer.wte"][ids].reshape(b * s, -1) + names["transformer.wpe"][:s].repeat(b, 1)
        e = cfg.n_embd
        for i in range(cfg.n_layer):
            w = {n.split(".", 3)[3]: p for n, p in names.items() if n.startswith(f"transformer.h.{i}.")}
            qkv = _ln64(x, w["ln_1.weight"], w["ln_1.bias"]) @ w["attn.c_attn.weight"].t() + w["attn.c_attn.bias"]
            q, k, v = (qkv[:, j * e:(j + 1) * e].reshape(b, s, cfg.n_head, -1).transpose(1, 2) for j in range(3))
            ctx = _attention64(q, k, v, True).transpose(1, 2).reshape(b * s, e)
            x = x + ctx @ w["attn.c_proj.weight"].t() + w["attn.c_proj.bias"]
            h = _gelu64(_ln64(x, w["ln_2.weight"], w["ln_2.bias"]) @ w["mlp.c_fc.weight"].t() + w["mlp.c_fc.bias"])
            x = x + h @ w["mlp.c_proj.weight"].t() + w["mlp.c_proj.bias"]
        h = _ln64(x, names["transformer.ln_f.weight"], names["transformer.ln_f.bias"])
        return (h @ names["transformer.wte"][: cfg.vocab_size].t()).view(b, s, -1)
    if kind == "mlp":
        *args, dy = _mlp_inputs(case, seed)
        x, w1, b1, w2, b2, res = args = [_d(t).requires_grad_(case["train"]) for t in args]
        y = _gelu64(x @ w1.t() + b1) @ w2.t() + b2 + res
        return [y.detach(), *torch.autograd.grad(y, args, _d(dy))] if case["train"] else y
    if kind == "attention":
        b, s, h, d = case["batch"], case["seq"], case["heads"], case["dim"]
        args, dy = _attention_inputs(case, seed)
        heads_first = lambda t: _d(t).reshape(b, s, h, d).transpose(1, 2)  # noqa: E731
        if case["packed"]:
            q, k, v = (heads_first(t) for t in args[0].split(h * d, 1))
        else:
            q, k, v = (heads_first(t) for t in args)
        outs = [t.transpose(1, 2) for t in _attention_grads64(q, k, v, heads_first(dy), case["causal"], case["train"])]
        if case["packed"]:
            outs = [t.reshape(b * s, h * d) for t in outs]
            outs = [outs[0], torch.cat(outs[1:], 1)] if case["train"] else outs
        return outs if case["train"] else outs[0]
    if kind == "llama_block":
        cfg, blk, x, dy = _llama(case, seed)
        return _block_grads64(blk, x, dy, lambda names, t: _llama64(case, cfg, names, t))
    if kind == "norm":
        x, w, b, dy = _norm_inputs(case, seed)
        args = [_d(t).requires_grad_(True) for t in (x, w, b) if t is not None]
        y = _rms64(*args) if case["rms"] else _ln64(*args)
        return [y.detach(), *torch.autograd.grad(y, args, _d(dy))]
    if kind == "head":
        h, w, targets = _head_inputs(case, seed)
        h, w = _d(h).requires_grad_(True), _d(w).requires_grad_(True)
        loss = torch.nn.functional.cross_entropy(h @ w[: case["vocab"]].t(), targets)
        return [loss.detach(), *torch.autograd.grad(loss, (h, w))]
    if kind == "bottleneck":
        blk, x, dy = _bottleneck(case, seed)
        return _block_grads64(blk, x, dy, _bottleneck64)
    return None  # several optimizer steps of a whole model
