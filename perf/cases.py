"""The single-GPU work that programs built on this package spend their time in, as measurable cases.

Each case is one pass of a layer, block, loss or optimizer step through the package's public modules and functions:
the parts of the ResNet-50 and GPT-2 training steps (forward and backward), of inference with the same layers, and of
the small MNIST-sized programs of ``examples/``.  ``listed()`` gives the named cases, ``draw(rng)`` more of the same
ranges, ``prepare`` the inputs and weights a program holds before the call, ``run`` the pass, ``exact`` the same
results in 64 bits from plain PyTorch.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from torchmpi_b200.models import to_bf16_mixed
from torchmpi_b200.models.gpt2 import Block, GPT2Config, LMLoss
from torchmpi_b200.models.resnet import Bottleneck, _bn
from torchmpi_b200.ops import attention, elementwise, gemm, layernorm, xent
from torchmpi_b200.ops.bn_relu import FusedBatchNormReLUMaxPool
from torchmpi_b200.ops.stem_conv import StemConv7x7

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
HEAD = 64


def listed():
    return [
        # the loss of the MNIST examples: their global batch of 336 on one GPU, ten classes, fp32 (latency counts)
        {"name": "mnist_loss", "kind": "loss", "rows": 336, "classes": 10, "dtype": "fp32"},
        # the classifier of ResNet-50 at the benchmark's batch of 256
        {"name": "classifier", "kind": "linear", "rows": 256, "inp": 2048, "out": 1000, "gelu": False},
        # the layer norms of GPT-2 medium at the benchmark's 8 x 1024 tokens
        {"name": "layernorm", "kind": "layernorm", "rows": 8192, "width": 1024, "dtype": "bf16"},
        # the up-projection of the GPT-2 medium MLP (GELU), 8 x 1024 tokens
        {"name": "mlp_up", "kind": "linear", "rows": 8192, "inp": 1024, "out": 4096, "gelu": True},
        # the attention output projection of GPT-2 medium for one sequence of 1024 tokens (a small per-GPU batch)
        {"name": "proj_one_sequence", "kind": "linear", "rows": 1024, "inp": 1024, "out": 1024, "gelu": False},
        # attention of GPT-2 medium in training, 8 sequences of 1024 tokens
        {"name": "attention_train", "kind": "attention", "batch": 8, "seq": 1024, "heads": 16, "train": True},
        # attention over the prompt of one request: forward only, twice the training context
        {"name": "attention_prefill", "kind": "attention", "batch": 1, "seq": 2048, "heads": 16, "train": False},
        # LM head (tied embedding, vocabulary of 50257) and next-token loss of GPT-2 medium, 8 x 1024 tokens
        {"name": "lm_head_loss", "kind": "head", "rows": 8192, "vocab": 50257, "width": 1024},
        # one whole transformer block of GPT-2 medium, forward and backward, 8 x 1024 tokens
        {"name": "gpt2_block", "kind": "block", "batch": 8, "seq": 1024, "heads": 16},
        # a residual block of the second ResNet-50 stage at the benchmark's batch of 256, forward and backward
        {"name": "bottleneck", "kind": "bottleneck", "batch": 256, "planes": 128, "size": 28, "first": False, "train": True},
        # the ResNet-50 stem (convolution, batch-norm, ReLU, max-pool) on 256 images of 224 x 224, forward and backward
        {"name": "stem", "kind": "stem", "batch": 256, "size": 224},
        # an SGD step on as many parameters as ResNet-50 has: bf16 weights, fp32 master weights and momentum
        {"name": "sgd_step", "kind": "update", "op": "sgd", "numel": 25557032, "dtype": "bf16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loss", "linear", "linear", "layernorm", "attention", "attention", "head", "block", "bottleneck",
                       "stem", "update"])
    if kind == "loss":
        return {"kind": kind, "rows": _log(rng, 16, 8192), "classes": _log(rng, 10, 1000), "dtype": rng.choice(["fp32", "bf16"])}
    if kind == "linear":
        # whole sequences, per-GPU image batches and, one time in four, an odd number of rows
        rows = _log(rng, 8, 8192)
        rows = rows if rng.random() < 0.25 else max(8, rows // 8 * 8)
        out = rng.choice([128, 384, 512, 768, 1000, 1024, 1536, 2048, 3072, 4096])
        inp = rng.choice([128, 256, 512, 768, 1024, 2048])
        return {"kind": kind, "rows": rows, "inp": inp, "out": out, "gelu": rng.random() < 0.5}
    if kind == "layernorm":
        return {"kind": kind, "rows": _log(rng, 1, 32768), "width": rng.choice([256, 512, 768, 1024]),
                "dtype": rng.choice(["bf16", "bf16", "fp16", "fp32"])}
    if kind == "attention":
        seq = _log(rng, 128, 2048)
        seq = seq if rng.random() < 0.25 else seq // 128 * 128
        heads = rng.choice([4, 8, 12, 16])
        batch = _log(rng, 1, max(1, min(16, 8 * 1024 * 1024 * 16 // (seq * seq * heads))))
        return {"kind": kind, "batch": batch, "seq": seq, "heads": heads, "train": rng.random() < 0.6}
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 256, 4096), "vocab": rng.choice([512, 5003, 32000, 50257]),
                "width": rng.choice([256, 512, 768, 1024])}
    if kind == "block":
        seq = 128 * _log(rng, 1, 8)
        return {"kind": kind, "batch": _log(rng, 1, 8192 // seq), "seq": seq, "heads": rng.choice([4, 8, 12, 16])}
    if kind == "bottleneck":
        planes, size = rng.choice([(64, 56), (128, 28), (256, 14), (512, 7)])
        first = rng.random() < 0.35
        return {"kind": kind, "batch": _log(rng, 8, 96 if first or planes == 64 else 256), "planes": planes, "size": size,
                "first": first, "train": rng.random() < 0.7}
    if kind == "stem":
        return {"kind": kind, "batch": _log(rng, 8, 256), "size": rng.choice([96, 128, 160, 192, 224])}
    return {"kind": kind, "op": rng.choice(["sgd", "sgd", "easgd", "downpour"]), "numel": _log(rng, 1000, 25_000_000) // 8 * 8,
            "dtype": rng.choice(["bf16", "fp32"])}


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(shape, generator=g, device=DEV) * scale).to(dtype)


def _images(g, n, c, h, w, scale=1.0):
    return _randn(g, (n, h, w, c), scale=scale).permute(0, 3, 1, 2)          # channels-last


def _trained_bn(module, g):
    """Scales and shifts as a network under training has them (not the initial ones and zeros)."""
    for m in module.modules():
        if isinstance(m, torch.nn.BatchNorm2d):
            with torch.no_grad():
                m.weight.copy_(torch.rand(m.weight.shape, generator=g, device=DEV) + 0.5)
                m.bias.copy_(torch.randn(m.bias.shape, generator=g, device=DEV) * 0.1)
                m.running_var.fill_(1.5)


def _geometry(case):
    """(input planes, input size, stride) of a bottleneck: the first one of a stage widens and halves the image."""
    if not case["first"]:
        return case["planes"] * 4, case["size"], 1
    stride = 1 if case["planes"] == 64 else 2
    return (64 if case["planes"] == 64 else case["planes"] * 2), case["size"] * stride, stride


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    s = {"case": case}
    if kind == "loss":
        s["logits"] = _randn(g, (case["rows"], case["classes"]), DTYPES[case["dtype"]], 2.0).requires_grad_(True)
        s["labels"] = torch.randint(0, case["classes"], (case["rows"],), generator=g, device=DEV)
        s["criterion"] = xent.CrossEntropyLoss()
    elif kind == "linear":
        with torch.device(DEV):
            m = gemm.Linear(case["inp"], case["out"], gelu=case["gelu"], dtype=torch.bfloat16)
        with torch.no_grad():
            m.weight.copy_(_randn(g, m.weight.shape, scale=case["inp"] ** -0.5))
            m.bias.copy_(_randn(g, m.bias.shape, scale=0.1))
        s["module"] = m
        s["x"] = _randn(g, (case["rows"], case["inp"])).requires_grad_(True)
        s["dy"] = _randn(g, (case["rows"], case["out"]))
    elif kind == "layernorm":
        dt = DTYPES[case["dtype"]]
        m = layernorm.LayerNorm(case["width"], device=DEV, dtype=dt)
        with torch.no_grad():
            m.weight.copy_(1.0 + _randn(g, m.weight.shape, dt, 0.1))
            m.bias.copy_(_randn(g, m.bias.shape, dt, 0.1))
        s["module"] = m
        s["x"] = (_randn(g, (case["rows"], case["width"]), dt, 1.5) + 0.25).requires_grad_(True)
        s["dy"] = _randn(g, (case["rows"], case["width"]), dt)
    elif kind == "attention":
        shape = (case["batch"], case["seq"], case["heads"] * HEAD)
        s["qkv"] = _randn(g, shape[:2] + (3 * shape[2],)).requires_grad_(case["train"])
        s["dy"] = _randn(g, shape) if case["train"] else None
    elif kind == "head":
        s["x"] = _randn(g, (case["rows"], case["width"])).requires_grad_(True)
        s["w"] = _randn(g, (case["vocab"], case["width"]), scale=0.02).requires_grad_(True)
        s["labels"] = torch.randint(0, case["vocab"], (case["rows"],), generator=g, device=DEV)
        s["criterion"] = LMLoss(unit_grad=True)
    elif kind == "block":
        width = case["heads"] * HEAD
        with torch.device(DEV):
            m = Block(GPT2Config(n_head=case["heads"], n_embd=width, tc_linear=True)).to(torch.bfloat16)
        with torch.no_grad():
            for n, p in m.named_parameters():
                if p.dim() == 2:
                    p.copy_(_randn(g, p.shape, scale=p.shape[1] ** -0.5))
                else:                        # scales of the layer norms around one, every bias around zero
                    p.copy_(_randn(g, p.shape, scale=0.05) + (1.0 if n.endswith("weight") else 0.0))
        s["module"] = m
        s["x"] = _randn(g, (case["batch"], case["seq"], width)).requires_grad_(True)
        s["dy"] = _randn(g, (case["batch"], case["seq"], width))
    elif kind == "bottleneck":
        inp, size, stride = _geometry(case)
        down = None
        with torch.device(DEV):
            if case["first"]:
                down = torch.nn.Sequential(torch.nn.Conv2d(inp, case["planes"] * 4, 1, stride=stride, bias=False),
                                           _bn(case["planes"] * 4, True, relu=False))
            m = Bottleneck(inp, case["planes"], stride, down, fused_bn=True)
        m = to_bf16_mixed(m).to(memory_format=torch.channels_last)
        with torch.no_grad():
            for p in m.parameters():
                if p.dim() == 4:
                    p.copy_(_randn(g, p.shape, scale=(2.0 / (p.shape[0] * p.shape[2] * p.shape[3])) ** 0.5))
        _trained_bn(m, g)
        s["module"] = m.train(case["train"])
        s["x"] = _images(g, case["batch"], inp, size, size).relu_().requires_grad_(case["train"])
        s["dy"] = _images(g, case["batch"], case["planes"] * 4, case["size"], case["size"]) if case["train"] else None
    elif kind == "stem":
        with torch.device(DEV):
            m = torch.nn.Sequential(StemConv7x7(64), FusedBatchNormReLUMaxPool(64))
        m = to_bf16_mixed(m).to(memory_format=torch.channels_last)
        with torch.no_grad():
            m[0].weight.copy_(_randn(g, m[0].weight.shape, scale=(2.0 / (64 * 49)) ** 0.5))
        _trained_bn(m, g)
        s["module"] = m.train()
        s["x"] = _images(g, case["batch"], 3, case["size"], case["size"])
        out = case["size"] // 4
        s["dy"] = _images(g, case["batch"], 64, out, out)
    else:
        n, dt = case["numel"], DTYPES[case["dtype"]]
        if case["op"] == "sgd":
            master = torch.randn(n, generator=g, device=DEV) * 0.05
            s["weight"] = master.to(dt)
            s["master"] = master if dt != torch.float32 else None
            s["momentum"] = torch.randn(n, generator=g, device=DEV) * 1e-3
            s["grad"] = _randn(g, (n,), dt, 1e-3)
        elif case["op"] == "easgd":
            s["local"], s["center"] = _randn(g, (n,), dt, 0.05), _randn(g, (n,), dt, 0.05)
            s["delta"] = torch.empty_like(s["local"])
        else:
            s["accum"], s["grad"] = _randn(g, (n,), dt, 1e-3), _randn(g, (n,), dt, 1e-3)
    return s


def _train(module, x, dy):
    """One forward and backward with fresh gradients; the output and every gradient."""
    module.zero_grad(set_to_none=True)
    x.grad = None
    y = module(x)
    y.backward(dy)
    return {"y": y.detach(), "dx": x.grad, "params": {n: p.grad for n, p in module.named_parameters()}}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loss":
        state["logits"].grad = None
        loss = state["criterion"](state["logits"], state["labels"])
        loss.backward()
        return {"loss": loss.detach(), "dx": state["logits"].grad}
    if kind in ("linear", "layernorm", "block"):
        return _train(state["module"], state["x"], state["dy"])
    if kind == "attention":
        if not case["train"]:
            with torch.no_grad():
                return attention.causal_attention(state["qkv"], case["heads"])
        state["qkv"].grad = None
        y = attention.causal_attention(state["qkv"], case["heads"])
        y.backward(state["dy"])
        return {"y": y.detach(), "dx": state["qkv"].grad}
    if kind == "head":
        state["x"].grad = state["w"].grad = None
        logits = gemm.wide_head(state["x"], state["w"])
        loss = state["criterion"](logits, state["labels"])
        loss.backward()
        return {"logits": logits.detach(), "loss": loss.detach(), "dx": state["x"].grad, "dw": state["w"].grad}
    if kind == "bottleneck":
        if not case["train"]:
            with torch.no_grad():
                return state["module"](state["x"])
        return _train(state["module"], state["x"], state["dy"])
    if kind == "stem":
        state["module"].zero_grad(set_to_none=True)
        y = state["module"](state["x"])
        y.backward(state["dy"])
        return {"y": y.detach(), "params": {n: p.grad for n, p in state["module"].named_parameters()}}
    if case["op"] == "sgd":
        elementwise.sgd_momentum_(state["weight"], state["grad"], lr=0.1, momentum=0.9, weight_decay=1e-4,
                                  master=state["master"], momentum_buf=state["momentum"])
        return {"weight": state["weight"], "master": state["master"], "momentum": state["momentum"]}
    if case["op"] == "easgd":
        elementwise.easgd_elastic(state["local"], state["center"], state["delta"], 0.225)
        return {"local": state["local"], "delta": state["delta"]}
    elementwise.downpour_accum(state["accum"], state["grad"], scale=0.5)
    return state["accum"]


def work(case):
    kind = case["kind"]
    if kind == "loss":
        n = case["rows"] * case["classes"]
        return {"bytes": 2 * n * SIZE[case["dtype"]] + 8 * case["rows"] + 4, "flops": 8 * n}
    if kind == "linear":
        r, i, o = case["rows"], case["inp"], case["out"]
        # x, dy, w and bias read; y, dx, dw and dbias written
        return {"bytes": 2 * (2 * r * i + 2 * r * o + 2 * i * o + 2 * o), "flops": 6.0 * r * i * o}
    if kind == "layernorm":
        n = case["rows"] * case["width"]
        return {"bytes": (4 * n + 4 * case["width"]) * SIZE[case["dtype"]], "flops": 20 * n}
    if kind == "attention":
        n = case["batch"] * case["seq"] * case["heads"] * HEAD
        products = 2.0 * n * (case["seq"] + 1) / 2                  # one causal product
        return ({"bytes": 2 * (8 * n), "flops": 7 * products} if case["train"]      # qkv, dy read; y, dqkv written
                else {"bytes": 2 * (4 * n), "flops": 2 * products})
    if kind == "head":
        r, v, d = case["rows"], case["vocab"], case["width"]
        return {"bytes": 2 * (2 * r * d + 2 * v * d + r * v) + 8 * r, "flops": 6.0 * r * v * d}
    if kind == "block":
        t, d = case["batch"] * case["seq"], case["heads"] * HEAD
        return {"bytes": 2 * (4 * t * d + 2 * 12 * d * d),
                "flops": 6.0 * t * 12 * d * d + 7 * 2.0 * t * d * (case["seq"] + 1) / 2}
    if kind == "bottleneck":
        inp, size, stride = _geometry(case)
        n, p, o = case["batch"], case["planes"], case["size"]
        x, y = n * inp * size * size, n * 4 * p * o * o
        weights = inp * p + 9 * p * p + 4 * p * p + (inp * 4 * p if case["first"] else 0)
        macs = n * (inp * p * size * size + 9 * p * p * o * o + 4 * p * p * o * o + (inp * 4 * p * o * o if case["first"] else 0))
        if not case["train"]:
            return {"bytes": 2 * (x + y + weights), "flops": 2.0 * macs}
        return {"bytes": 2 * (2 * x + 2 * y + 2 * weights), "flops": 6.0 * macs}
    if kind == "stem":
        n, h = case["batch"], case["size"]
        out = n * 64 * (h // 4) ** 2
        return {"bytes": 2 * (n * 3 * h * h + 2 * out), "flops": 4.0 * n * 64 * 147 * (h // 2) ** 2}
    n, e = case["numel"], SIZE[case["dtype"]]
    if case["op"] == "sgd":
        return {"bytes": n * (4 + 4 + 4 + 4 + 2 + 2 if case["dtype"] == "bf16" else 4 * 5), "flops": 6 * n}
    return {"bytes": n * e * (4 if case["op"] == "easgd" else 3), "flops": 3 * n}


def tolerance(case):
    """Relative errors of another implementation that holds the same values in the same types."""
    kind = case["kind"]
    wide = case.get("dtype") == "fp32"
    if kind in ("loss", "layernorm", "update") and wide:
        return {"rel": 2e-5, "max": 1e-3}
    if kind == "update":
        return {"rel": 4e-3, "max": 2e-2}
    if kind in ("loss", "layernorm"):
        return {"rel": 8e-3, "max": 8e-2}
    if kind == "attention":
        return {"rel": 1e-2, "max": 2e-1}
    if kind in ("linear", "head"):
        return {"rel": 1e-2, "max": 1e-1}
    return {"rel": 3e-2, "max": 9e-1}       # several layers in 16 bits; a ReLU mask or a pooled maximum may flip


def _leaf(t):
    return t.detach().double().requires_grad_(True)


def _attention64(qkv, heads):
    B, T, C3 = qkv.shape
    q, k, v = (t.reshape(B, T, heads, HEAD).transpose(1, 2) for t in qkv.split(C3 // 3, dim=2))
    mask = torch.ones(T, T, dtype=torch.bool, device=qkv.device).triu(1)
    out = []
    for b in range(B):                       # one sequence at a time: the score matrix stays small
        s = (q[b] @ k[b].transpose(1, 2)) * HEAD ** -0.5
        out.append(torch.softmax(s.masked_fill(mask, -math.inf), -1) @ v[b])
    return torch.stack(out).transpose(1, 2).reshape(B, T, C3 // 3)


def _conv64(x, w, stride, pad):
    """A convolution in 64 bits as matrix products over chunks of images (the library has no fast one)."""
    if w.shape[2] == 1 and pad == 0:
        x = x[:, :, ::stride, ::stride]
        return torch.einsum("nchw,oc->nohw", x, w[:, :, 0, 0])
    n, _, h, wd = x.shape
    oh, ow = (h + 2 * pad - w.shape[2]) // stride + 1, (wd + 2 * pad - w.shape[3]) // stride + 1
    cols = [F.unfold(c, w.shape[2], padding=pad, stride=stride) for c in x.split(16)]
    return torch.cat([(w.reshape(w.shape[0], -1) @ c) for c in cols]).reshape(n, w.shape[0], oh, ow)


def _bn64(x, p, name, bn, train):
    gamma, beta = p[name + ".weight"][:, None, None], p[name + ".bias"][:, None, None]
    if train:
        mean, var = x.mean((0, 2, 3), keepdim=True), x.var((0, 2, 3), unbiased=False, keepdim=True)
    else:
        mean, var = bn.running_mean.double()[:, None, None], bn.running_var.double()[:, None, None]
    return (x - mean) * torch.rsqrt(var + bn.eps) * gamma + beta


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "loss":
        x = _leaf(s["logits"])
        loss = F.cross_entropy(x, s["labels"])
        loss.backward()
        return {"loss": loss.detach(), "dx": x.grad}
    if kind == "update":
        if case["op"] == "sgd":
            master = s["master"] if s["master"] is not None else s["weight"]
            w, m = master.double(), s["momentum"].double()
            m = 0.9 * m + (s["grad"].double() + 1e-4 * w)
            w = w - 0.1 * m
            return {"weight": w, "master": w if s["master"] is not None else None, "momentum": m}
        if case["op"] == "easgd":
            d = s["center"].double() - s["local"].double()
            return {"local": s["local"].double() + 0.225 * d, "delta": -0.225 * d}
        return s["accum"].double() + 0.5 * s["grad"].double()
    if kind == "attention":
        x = _leaf(s["qkv"])
        if not case["train"]:
            with torch.no_grad():
                return _attention64(x, case["heads"])
        y = _attention64(x, case["heads"])
        y.backward(s["dy"].double())
        return {"y": y.detach(), "dx": x.grad}
    if kind == "head":
        x, w = _leaf(s["x"]), _leaf(s["w"])
        logits = x @ w.t()
        loss = F.cross_entropy(logits, s["labels"])
        loss.backward()
        return {"logits": logits.detach(), "loss": loss.detach(), "dx": x.grad, "dw": w.grad}
    module = s["module"]
    x, p = _leaf(s["x"]), {n: _leaf(v) for n, v in module.named_parameters()}
    if kind == "linear":
        y = F.linear(x, p["weight"], p["bias"])
        y = F.gelu(y) if case["gelu"] else y
    elif kind == "layernorm":
        y = F.layer_norm(x, (case["width"],), p["weight"], p["bias"], module.eps)
    elif kind == "block":
        width = x.shape[-1]
        norm = lambda t, n: F.layer_norm(t, (width,), p[n + ".weight"], p[n + ".bias"], module.ln1.eps)
        lin = lambda t, n: F.linear(t, p[n + ".weight"], p[n + ".bias"])
        a = x + lin(_attention64(lin(norm(x, "ln1"), "qkv"), case["heads"]), "proj")
        y = a + lin(F.gelu(lin(norm(a, "ln2"), "fc")), "out")
    elif kind == "bottleneck":
        stride, train = _geometry(case)[2], case["train"]
        conv = lambda t, n, st, pad: _conv64(t, p[n + ".weight"], st, pad)
        with torch.set_grad_enabled(train):
            identity = x
            if case["first"]:
                identity = _bn64(conv(x, "downsample.0", stride, 0), p, "downsample.1", module.downsample[1], train)
            out = torch.relu(_bn64(conv(x, "conv1", 1, 0), p, "bn1", module.bn1, train))
            out = torch.relu(_bn64(conv(out, "conv2", stride, 1), p, "bn2", module.bn2, train))
            y = torch.relu(_bn64(conv(out, "conv3", 1, 0), p, "bn3", module.bn3, train) + identity)
        if not train:
            return y
    else:
        z = _conv64(x.detach(), p["0.weight"], 2, 3)
        y = F.max_pool2d(torch.relu(_bn64(z, p, "1", module[1], True)), 3, 2, 1)
    y.backward(s["dy"].double())
    out = {"y": y.detach(), "params": {n: v.grad for n, v in p.items()}}
    return out if kind == "stem" else {**out, "dx": x.grad}
