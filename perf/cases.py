"""The work that training and evaluation programs have this framework do on one GPU, as timed cases.

``listed()`` are the standing cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` builds
what a program holds before the call, ``run`` is one pass through the public entry points, ``work`` the bytes
and operations the pass cannot do without, ``exact`` the same outputs in 64 bits by plain PyTorch.

Every number in a case is a size of the path: ``tokens`` rows of activations, ``d`` the model width, ``heads``
attention heads of 128 features, ``vocab`` the unpadded vocabulary.  16-bit data is bf16.
"""
from __future__ import annotations

import math
import random

import torch

D_HEAD = 128
VOCAB_PAD = 2048


# ----------------------------------------------------------------------------------------------
# cases
# ----------------------------------------------------------------------------------------------
def listed():
    return [
        # a projection of a small model (width 512) on one short batch: launches and latency count
        {"name": "linear_small", "kind": "linear", "flow": "os", "tokens": 512, "d_in": 512, "d_out": 1536},
        # a left-stationary layer (second MLP product) with extents that fill no tile evenly
        {"name": "linear_ragged", "kind": "linear", "flow": "ls", "tokens": 1992, "d_in": 4104, "d_out": 1032},
        # first MLP product of a 6.7B-parameter decoder, micro-batch of 4 x 2048 tokens
        {"name": "linear_large", "kind": "linear", "flow": "os", "tokens": 8192, "d_in": 4096, "d_out": 16384},
        # attention of the same decoder in a training step: forward and backward, causal
        {"name": "attention_train", "kind": "attention", "batch": 4, "seq": 2048, "heads": 32, "causal": True,
         "train": True},
        # bidirectional attention of the encoder-style block, odd head count, short sequence, training
        {"name": "attention_full", "kind": "attention", "batch": 3, "seq": 640, "heads": 5, "causal": False,
         "train": True},
        # scoring a long document: forward only
        {"name": "attention_long", "kind": "attention", "batch": 1, "seq": 8192, "heads": 16, "causal": True,
         "train": False},
        # pre-attention LayerNorm with the fused residual add and affine parameters, training
        {"name": "layernorm_train", "kind": "layernorm", "tokens": 32768, "d": 4096, "affine": True,
         "residual": True, "train": True},
        # LayerNorm of the plain block (no affine, no residual) at a width that fills no vector evenly
        {"name": "layernorm_odd", "kind": "layernorm", "tokens": 4099, "d": 1544, "affine": False,
         "residual": False, "train": True},
        # LM head, softmax cross-entropy and their gradients over a 50k vocabulary
        {"name": "head_loss", "kind": "head_loss", "tokens": 4096, "d": 1024, "vocab": 50257},
        # optimizer step with global-norm clipping over the flat buffers of a 200M-parameter model
        {"name": "adamw", "kind": "adamw", "n_sharded": 134217728 + 384, "n_rep": 53504000},
        # one decoder block of the 6.7B-parameter model, forward and backward of a micro-batch
        {"name": "gpt_block", "kind": "gpt_block", "batch": 4, "seq": 2048, "d": 4096, "heads": 32, "ffn": 16384},
        # a whole small model, one micro-batch: embedding to loss and back to every gradient
        {"name": "gpt_small", "kind": "gpt_model", "batch": 2, "seq": 256, "layers": 2, "d": 512, "heads": 4,
         "ffn": 2048, "vocab": 1000},
    ]


def _log(rng: random.Random, lo: int, hi: int, step: int = 1) -> int:
    """A multiple of ``step`` in [lo, hi], spread evenly over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng: random.Random):
    kind = rng.choice(["linear", "linear", "attention", "attention", "attention", "layernorm", "layernorm",
                       "head_loss", "adamw", "gpt_block", "gpt_model"])
    if kind == "linear":
        # tokens take any value on the 'os' layer; 16-byte rows ask for multiples of 8 features
        return {"kind": kind, "flow": rng.choice(["os", "ls"]), "tokens": _log(rng, 128, 8192, 8),
                "d_in": _log(rng, 256, 4096, 8), "d_out": _log(rng, 256, 16384, 8)}
    if kind == "attention":
        seq = _log(rng, 128, 8192, 128)
        heads = _log(rng, 1, 32)
        most = max(1, min(8, 4 * 2048 * 2048 * 32 // (seq * seq * heads)))
        return {"kind": kind, "batch": rng.randint(1, most), "seq": seq, "heads": heads,
                "causal": rng.random() < 0.6, "train": rng.random() < 0.6}
    if kind == "layernorm":
        d = _log(rng, 256, 8192, 8)
        return {"kind": kind, "tokens": _log(rng, 128, min(32768, 32768 * 4096 // d)), "d": d,
                "affine": rng.random() < 0.6, "residual": rng.random() < 0.6, "train": rng.random() < 0.7}
    if kind == "head_loss":
        return {"kind": kind, "tokens": _log(rng, 128, 4096, 8), "d": _log(rng, 256, 1024, 64),
                "vocab": _log(rng, 1000, 50257)}
    if kind == "adamw":
        return {"kind": kind, "n_sharded": _log(rng, 100000, 134217728, 128), "n_rep": _log(rng, 1024, 50000000, 128)}
    if kind == "gpt_block":
        heads = rng.randint(2, 32)
        return {"kind": kind, "batch": rng.randint(1, 4), "seq": rng.choice([128, 256, 640, 1024, 2048]),
                "d": heads * D_HEAD, "heads": heads, "ffn": heads * D_HEAD * 4}
    heads = rng.randint(1, 8)
    return {"kind": kind, "batch": rng.randint(1, 4), "seq": rng.choice([128, 256, 384, 512]),
            "layers": rng.randint(1, 4), "d": heads * D_HEAD, "heads": heads, "ffn": heads * D_HEAD * 4,
            "vocab": rng.randint(500, 8000)}


# ----------------------------------------------------------------------------------------------
# inputs, made from the seed alone
# ----------------------------------------------------------------------------------------------
class _Source:
    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
        return torch.empty(shape, device="cuda", dtype=dtype).normal_(mean, std, generator=self.g)

    def ids(self, n, high):
        return torch.randint(0, high, (n,), device="cuda", generator=self.g)


def _padded(vocab: int) -> int:
    return -(-vocab // VOCAB_PAD) * VOCAB_PAD


def _block_shapes(d: int, ffn: int):
    """Parameters of a decoder block in the order the framework lists them; ff2 is stored [out, in]."""
    return [("ln1.gamma", (d,)), ("ln1.bias", (d,)), ("in_proj", (d, 3 * d)), ("out_proj", (d, d)),
            ("ln2.gamma", (d,)), ("ln2.bias", (d,)), ("ff1", (d, ffn)), ("ff2", (d, ffn))]


def _model_shapes(case):
    d, vp = case["d"], _padded(case["vocab"])
    out = [("tok", (vp, d)), ("pos", (case["seq"], d))]
    for i in range(case["layers"]):
        out += [(f"{i}.{n}", s) for n, s in _block_shapes(d, case["ffn"])]
    return out + [("ln_f.gamma", (d,)), ("ln_f.bias", (d,)), ("head", (d, vp))]


def _weights(src: _Source, shapes):
    """Values that a trained model holds: weights of std 0.02, LayerNorm scales near one."""
    out = {}
    for name, s in shapes:
        if name.endswith("gamma"):
            out[name] = src.normal(*s, mean=1.0, std=0.1)
        elif name.endswith("bias"):
            out[name] = src.normal(*s, std=0.1)
        else:
            out[name] = src.normal(*s, std=0.02)
    return out


def _inputs(case, seed):
    src, k = _Source(seed), case["kind"]
    if k == "linear":
        t, i, o = case["tokens"], case["d_in"], case["d_out"]
        return {"x": src.normal(t, i), "dy": src.normal(t, o, std=0.01),
                "w": src.normal(*((o, i) if case["flow"] == "ls" else (i, o)), std=0.02)}
    if k == "attention":
        t, h = case["batch"] * case["seq"], case["heads"]
        return {"qkv": src.normal(t, h * 3 * D_HEAD), "dy": src.normal(t, h * D_HEAD, std=0.01)}
    if k == "layernorm":
        t, d = case["tokens"], case["d"]
        return {"x": src.normal(t, d, std=2.0, mean=0.1), "res": src.normal(t, d), "dy": src.normal(t, d, std=0.01),
                "dres": src.normal(t, d, std=0.01), "gamma": src.normal(d, mean=1.0, std=0.1),
                "bias": src.normal(d, std=0.1)}
    if k == "head_loss":
        t, d = case["tokens"], case["d"]
        return {"x": src.normal(t, d), "w": src.normal(d, _padded(case["vocab"]), std=0.05),
                "targets": src.ids(t, case["vocab"])}
    if k == "adamw":
        out = {}
        for n in ("n_sharded", "n_rep"):
            out[n] = (src.normal(case[n], std=0.02), src.normal(case[n], std=2e-4, dtype=torch.float32),
                      src.normal(case[n], std=1e-4, dtype=torch.float32),
                      src.normal(case[n], std=1e-4, dtype=torch.float32).square_())
        return out
    if k == "gpt_block":
        t, d = case["batch"] * case["seq"], case["d"]
        return {"x": src.normal(t, d), "delta": src.normal(t, d, std=0.5), "dh": src.normal(t, d, std=0.01),
                "dm": src.normal(t, d, std=0.01), "w": _weights(src, _block_shapes(d, case["ffn"]))}
    t = case["batch"] * case["seq"]
    return {"tokens": src.ids(t, case["vocab"]), "targets": src.ids(t, case["vocab"]),
            "w": _weights(src, _model_shapes(case))}


# ----------------------------------------------------------------------------------------------
# the framework's side
# ----------------------------------------------------------------------------------------------
KEY = (0, 0)


def _mesh():
    from meshslice_b200.parallel.engine import LocalGemmEngine
    from meshslice_b200.parallel.mesh import EmuMesh
    mesh = EmuMesh(1, 1)
    LocalGemmEngine(mesh)
    return mesh


def _gpt_config(case):
    from meshslice_b200.models.gpt import GPTConfig
    return GPTConfig(n_layers=case.get("layers", 1), d_model=case["d"], n_heads=case["heads"], ffn=case["ffn"],
                     vocab=case.get("vocab", 50257), seq=case["seq"], ksplits=(1, 1, 1, 1), vocab_pad=VOCAB_PAD)


def prepare(case, seed):
    from meshslice_b200.models.gpt import GPTBlock
    from meshslice_b200.models.sharded_layers import ShardedAttention, ShardedFFLayer, ShardedLayerNorm
    from meshslice_b200.optim import AdamW, FlatGroup
    from meshslice_b200.parallel.mesh import ShardedTensor
    from meshslice_b200.trainer import TrainConfig, Trainer

    k, v, dev = case["kind"], _inputs(case, seed), torch.device("cuda", torch.cuda.current_device())
    s = {"case": case}
    if k == "adamw":
        groups = []
        for n, label in (("n_sharded", "sharded"), ("n_rep", "row_replicated")):
            param, grad, m, var = v[n]
            g = FlatGroup(param, grad, label)
            g.m.copy_(m)
            g.v.copy_(var)
            groups.append(g)
        s["opt"] = AdamW(groups, lr=1e-4, weight_decay=0.01)
        s["opt"].step_count = 99
        return s
    if k == "gpt_model":
        tr = Trainer(_gpt_config(case), TrainConfig(global_batch=case["batch"], micro_batch=case["batch"]),
                     mesh_shape=(1, 1), device=dev)
        for (_, p, _, _), w in zip(tr.model.parameters(), v["w"].values()):
            p.shards[KEY].copy_(w)
        s["trainer"] = tr
        s["tokens"], s["targets"] = (ShardedTensor(tr.mesh, {KEY: v[n]}) for n in ("tokens", "targets"))
        return s
    mesh = _mesh()
    s.update({n: ShardedTensor(mesh, {KEY: t}) for n, t in v.items() if isinstance(t, torch.Tensor)})
    if k in ("linear", "head_loss"):
        flow = case.get("flow", "os")
        d_in, d_out = v["w"].shape[::-1] if flow == "ls" else v["w"].shape
        s["layer"] = ShardedFFLayer(mesh, "meshslice", flow, 1, d_in, d_out, device=dev)
        s["layer"].weight.shards[KEY].copy_(v["w"])
    elif k == "attention":
        s["layer"] = ShardedAttention(mesh, case["heads"], case["seq"], causal=case["causal"])
    elif k == "layernorm":
        s["layer"] = ShardedLayerNorm(mesh, case["d"], affine=case["affine"], eps=1e-5, device=dev)
        s["layer"].gamma.shards[KEY].copy_(v["gamma"])
        s["layer"].bias.shards[KEY].copy_(v["bias"])
    else:
        s["block"] = GPTBlock(mesh, _gpt_config(case), 0, dev, None, None, None)
        params = [p for l in s["block"].layers() for _, p, _, _ in l.parameters()]
        for p, w in zip(params, v["w"].values()):
            p.shards[KEY].copy_(w)
    return s


def run(s):
    from meshslice_b200.ops import functional as F
    case = s["case"]
    k = case["kind"]
    if k == "linear":
        layer = s["layer"]
        layer.zero_grad()
        y = layer.forward(s["x"])
        dx = layer.backward(s["dy"])
        return {"y": y.shards[KEY], "dx": dx.shards[KEY], "dw": layer.grad.shards[KEY]}
    if k == "attention":
        y = s["layer"].forward(s["qkv"])
        if not case["train"]:
            return {"y": y.shards[KEY]}
        return {"y": y.shards[KEY], "dqkv": s["layer"].backward(s["dy"]).shards[KEY]}
    if k == "layernorm":
        layer = s["layer"]
        res = s["res"] if case["residual"] else None
        y = layer.forward(s["x"], res)
        out = {"y": y.shards[KEY]}
        if case["residual"]:
            out["h"] = layer.h.shards[KEY]
        if case["train"]:
            layer.zero_grad()
            out["dx"] = layer.backward(s["dy"], s["dres"] if case["residual"] else None).shards[KEY]
            if case["affine"]:
                out["dgamma"], out["dbias"] = layer.dgamma.shards[KEY], layer.dbias.shards[KEY]
        return out
    if k == "head_loss":
        layer, t = s["layer"], s["targets"].shards[KEY]
        layer.zero_grad()
        logits = layer.forward(s["x"])
        l = logits.shards[KEY]
        mx, se, target = F.ce_partial(l, t, 0, case["vocab"])
        loss = torch.log(se) + mx - target
        F.ce_grad_(l, t, 0, case["vocab"], mx, se, 1.0 / case["tokens"])
        dx = layer.backward(logits)
        return {"loss": loss, "dlogits": l, "dx": dx.shards[KEY], "dw": layer.grad.shards[KEY]}
    if k == "adamw":
        s["opt"].step()
        return [{"param": g.param, "master": g.master, "m": g.m, "v": g.v} for g in s["opt"].groups]
    if k == "gpt_block":
        b = s["block"]
        for layer in b.layers():
            layer.zero_grad()
        h, m = b.forward(s["x"], s["delta"])
        dx, _ = b.backward(s["dh"], s["dm"])
        grads = [g.shards[KEY] for layer in b.layers() for _, _, g, _ in layer.parameters()]
        return {"h": h.shards[KEY], "m": m.shards[KEY], "dx": dx.shards[KEY], "grads": grads}
    tr = s["trainer"]
    tr.opt.zero_grad()
    loss = tr.model.forward_backward(s["tokens"], s["targets"], case["batch"] * case["seq"])
    return {"loss": loss.shards[KEY], "grads": [g.shards[KEY] for _, _, g, _ in tr.model.parameters()]}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def _attention_flops(case, train):
    pairs = case["batch"] * case["heads"] * case["seq"] ** 2 * (0.5 if case.get("causal", True) else 1.0)
    return pairs * 4 * D_HEAD * (3.5 if train else 1.0)      # two products forward, five backward


def work(case):
    k = case["kind"]
    if k == "linear":
        t, i, o = case["tokens"], case["d_in"], case["d_out"]
        return {"bytes": 2 * (2 * t * i + 2 * t * o + i * o) + 4 * i * o, "flops": 6 * t * i * o}
    if k == "attention":
        n = case["batch"] * case["seq"] * case["heads"] * D_HEAD
        return {"bytes": 2 * n * (8 if case["train"] else 4), "flops": _attention_flops(case, case["train"])}
    if k == "layernorm":
        n = case["tokens"] * case["d"]
        passes = 2 + 2 * case["residual"] + (2 + case["residual"] if case["train"] else 0)
        return {"bytes": 2 * n * passes, "flops": 8 * n}
    if k == "head_loss":
        t, d, vp = case["tokens"], case["d"], _padded(case["vocab"])
        return {"bytes": 2 * (2 * t * d + t * vp + d * vp) + 4 * d * vp, "flops": 6 * t * d * vp}
    if k == "adamw":
        n = case["n_sharded"] + case["n_rep"]
        return {"bytes": 30 * n, "flops": 20 * n}
    t, d = case["batch"] * case["seq"], case["d"]
    per_layer = 4 * d * d + 2 * d * case["ffn"]
    layers = case.get("layers", 1)
    flops = layers * (6 * t * per_layer + _attention_flops(case, True))
    if k == "gpt_block":
        return {"bytes": 6 * per_layer + 2 * 7 * t * d, "flops": flops}
    vp = _padded(case["vocab"])
    return {"bytes": 6 * (layers * per_layer + (2 * vp + case["seq"]) * d),
            "flops": flops + 6 * t * d * vp}


def tolerance(case):
    # about four times what the kernels show against ``exact``: single products, norms and the optimizer are off by
    # the rounding of their bf16 results (1.7e-3 to 2.4e-3), attention gradients 2.7e-3, blocks and models 5e-3 to 9e-3
    return {"rel": {"linear": 8e-3, "attention": 1.2e-2, "layernorm": 8e-3, "head_loss": 8e-3, "adamw": 8e-3,
                    "gpt_block": 3e-2, "gpt_model": 3e-2}[case["kind"]]}


# ----------------------------------------------------------------------------------------------
# the same outputs in 64 bits
# ----------------------------------------------------------------------------------------------
def _attend(qkv, batch, seq, heads, causal, dy=None):
    """softmax(q k^T / sqrt(128)) v per sequence and head on the per-head [q | k | v] layout, and the
    gradient with respect to qkv; one head at a time, queries in strips."""
    y = torch.empty(batch * seq, heads * D_HEAD, device=qkv.device, dtype=torch.float64)
    dqkv = torch.zeros_like(qkv) if dy is not None else None
    strip = max(128, min(seq, (1 << 26) // seq))
    for b in range(batch):
        rows = slice(b * seq, (b + 1) * seq)
        for h in range(heads):
            c = h * 3 * D_HEAD
            q, kk, v = (qkv[rows, c + i * D_HEAD:c + (i + 1) * D_HEAD] for i in range(3))
            for i in range(0, seq, strip):
                at = slice(b * seq + i, b * seq + min(seq, i + strip))
                n = at.stop - b * seq if causal else seq
                sc = q[i:i + strip] @ kk[:n].t() / math.sqrt(D_HEAD)
                if causal:
                    sc.masked_fill_(torch.arange(n, device=sc.device)[None, :] >
                                    torch.arange(i, i + sc.shape[0], device=sc.device)[:, None], float("-inf"))
                p = torch.softmax(sc, -1)
                o = p @ v[:n]
                cols = slice(h * D_HEAD, (h + 1) * D_HEAD)
                y[at, cols] = o
                if dy is not None:
                    do = dy[at, cols]
                    ds = p * (do @ v[:n].t() - (do * o).sum(1, keepdim=True)) / math.sqrt(D_HEAD)
                    dqkv[at, c:c + D_HEAD] = ds @ kk[:n]
                    dqkv[b * seq:b * seq + n, c + D_HEAD:c + 2 * D_HEAD] += ds.t() @ q[i:i + strip]
                    dqkv[b * seq:b * seq + n, c + 2 * D_HEAD:c + 3 * D_HEAD] += p.t() @ do
    return y, dqkv


class _Attention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, batch, seq, heads):
        ctx.save_for_backward(qkv)
        ctx.dims = (batch, seq, heads)
        return _attend(qkv, batch, seq, heads, True)[0]

    @staticmethod
    def backward(ctx, dy):
        return _attend(*ctx.saved_tensors, *ctx.dims, True, dy)[1], None, None, None


def _norm(x, gamma=None, bias=None):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], gamma, bias, 1e-5)


def _exact_block(x, delta, w, case):
    h = x if delta is None else x + delta
    a = _Attention.apply(_norm(h, w["ln1.gamma"], w["ln1.bias"]) @ w["in_proj"], case["batch"], case["seq"],
                         case["heads"])
    h = h + a @ w["out_proj"]
    g = torch.nn.functional.gelu(_norm(h, w["ln2.gamma"], w["ln2.bias"]) @ w["ff1"], approximate="tanh")
    return h, g @ w["ff2"].t()


def _leaf(t):
    return t.double().requires_grad_(True)


def exact(case, seed):
    k, v = case["kind"], _inputs(case, seed)
    if k == "linear":
        x, w, dy = (v[n].double() for n in ("x", "w", "dy"))
        if case["flow"] == "ls":
            return {"y": x @ w.t(), "dx": dy @ w, "dw": dy.t() @ x}
        return {"y": x @ w, "dx": dy @ w.t(), "dw": x.t() @ dy}
    if k == "attention":
        y, dqkv = _attend(v["qkv"].double(), case["batch"], case["seq"], case["heads"], case["causal"],
                          v["dy"].double() if case["train"] else None)
        return {"y": y, "dqkv": dqkv} if case["train"] else {"y": y}
    if k == "layernorm":
        h = v["x"].double() + v["res"].double() if case["residual"] else v["x"].double()
        h.requires_grad_(case["train"])
        gamma, bias = (_leaf(v[n]) for n in ("gamma", "bias")) if case["affine"] else (None, None)
        y = _norm(h, gamma, bias)
        out = {"y": y.detach()}
        if case["residual"]:
            out["h"] = h.detach()
        if case["train"]:
            y.backward(v["dy"].double())
            out["dx"] = h.grad + v["dres"].double() if case["residual"] else h.grad
            if case["affine"]:
                out["dgamma"], out["dbias"] = gamma.grad, bias.grad
        return out
    if k == "head_loss":
        x, w, t = v["x"].double(), v["w"].double(), v["targets"]
        logits = x @ w
        logits[:, case["vocab"]:] = float("-inf")
        loss = torch.logsumexp(logits, 1) - logits.gather(1, t[:, None])[:, 0]
        d = torch.softmax(logits, 1)
        del logits
        d.scatter_add_(1, t[:, None], torch.full_like(t, -1.0, dtype=torch.float64)[:, None])
        d /= case["tokens"]
        return {"loss": loss, "dlogits": d, "dx": d @ w.t(), "dw": x.t() @ d}
    if k == "adamw":
        b1, b2, lr, eps, wd, step = 0.9, 0.95, 1e-4, 1e-8, 0.01, 100
        norm = math.sqrt(sum(float(g[1].double().square().sum()) for g in v.values()))
        scale = min(1.0, 1.0 / (norm + 1e-6))
        out = []
        for param, grad, m, var in v.values():
            p, g = param.double(), grad.double() * scale
            m = b1 * m.double() + (1 - b1) * g
            var = b2 * var.double() + (1 - b2) * g * g
            p = p - lr * ((m / (1 - b1 ** step)) / ((var / (1 - b2 ** step)).sqrt() + eps) + wd * p)
            out.append({"param": p, "master": p, "m": m, "v": var})
        return out
    w = {n: _leaf(t) for n, t in v["w"].items()}
    if k == "gpt_block":
        x, delta = _leaf(v["x"]), v["delta"].double()
        h, m = _exact_block(x, delta, w, case)
        torch.autograd.backward([h, m], [v["dh"].double(), v["dm"].double()])
        return {"h": h.detach(), "m": m.detach(), "dx": x.grad, "grads": [t.grad for t in w.values()]}
    pos = torch.arange(case["batch"] * case["seq"], device="cuda") % case["seq"]
    x, delta = w["tok"][v["tokens"]] + w["pos"][pos], None
    for i in range(case["layers"]):
        x, delta = _exact_block(x, delta, {n: w[f"{i}.{n}"] for n, _ in _block_shapes(case["d"], case["ffn"])}, case)
    y = _norm(x + delta, w["ln_f.gamma"], w["ln_f.bias"])
    logits = (y @ w["head"])[:, :case["vocab"]]
    loss = torch.nn.functional.cross_entropy(logits, v["targets"])
    loss.backward()
    return {"loss": loss.detach(), "grads": [t.grad for t in w.values()]}
