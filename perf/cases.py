"""Performance cases of the library on one GPU.

The cases are what a training or serving program has this library do on every step, through its public Python entry
points: the projection matmuls, the FFN half of a decoder layer with its backward pass, the single-pass pieces of a layer, the optimizer step, expert routing with dispatch and combine, collectives, and one whole decoder stack.  Sizes are
those of the Llama-3-70B-shaped benchmark model (hidden 8192, 64 query and 8 key / value heads of 128, FFN 28672), of its
8-way tensor-parallel shards and of the MoE benchmark (hidden 7168, 256 experts, top-8).  Operators that need several
ranks run on ranks emulated on one GPU, which is how the library runs them where a single GPU is at hand.

``listed()`` holds the fixed cases, ``draw(rng)`` one more of the same ranges.
"""
import math

import torch

import hccl_b200 as hb
from hccl_b200 import Communicator, ReduceOp
from hccl_b200.models import LlamaConfig, LlamaStack
from hccl_b200.ops import FusedAdamW, fused, mc2
from hccl_b200.ops.moe import MoeDispatcher, expert_offsets
from hccl_b200.parallel import ColumnParallelLinear, RowParallelLinear, TPContext

EPS = 1e-5
ADAM = {"lr": 1e-3, "betas": (0.9, 0.95), "eps": 1e-8, "weight_decay": 0.1}
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp32": 4}


def listed():
    return [
        # one decode step's output projection: 16 sequences, the whole weight is read for 16 rows
        {"name": "matmul_decode", "kind": "matmul", "m": 16, "n": 8192, "k": 8192, "trans_a": False, "trans_b": True},
        # QKV projection of a 1000-token prompt: rows that are no multiple of a tile
        {"name": "matmul_prefill", "kind": "matmul", "m": 1000, "n": 10240, "k": 8192, "trans_a": False, "trans_b": True},
        # FFN half of a decoder layer on one rank of an 8-way tensor-parallel group: add + norm, gate / up projection,
        # SwiGLU, down projection, the next add + norm, a training step's forward and backward
        {"name": "ffn_train", "kind": "ffn", "s": 4096, "hidden": 8192, "ffn": 3584},
        # residual add + RMSNorm of a training step, forward and backward
        {"name": "norm_train", "kind": "norm", "rows": 4096, "hidden": 8192, "delta": True, "backward": True},
        # the same norm in a decode step of 16 sequences
        {"name": "norm_decode", "kind": "norm", "rows": 16, "hidden": 8192, "delta": True, "backward": False},
        # SwiGLU at the full FFN width, forward and backward
        {"name": "swiglu_train", "kind": "swiglu", "rows": 4096, "f": 28672, "backward": True},
        # rotary embedding of the query heads, a column slice of the QKV projection's output, forward and backward
        {"name": "rope_train", "kind": "rope", "s": 8192, "heads": 64, "d": 128, "extra": 2048, "backward": True},
        # optimizer step over one decoder layer of an 8-way tensor-parallel rank (norms, QKV, O, gate / up, down)
        {"name": "adamw_layer", "kind": "adamw", "param": "bf16", "state": "fp32",
         "sizes": "8192,8192,10485760,8388608,58720256,29360128"},
        # row range of every expert for a batch's routing table
        {"name": "expert_offsets", "kind": "offsets", "tokens": 8192, "topk": 8, "experts": 256},
        # expert-parallel layer on 8 ranks: dispatch (fp8 with block scales), an expert that only dequantises, combine
        {"name": "moe_8_ranks", "kind": "moe", "ranks": 8, "tokens": 256, "hidden": 7168, "experts": 256, "topk": 8},
        # a small tensor-parallel AllReduce of a decode step (16 rows of 8192), 8 ranks
        {"name": "all_reduce_decode", "kind": "collective", "op": "all_reduce", "ranks": 8, "count": 131072, "dtype": "bf16"},
        # one whole call of the decoder stack: embedding, one layer at full width, final norm, forward and backward
        {"name": "stack_train", "kind": "stack", "s": 1024, "hidden": 8192, "heads": 64, "kv_heads": 8, "ffn": 28672, "layers": 1, "vocab": 4096},
    ]


# ----------------------------------------------------------------------------- drawn cases
def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v) // step * step)) if step == 1 or int(v) >= step else step


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "ffn", "norm", "norm", "swiglu", "rope", "adamw", "offsets", "moe", "collective", "collective", "stack"])
    if kind == "matmul":
        while True:
            c = {"kind": kind, "m": _log(rng, 1, 8192), "n": _log(rng, 64, 16384, 8), "k": _log(rng, 64, 16384, 8),
                 "trans_a": rng.random() < 0.25, "trans_b": rng.random() < 0.7}
            if c["trans_a"]:
                c["m"] = max(8, c["m"] // 8 * 8)
            if 2 * c["m"] * c["n"] * c["k"] <= 1.2e12:
                return c
    if kind == "ffn":
        return {"kind": kind, "s": _log(rng, 64, 4096, 8), "hidden": _log(rng, 512, 8192, 8), "ffn": _log(rng, 256, 3584, 8)}
    if kind == "norm":
        return {"kind": kind, "rows": _log(rng, 1, 8192), "hidden": _log(rng, 128, 8192, 8), "delta": rng.random() < 0.8, "backward": rng.random() < 0.6}
    if kind == "swiglu":
        return {"kind": kind, "rows": _log(rng, 1, 4096), "f": _log(rng, 128, 28672, 8), "backward": rng.random() < 0.6}
    if kind == "rope":
        d = rng.choice([64, 128])
        return {"kind": kind, "s": _log(rng, 1, 8192), "heads": _log(rng, 1, 64), "d": d, "extra": rng.choice([0, 2, 16]) * d, "backward": rng.random() < 0.6}
    if kind == "adamw":
        param, state = rng.choice([("bf16", "bf16"), ("bf16", "fp32"), ("fp32", "fp32")])
        return {"kind": kind, "param": param, "state": state, "sizes": ",".join(str(_log(rng, 64, 1 << 25)) for _ in range(rng.randint(1, 12)))}
    if kind == "offsets":
        return {"kind": kind, "tokens": _log(rng, 1, 32768), "topk": rng.choice([1, 2, 4, 6, 8]), "experts": rng.choice([8, 16, 60, 64, 128, 160, 256, 512])}
    if kind == "moe":
        return {"kind": kind, "ranks": rng.choice([2, 4, 8]), "tokens": _log(rng, 1, 256), "hidden": _log(rng, 1024, 7168, 128),
                "experts": rng.choice([32, 64, 128, 256]), "topk": rng.choice([1, 2, 4, 8])}
    if kind == "collective":
        return {"kind": kind, "op": rng.choice(["all_reduce", "reduce_scatter", "all_gather", "all_to_all"]), "ranks": rng.choice([2, 4, 8]),
                "count": _log(rng, 64, 1 << 22), "dtype": rng.choice(["bf16", "fp32"])}
    heads = rng.choice([8, 16, 32])
    return {"kind": "stack", "s": _log(rng, 64, 1024, 8), "hidden": heads * 128, "heads": heads, "kv_heads": 8, "ffn": _log(rng, 1024, 14336, 64),
            "layers": rng.randint(1, 2), "vocab": 4096}


# ----------------------------------------------------------------------------- inputs
# A program keeps its communicator, and the receive buffers of its expert layer, for as long as it runs.
_comms = {}
_moe = {}


def _communicators(ranks):
    if ranks not in _comms:
        _comms[ranks] = Communicator.emulated(ranks, hb.make_config(buffer_mib=64))
    return _comms[ranks]


def _dispatchers(case):
    key = (case["ranks"], case["tokens"], case["hidden"], case["experts"], case["topk"])
    if key not in _moe:
        comms = _communicators(case["ranks"])
        while _moe:                          # another configuration: its buffers go back first
            old, ds = _moe.popitem()
            torch.cuda.synchronize()
            for name in ("recv_x", "recv_scale", "recv_src", "y"):
                for c, d in zip(_communicators(old[0]), ds):
                    c.free(getattr(d, name))
        # room for routing an eighth more uneven than an even one, and a few rows more where there are few tokens
        capacity = int(1.125 * case["tokens"] * case["topk"]) + 16 * case["topk"]
        _moe[key] = [MoeDispatcher(c, case["tokens"], case["hidden"], case["topk"], case["experts"], capacity=capacity) for c in comms]
    return _moe[key]


class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        out = torch.empty(shape, device="cuda", dtype=dtype)
        flat, step = out.view(-1), 1 << 26
        for o in range(0, flat.numel(), step):
            m = min(step, flat.numel() - o)
            flat[o:o + m] = torch.randn(m, device="cuda", generator=self.g).mul_(std)
        return out

    def weight(self, n):          # a norm's weight
        return (1 + 0.1 * torch.randn(n, device="cuda", generator=self.g)).bfloat16()


def _inputs(case, seed):
    """The tensors of a case, made from the seed alone."""
    r, k = _Rand(seed), case["kind"]
    if k == "matmul":
        m, n, kk = case["m"], case["n"], case["k"]
        return {"a": r.normal(*((kk, m) if case["trans_a"] else (m, kk))), "b": r.normal(*((n, kk) if case["trans_b"] else (kk, n)), std=0.02)}
    if k == "ffn":
        s, h, f = case["s"], case["hidden"], case["ffn"]
        return {"x": r.normal(s, h), "delta": r.normal(s, h, std=0.5), "norm1": r.weight(h), "norm2": r.weight(h), "gate_up": r.normal(2 * f, h, std=0.02),
                "down": r.normal(h, f, std=0.02), "d_out": r.normal(s, h), "d_h": r.normal(s, h)}
    if k == "norm":
        rows, h = case["rows"], case["hidden"]
        d = {"x": r.normal(rows, h), "delta": r.normal(rows, h, std=0.5) if case["delta"] else None, "w": r.weight(h)}
        if case["backward"]:
            d["d_out"], d["d_h"] = r.normal(rows, h), r.normal(rows, h)
        return d
    if k == "swiglu":
        d = {"x": r.normal(case["rows"], 2 * case["f"])}
        if case["backward"]:
            d["dy"] = r.normal(case["rows"], case["f"])
        return d
    if k == "rope":
        s, nh, dim = case["s"], case["heads"], case["d"]
        d = {"wide": r.normal(s, nh * dim + case["extra"])}
        ang = torch.outer(torch.arange(s, device="cuda", dtype=torch.float32),
                          1.0 / (500000.0 ** (torch.arange(0, dim, 2, device="cuda", dtype=torch.float32) / dim)))
        d["cos"], d["sin"] = ang.cos(), ang.sin()
        if case["backward"]:
            d["dy"] = r.normal(s, nh, dim)
        return d
    if k == "adamw":
        sizes = [int(v) for v in case["sizes"].split(",")]
        return {"p": [r.normal(n, std=0.02, dtype=DTYPES[case["param"]]) for n in sizes], "g": [r.normal(n, std=0.01, dtype=DTYPES[case["param"]]) for n in sizes]}
    if k == "offsets":
        logits = torch.randn(case["tokens"], case["experts"], device="cuda", generator=r.g)
        return {"idx": torch.topk(logits, min(case["topk"], case["experts"]), dim=-1)[1].int().contiguous()}
    if k == "moe":
        d = {"x": [], "idx": [], "w": []}
        for _ in range(case["ranks"]):
            d["x"].append(r.normal(case["tokens"], case["hidden"]))
            w, i = torch.topk(torch.softmax(torch.randn(case["tokens"], case["experts"], device="cuda", generator=r.g), -1), case["topk"], dim=-1)
            d["idx"].append(i.int().contiguous())
            d["w"].append((w / w.sum(-1, keepdim=True)).float().contiguous())
        return d
    if k == "collective":
        p, n = case["ranks"], case["count"]
        many = n * p if case["op"] in ("reduce_scatter", "all_to_all") else n
        return {"send": [r.normal(many, dtype=DTYPES[case["dtype"]]) for _ in range(p)]}
    assert k == "stack", k
    q, kv = case["heads"] * 128, case["kv_heads"] * 128
    d = {"embed": r.normal(case["vocab"], case["hidden"], std=0.5), "final_norm": r.weight(case["hidden"]), "layers": []}
    for _ in range(case["layers"]):
        d["layers"].append({"attn_norm": r.weight(case["hidden"]), "ffn_norm": r.weight(case["hidden"]),
                            "qkv": r.normal(q + 2 * kv, case["hidden"], std=0.02), "o": r.normal(case["hidden"], q, std=0.02),
                            "gate_up": r.normal(2 * case["ffn"], case["hidden"], std=0.02), "down": r.normal(case["hidden"], case["ffn"], std=0.02)})
    d["tokens"] = torch.randint(0, case["vocab"], (case["s"],), device="cuda", generator=r.g)
    d["dy"] = r.normal(case["s"], case["hidden"])
    return d


def prepare(case, seed):
    d, k = _inputs(case, seed), case["kind"]
    d["case"] = case
    if k == "ffn":
        ctx = TPContext(None)
        for name, module in (("gate_up", ColumnParallelLinear(case["hidden"], 2 * case["ffn"], ctx, "gate_up")),
                             ("down", RowParallelLinear(case["ffn"], case["hidden"], ctx, "down"))):
            module.weight.data.copy_(d[name])
            d[name] = module
        for name in ("x", "delta", "norm1", "norm2"):
            d[name].requires_grad_()
    elif k == "rope":
        d["x"] = d.pop("wide")[:, :case["heads"] * case["d"]].view(case["s"], case["heads"], case["d"]).requires_grad_(case["backward"])
    elif k in ("norm", "swiglu") and case["backward"]:
        for name in ("x", "delta", "w"):
            if d.get(name) is not None:
                d[name].requires_grad_()
    elif k == "adamw":
        d["p"] = [torch.nn.Parameter(p) for p in d["p"]]
        for p, g in zip(d["p"], d["g"]):
            p.grad = g
        d["opt"] = FusedAdamW(d["p"], state_dtype=DTYPES[case["state"]], **ADAM)
    elif k == "moe":
        d["disp"] = _dispatchers(case)
    elif k == "collective":
        p, n = case["ranks"], case["count"]
        many = n * p if case["op"] in ("all_gather", "all_to_all") else n
        d["comms"] = _communicators(p)
        d["recv"] = [torch.empty(many, device="cuda", dtype=DTYPES[case["dtype"]]) for _ in range(p)]
    elif k == "stack":
        cfg = LlamaConfig(hidden=case["hidden"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], ffn=case["ffn"], n_layers=case["layers"],
                          vocab=case["vocab"], norm_eps=EPS)
        model = LlamaStack(cfg, TPContext(None))
        with torch.no_grad():
            model.embed.copy_(d.pop("embed"))
            model.final_norm.copy_(d.pop("final_norm"))
            for layer, w in zip(model.layers, d.pop("layers")):
                layer.attn_norm.copy_(w["attn_norm"])
                layer.ffn_norm.copy_(w["ffn_norm"])
                for name in ("qkv", "o", "gate_up", "down"):
                    getattr(layer, name).weight.copy_(w[name])
        d["model"] = model
    return d


# ----------------------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "matmul":
        return mc2.matmul(s["a"], s["b"], trans_a=case["trans_a"], trans_b=case["trans_b"])
    if k == "ffn":
        leaves = [s["x"], s["delta"], s["norm1"], s["gate_up"].weight, s["down"].weight, s["norm2"]]
        for t in leaves:
            t.grad = None
        x, h = fused.add_rms_norm(s["x"], s["delta"], s["norm1"], EPS)
        x, h = fused.add_rms_norm(x, s["down"](fused.swiglu(s["gate_up"](h))), s["norm2"], EPS)
        torch.autograd.backward([x, h], [s["d_out"], s["d_h"]])
        return {"x": x.detach(), "h": h.detach(), "grads": [t.grad for t in leaves]}
    if k == "norm":
        x, delta, w = s["x"], s["delta"], s["w"]
        x_out, h = fused.add_rms_norm(x, delta, w, EPS)
        if not case["backward"]:
            return {"x_out": x_out, "h": h}
        x.grad = w.grad = None
        if delta is not None:
            delta.grad = None
            torch.autograd.backward([x_out, h], [s["d_out"], s["d_h"]])
            return {"x_out": x_out.detach(), "h": h.detach(), "dx": x.grad, "ddelta": delta.grad, "dw": w.grad}
        torch.autograd.backward(h, s["d_h"])
        return {"h": h.detach(), "dx": x.grad, "dw": w.grad}
    if k == "swiglu":
        x = s["x"]
        y = fused.swiglu(x)
        if not case["backward"]:
            return y
        x.grad = None
        y.backward(s["dy"])
        return {"y": y.detach(), "dx": x.grad}
    if k == "rope":
        y = fused.rope(s["x"], s["cos"], s["sin"])
        if not case["backward"]:
            return y
        return {"y": y.detach(), "dx": torch.autograd.grad(y, s["x"], s["dy"])[0]}
    if k == "adamw":
        s["opt"].step()
        st = s["opt"].state
        return {"p": [p.detach() for p in s["p"]], "m": [st[p]["exp_avg"] for p in s["p"]], "v": [st[p]["exp_avg_sq"] for p in s["p"]]}
    if k == "offsets":
        return expert_offsets(s["idx"], case["experts"])
    if k == "moe":
        got = [d.dispatch(x, i) for d, x, i in zip(s["disp"], s["x"], s["idx"])]
        for d, g in zip(s["disp"], got):     # the expert: dequantise
            blocks = (d.cfg.capacity, case["hidden"] // 128, 128)
            torch.mul(g.x_fp8.to(torch.bfloat16).view(blocks), g.scales.unsqueeze(-1), out=d.y.view(blocks))
        return {"out": [d.combine(w) for d, w in zip(s["disp"], s["w"])], "offsets": [g.offsets.clone() for g in got]}
    if k == "collective":
        for c, a, b in zip(s["comms"], s["send"], s["recv"]):
            if case["op"] == "all_reduce":
                c.all_reduce(a, b, ReduceOp.SUM)
            elif case["op"] == "reduce_scatter":
                c.reduce_scatter(a, b, ReduceOp.SUM)
            elif case["op"] == "all_gather":
                c.all_gather(a, b)
            else:
                c.all_to_all(a, b)
        return s["recv"]
    model = s["model"]
    for p in model.parameters():
        p.grad = None
    y = model(s["tokens"])
    y.backward(s["dy"])
    return {"y": y.detach(), "grads": {name: p.grad for name, p in model.named_parameters()}}


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    k = case["kind"]
    if k == "matmul":
        m, n, kk = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * kk + n * kk + m * n), "flops": 2 * m * n * kk}
    if k == "ffn":
        s, h, f = case["s"], case["hidden"], case["ffn"]
        # x, delta, the two gradients in, the stream, its norm and the input's gradient out; weights in, their gradients out
        return {"bytes": 2 * (7 * s * h + 2 * (3 * f * h + 2 * h)), "flops": 18 * s * h * f}
    if k == "norm":
        n = case["rows"] * case["hidden"]
        fwd = 4 if case["delta"] else 2                                      # x, delta in; x_out, h out
        bwd = (3 if case["delta"] else 1) if case["backward"] else 0         # the gradients in, dx out (dx is delta's gradient too)
        bwd += 1 if case["backward"] and not case["delta"] else 0
        return {"bytes": 2 * n * (fwd + bwd), "flops": n * (8 if not case["backward"] else 20)}
    if k == "swiglu":
        n = case["rows"] * case["f"]
        return {"bytes": 2 * n * (3 + (3 if case["backward"] else 0)), "flops": n * (6 if not case["backward"] else 20)}
    if k == "rope":
        n = case["s"] * case["heads"] * case["d"]
        return {"bytes": 2 * n * (4 if case["backward"] else 2) + 4 * case["s"] * case["d"], "flops": 3 * n * (2 if case["backward"] else 1)}
    if k == "adamw":
        n = sum(int(v) for v in case["sizes"].split(","))
        return {"bytes": n * (3 * SIZE[case["param"]] + 4 * SIZE[case["state"]]), "flops": 14 * n}
    if k == "offsets":
        return {"bytes": 4 * (case["tokens"] * min(case["topk"], case["experts"]) + case["experts"] + 1), "flops": case["tokens"] * case["topk"]}
    if k == "moe":
        t, h = case["ranks"] * case["tokens"], case["hidden"]
        rows = t * case["topk"]
        # x in, fp8 rows and scales out and in again, bf16 expert rows out and in again, the sum out
        return {"bytes": 2 * t * h + 2 * rows * (h + h // 32) + 4 * rows * h + 2 * t * h, "flops": 6 * rows * h}
    if k == "collective":
        p, n, es = case["ranks"], case["count"], SIZE[case["dtype"]]
        one = n * p if case["op"] != "all_reduce" else n
        moved = {"all_reduce": 2 * n, "reduce_scatter": one + n, "all_gather": one + n, "all_to_all": 2 * one}[case["op"]]
        adds = (p - 1) * one if case["op"] in ("all_reduce", "reduce_scatter") else 0
        return {"bytes": p * moved * es, "flops": adds}
    s, h = case["s"], case["hidden"]
    layer = h * 128 * (case["heads"] + 2 * case["kv_heads"]) + h * 128 * case["heads"] + 3 * h * case["ffn"]
    attention = 2 * 2 * s * s * 128 * case["heads"] / 2
    return {"bytes": 2 * 2 * (case["layers"] * (layer + 2 * h) + case["vocab"] * h + h + s * h), "flops": case["layers"] * (6 * s * layer + 3.5 * attention)}


# Rounding a result to bf16 is off by 1.7e-3 of it (2-norm) and by 3.9e-3 at most, one unit in the last place being up to
# 7.8e-3; the figures allow about four times what a single rounding, or for the stack the whole chain, was measured at.
def tolerance(case):
    k = case["kind"]
    if k == "offsets" or (k == "collective" and case["op"] in ("all_gather", "all_to_all")):
        return "exact"
    if k == "collective":
        return {"rel": 1e-6, "max": 1e-5} if case["dtype"] == "fp32" else {"rel": 7e-3, "max": 0.04}
    if k == "adamw":
        # moments and parameters of one step; bf16 storage rounds each of them once
        return {"rel": 7e-3, "max": 0.04} if "bf16" in (case["param"], case["state"]) else {"rel": 2e-6, "max": 1e-4}
    if k == "moe":
        return {"rel": 0.01, "max": 0.06}
    if k == "ffn":
        return {"rel": 0.02, "max": 0.2}
    if k == "stack":
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 7e-3, "max": 0.04}


# ----------------------------------------------------------------------------- the same in 64 bits
def _norm64(x, w):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w


def _rope64(x, cos, sin):
    h = x.shape[-1] // 2
    a, b, c, s = x[..., :h], x[..., h:], cos[:, None, :], sin[:, None, :]
    return torch.cat((a * c - b * s, b * c + a * s), dim=-1)


def _swiglu64(x):
    g, u = x.chunk(2, dim=-1)
    return g * torch.sigmoid(g) * u


def _quantised64(x):
    """e4m3 values with one scale per 128 elements, in 64 bits."""
    b = x.double().view(x.shape[0], -1, 128)
    scale = b.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
    return ((b / scale).float().to(torch.float8_e4m3fn).double() * scale).view(x.shape)


def exact(case, seed):
    d, k = _inputs(case, seed), case["kind"]
    if k == "matmul":
        a, b = d["a"].double(), d["b"].double()
        return (a.t() if case["trans_a"] else a) @ (b.t() if case["trans_b"] else b)
    if k == "ffn":
        p = [d[name].double().requires_grad_() for name in ("x", "delta", "norm1", "gate_up", "down", "norm2")]
        x = p[0] + p[1]
        x = x + _swiglu64(_norm64(x, p[2]) @ p[3].t()) @ p[4].t()
        h = _norm64(x, p[5])
        grads = torch.autograd.grad([x, h], p, [d["d_out"].double(), d["d_h"].double()])
        return {"x": x.detach(), "h": h.detach(), "grads": list(grads)}
    if k == "norm":
        x, w = d["x"].double().requires_grad_(), d["w"].double().requires_grad_()
        if d["delta"] is None:
            h = _norm64(x, w)
            if not case["backward"]:
                return {"x_out": x.detach(), "h": h.detach()}
            dx, dw = torch.autograd.grad(h, [x, w], d["d_h"].double())
            return {"h": h.detach(), "dx": dx, "dw": dw}
        # the stored sum is bf16 by definition, and the norm is taken of it
        x_out = (d["x"] + d["delta"]).double().requires_grad_()
        h = _norm64(x_out, w)
        whole = d["x"].double() + d["delta"].double()
        if not case["backward"]:
            return {"x_out": whole, "h": h.detach()}
        dx, dw = torch.autograd.grad(h, [x_out, w], d["d_h"].double())
        dx = dx + d["d_out"].double()
        return {"x_out": whole, "h": h.detach(), "dx": dx, "ddelta": dx, "dw": dw}
    if k == "swiglu":
        x = d["x"].double().requires_grad_()
        y = _swiglu64(x)
        if not case["backward"]:
            return y.detach()
        return {"y": y.detach(), "dx": torch.autograd.grad(y, x, d["dy"].double())[0]}
    if k == "rope":
        n, nh, dim = case["s"], case["heads"], case["d"]
        x = d["wide"][:, :nh * dim].view(n, nh, dim).double().requires_grad_()
        y = _rope64(x, d["cos"].double(), d["sin"].double())
        if not case["backward"]:
            return y.detach()
        return {"y": y.detach(), "dx": torch.autograd.grad(y, x, d["dy"].double())[0]}
    if k == "adamw":
        (b1, b2), out = ADAM["betas"], {"p": [], "m": [], "v": []}
        for p, g in zip(d["p"], d["g"]):
            p, g = p.double(), g.double()
            m, v = (1 - b1) * g, (1 - b2) * g * g
            step = (m / (1 - b1)) / ((v / (1 - b2)).sqrt() + ADAM["eps"])
            out["p"].append(p * (1 - ADAM["lr"] * ADAM["weight_decay"]) - ADAM["lr"] * step)
            out["m"].append(m)
            out["v"].append(v)
        return out
    if k == "offsets":
        n = torch.bincount(d["idx"].long().view(-1), minlength=case["experts"])
        return torch.cat((n.new_zeros(1), n.cumsum(0))).int()
    if k == "moe":
        out = [_quantised64(x) * w.double().sum(-1, keepdim=True) for x, w in zip(d["x"], d["w"])]
        return {"out": out, "offsets": None}
    if k == "collective":
        p, n, send = case["ranks"], case["count"], [t.double() for t in d["send"]]
        if case["op"] == "all_reduce":
            return [torch.stack(send).sum(0)] * p
        if case["op"] == "reduce_scatter":
            return list(torch.stack(send).sum(0).split(n))
        if case["op"] == "all_gather":
            return [torch.cat(send)] * p
        return [torch.cat([t[q * n:(q + 1) * n] for t in send]) for q in range(p)]
    s, heads, kv = case["s"], case["heads"], case["kv_heads"]
    names, params = [], []

    def leaf(name, t):
        names.append(name)
        params.append(t.double().requires_grad_())
        return params[-1]

    x = leaf("embed", d["embed"])[d["tokens"]]
    ang = torch.outer(torch.arange(s, device="cuda", dtype=torch.float64), 1.0 / (500000.0 ** (torch.arange(0, 128, 2, device="cuda", dtype=torch.float64) / 128)))
    cos, sin = ang.cos(), ang.sin()
    hidden_mask = torch.ones(s, s, device="cuda", dtype=torch.bool).triu(1)
    for i, w in enumerate(d["layers"]):
        w = {name: leaf("layers.%d.%s" % (i, name if name.endswith("norm") else name + ".weight"), t) for name, t in w.items()}
        q, kk, v = (_norm64(x, w["attn_norm"]) @ w["qkv"].t()).split([heads * 128, kv * 128, kv * 128], dim=-1)
        q, kk = _rope64(q.view(s, heads, 128), cos, sin), _rope64(kk.view(s, kv, 128), cos, sin)
        kk, v = (t.repeat_interleave(heads // kv, dim=1) for t in (kk, v.view(s, kv, 128)))
        p = torch.einsum("qhd,khd->hqk", q, kk).mul(128 ** -0.5).masked_fill(hidden_mask, -math.inf).softmax(-1)
        x = x + torch.einsum("hqk,khd->qhd", p, v).reshape(s, heads * 128) @ w["o"].t()
        x = x + _swiglu64(_norm64(x, w["ffn_norm"]) @ w["gate_up"].t()) @ w["down"].t()
    y = _norm64(x, leaf("final_norm", d["final_norm"]))
    grads = torch.autograd.grad(y, params, d["dy"].double())
    return {"y": y.detach(), "grads": dict(zip(names, grads))}
