"""Performance cases of the library, each one pass through its public entry points.

The ranges are those of the training engine and of the collective benchmarks: the linear layers, layer
norms, output head and optimizer shards of the GPT presets (``pccl/models/gpt.py``: widths 256 to 4096,
vocabulary 50304), from a single short sequence to a micro-batch of four times 2048 tokens, and the
collectives that gather and reduce one block's parameters over up to eight ranks.  The ranks of a collective are
driven by one process on one device (``Communicator.emulated_world``): the same kernels, flags and schedules as
across devices, with local memory in the place of the links.
"""
import math

import torch

import pccl
from pccl import schedule as sch
from pccl.models import gpt
from pccl.ops import gemm

DEV = "cuda:0"
BF16 = torch.bfloat16
_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_HEAP = 1 << 30
_STAGING = 128 << 20
_comms = {}


def _comm(world):
    """A program keeps one communicator per world for its whole life."""
    if world not in _comms:
        _comms[world] = pccl.Communicator.emulated_world(world, device=0, heap_bytes=_HEAP, staging_bytes=_STAGING)
    return _comms[world]


def listed():
    return [
        # qkv projection of the smallest preset, two sequences of 128 tokens: forward and both gradients; launches count
        {"name": "linear_small", "kind": "linear", "tokens": 256, "n_in": 256, "n_out": 768},
        # qkv projection of the 350M preset on a ragged token count, as a last, partly filled batch has
        {"name": "linear_ragged", "kind": "linear", "tokens": 1000, "n_in": 1024, "n_out": 3072},
        # first MLP layer of the 1.3B preset at a full micro-batch of 4 x 2048 tokens
        {"name": "linear_large", "kind": "linear", "tokens": 8192, "n_in": 2048, "n_out": 8192},
        # first MLP layer of the 350M preset with its activation in the same kernel (the engine's fused_gelu_gemm option)
        {"name": "linear_gelu", "kind": "linear_gelu", "tokens": 4096, "n_in": 1024, "n_out": 4096},
        # residual add + layer norm and its backward, 1.3B preset, full micro-batch
        {"name": "norm", "kind": "norm", "rows": 8192, "width": 2048},
        # the same for the 7B preset on an odd number of tokens
        {"name": "norm_ragged", "kind": "norm", "rows": 1501, "width": 4096},
        # final norm, tied output projection and loss, forward and backward, 350M preset, one sequence
        {"name": "head", "kind": "head", "tokens": 2048, "width": 1024, "vocab": 50304},
        # gradient norm and AdamW over one 1.3B block (12 d^2 weights + 13 d biases and gains), fp32 gradients
        {"name": "optimizer", "kind": "optimizer", "count": 50358272, "grad": "fp32"},
        # parameters of one 1.3B block gathered over eight ranks, symmetric buffers
        {"name": "all_gather", "kind": "all_gather", "world": 8, "algo": "direct", "dtype": "bf16", "count": 6294784, "symmetric": True},
        # its gradients reduced over eight ranks by recursive halving, private input, mean in fp32
        {"name": "reduce_scatter", "kind": "reduce_scatter", "world": 8, "algo": "recursive", "dtype": "bf16", "count": 6294784, "symmetric": False},
        # a ragged mid-size tensor averaged in place over four ranks
        {"name": "all_reduce", "kind": "all_reduce", "world": 4, "algo": "direct", "dtype": "fp32", "count": 1000003, "symmetric": True},
        # one transformer block of the 350M preset, forward and backward, two sequences of 2048 tokens
        {"name": "block", "kind": "block", "batch": 2, "seq": 2048, "width": 1024, "heads": 16, "ff": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear_gelu", "norm", "norm", "head", "optimizer", "all_gather", "reduce_scatter",
                       "all_reduce", "block"])
    if kind == "linear":
        # the weight gradient contracts over the tokens, in units of 8; features come in units of 64
        while True:
            c = {"kind": kind, "tokens": 8 * _log(rng, 4, 1024), "n_in": 64 * _log(rng, 4, 128), "n_out": 64 * _log(rng, 4, 128)}
            if c["tokens"] * c["n_in"] * c["n_out"] <= 8192 * 2048 * 8192:
                return c
    if kind == "linear_gelu":
        while True:
            c = {"kind": kind, "tokens": _log(rng, 16, 8192), "n_in": 8 * _log(rng, 32, 512), "n_out": 8 * _log(rng, 32, 1024)}
            if c["tokens"] * c["n_in"] * c["n_out"] <= 8192 * 2048 * 8192:
                return c
    if kind == "norm":
        return {"kind": kind, "rows": _log(rng, 8, 12000), "width": rng.choice([1024, 2048, 4096])}
    if kind == "head":
        while True:
            c = {"kind": kind, "tokens": 8 * _log(rng, 8, 256), "width": rng.choice([1024, 2048]),
                 "vocab": rng.choice([1024, 2048, 32000, 50304])}
            if c["tokens"] * c["width"] <= 2048 * 1024:
                return c
    if kind == "optimizer":
        return {"kind": kind, "count": _log(rng, 1000, 50000000), "grad": rng.choice(["fp32", "bf16"])}
    if kind == "block":
        return {"kind": kind, "batch": rng.choice([1, 2, 3]), "seq": 8 * _log(rng, 16, 256), "width": 1024, "heads": 16, "ff": 4096}
    world = rng.choice([2, 4, 8])
    dtype = rng.choice(["bf16", "bf16", "fp32", "fp16"])
    count = _log(rng, 64, 6000000 // (2 if dtype == "fp32" else 1))
    if rng.random() < 0.5:
        count = (count + 255) // 256 * 256
    c = {"kind": kind, "world": world, "dtype": dtype, "count": count, "symmetric": rng.random() < 0.5}
    if kind == "all_gather":
        c["algo"] = rng.choice(["direct", "ring", "recursive", "pull"])
    elif kind == "reduce_scatter":
        c["algo"] = rng.choice(["direct", "ring", "recursive"] + (["pull", "pull"] if c["symmetric"] else []))
    else:
        c["algo"] = rng.choice(["direct", "direct", "ring", "recursive"])
    return c


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, shape, std=1.0, dtype=BF16):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(dtype)


def _config(case):
    return gpt.GPTConfig(1, case["width"], case.get("heads", 16), case.get("ff", 4 * case["width"]), vocab=case.get("vocab", 64),
                         seq_len=case.get("seq", case.get("tokens", 0)))


def _params(case, unit_index, g):
    """One unit's parameters as the engine holds them: views into a flat buffer, and views for the gradients."""
    unit = gpt.unit_specs(_config(case))[unit_index]
    flat = torch.empty(unit.numel, dtype=BF16, device=DEV)
    views = gpt.views(unit, flat)
    for p in unit.params:
        # gains around one and small biases, as after some steps of training
        mean = 1.0 if p.init == "ones" else 0.0
        views[p.name].copy_(torch.randn(p.shape, generator=g, device=DEV) * 0.02 + mean)
    return views, gpt.views(unit, torch.zeros(unit.numel, dtype=BF16, device=DEV))


def _ranks(comm, case, elems, g, symmetric):
    """One tensor of `elems` values per rank."""
    dt = _DTYPES[case["dtype"]]
    vals = [torch.randn(elems, generator=g, device=DEV).to(dt) for _ in range(case["world"])]
    if not symmetric:
        return vals
    sym = comm.empty(elems, dt)
    for s, v in zip(sym, vals):
        s.copy_(v)
    return sym


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    s = {"case": case}
    if kind in ("linear", "linear_gelu"):
        s["x"] = _normal(g, (case["tokens"], case["n_in"]))
        s["w"] = _normal(g, (case["n_out"], case["n_in"]), 0.02)
        s["b"] = _normal(g, (case["n_out"],), 0.02)
        if kind == "linear":
            s["dy"] = _normal(g, (case["tokens"], case["n_out"]), 1e-3)
    elif kind == "norm":
        rows, d = case["rows"], case["width"]
        s["x"], s["branch"] = _normal(g, (rows, d)), _normal(g, (rows, d))
        s["dy"], s["resid"] = _normal(g, (rows, d), 1e-3), _normal(g, (rows, d), 1e-3)
        s["w"], s["b"] = (_normal(g, (d,), 0.02) + 1.0), _normal(g, (d,), 0.02)
        s["gw"], s["gb"], s["sum"] = (torch.empty(d, dtype=BF16, device=DEV) for _ in range(3))
    elif kind == "head":
        s["x"] = _normal(g, (case["tokens"], case["width"]))
        s["targets"] = torch.randint(0, case["vocab"], (case["tokens"],), generator=g, device=DEV)
        s["p"], s["gr"] = _params(case, 0, g)
        s["loss"] = torch.zeros(1, device=DEV)
        s["bad"] = torch.zeros(1, dtype=torch.int32, device=DEV)
    elif kind == "optimizer":
        n = case["count"]
        s["master"] = torch.randn(n, generator=g, device=DEV) * 0.02
        s["m"] = torch.randn(n, generator=g, device=DEV) * 1e-4
        s["v"] = (torch.randn(n, generator=g, device=DEV) * 1e-3).square_()
        s["grad"] = _normal(g, (n,), 1e-3, _DTYPES[case["grad"]])
        s["param"] = s["master"].to(BF16)
        s["norm"] = torch.zeros(1, device=DEV)
    elif kind == "block":
        s["cfg"] = _config(case)
        s["p"], s["gr"] = _params(case, 1, g)
        t = case["batch"] * case["seq"]
        s["x"], s["dy"] = _normal(g, (t, case["width"])), _normal(g, (t, case["width"]), 1e-3)
    else:
        comm, n, world = _comm(case["world"]), case["count"], case["world"]
        s["comm"] = comm
        s["gid"], s["algo"] = comm.world_group.gid, sch.ALGO_IDS[case["algo"]]
        dt, sym = _DTYPES[case["dtype"]], case["symmetric"]
        if kind == "all_gather":
            s["ins"] = _ranks(comm, case, n, g, sym)
            s["outs"] = comm.empty(world * n, dt) if sym else [torch.empty(world * n, dtype=dt, device=DEV) for _ in range(world)]
        elif kind == "reduce_scatter":
            s["ins"] = _ranks(comm, case, world * n, g, sym)
            s["outs"] = [torch.empty(n, dtype=torch.float32, device=DEV) for _ in range(world)]
        else:
            s["outs"] = _ranks(comm, case, n, g, sym)
    return s


# ------------------------------------------------------------------------------------------ one pass
_LANES = 64      # what the tuning table gives these sizes; the communicator caps it where all ranks share one device


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "linear":
        y = gemm.linear(s["x"], s["w"], s["b"])
        dx = gemm.matmul_nn(s["dy"], s["w"])
        dw = gemm.matmul_tn(s["dy"], s["x"])
        return {"y": y, "dx": dx, "dw": dw}
    if kind == "linear_gelu":
        u, a = gemm.linear_gelu(s["x"], s["w"], s["b"])
        return {"u": u, "a": a}
    if kind == "norm":
        # the residual stream is summed in place into the branch; the backward reads it there
        y, mean, rstd = pccl._C.ln_fwd(s["x"], s["branch"], s["w"], s["b"], 1e-5)
        dx = pccl._C.ln_bwd(s["dy"], s["branch"], mean, rstd, s["w"], s["gw"], s["gb"], s["resid"], s["sum"])
        return {"y": y, "mean": mean, "rstd": rstd, "stream": s["branch"], "dx": dx, "gw": s["gw"], "gb": s["gb"], "sum": s["sum"]}
    if kind == "head":
        s["loss"].zero_()

        def ce(logits, targets, loss_sum, grad_scale):
            pccl._C.ce_fwd_bwd(logits, targets, loss_sum, grad_scale, -100, s["bad"])

        with torch.no_grad():
            dx = gpt.head_forward_backward(s["x"], s["targets"], s["p"], s["gr"], _config(case), 1.0 / case["tokens"], s["loss"], ce)
        return {"loss": s["loss"], "dx": dx, "wte": s["gr"]["wte"], "lnf_w": s["gr"]["lnf_w"], "lnf_b": s["gr"]["lnf_b"]}
    if kind == "optimizer":
        s["norm"].zero_()
        pccl._C.sq_norm(s["grad"], s["norm"])
        pccl._C.adamw(s["master"], s["m"], s["v"], s["grad"], s["param"], 1e-4, 0.9, 0.95, 1e-8, 0.1, 10, 1.0, 1.0, s["norm"])
        return {"norm": s["norm"], "master": s["master"], "m": s["m"], "v": s["v"], "param": s["param"]}
    if kind == "block":
        with torch.no_grad():
            y, ctx = gpt.layer_forward(s["x"], s["p"], s["cfg"], case["batch"])
            dx = gpt.layer_backward(s["dy"], ctx, s["p"], s["gr"], s["cfg"], case["batch"])
        return {"y": y, "dx": dx, "gr": s["gr"]}
    native = s["comm"].native
    if kind == "all_gather":
        native.all_gather(s["gid"], s["outs"], s["ins"], s["algo"], _LANES)
    elif kind == "reduce_scatter":
        native.reduce_scatter(s["gid"], s["outs"], s["ins"], s["algo"], _LANES, 1.0 / case["world"], None)
    else:
        native.all_reduce(s["gid"], s["outs"], s["algo"], _LANES, 1.0 / case["world"])
    return list(s["outs"])


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("linear", "linear_gelu"):
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        if kind == "linear_gelu":
            return {"bytes": 2 * (t * i + o * i + o + 2 * t * o), "flops": 2 * t * i * o}
        return {"bytes": 2 * (2 * t * i + 2 * o * i + o + 2 * t * o), "flops": 6 * t * i * o}
    if kind == "norm":
        # forward: two reads, two writes; backward: three reads (gradient, stream, residual gradient), one write
        return {"bytes": 2 * 8 * case["rows"] * case["width"], "flops": 0}
    if kind == "head":
        t, d, v = case["tokens"], case["width"], case["vocab"]
        return {"bytes": 2 * (2 * t * d + 2 * v * d), "flops": 6 * t * d * v}
    if kind == "optimizer":
        # the gradient is read for its norm and again for the update; three fp32 states in and out, the bf16 copy out
        return {"bytes": case["count"] * (2 * _DTYPES[case["grad"]].itemsize + 26), "flops": 0}
    if kind == "block":
        t, d, f = case["batch"] * case["seq"], case["width"], case["ff"]
        weights = 4 * d * d + 2 * d * f
        # three products per weight, and causal attention (half the square) with two products forward and four backward
        return {"bytes": 2 * (2 * weights + 4 * t * d), "flops": 6 * t * weights + 6 * t * case["seq"] * d}
    size, n, world = _DTYPES[case["dtype"]].itemsize, case["count"], case["world"]
    if kind == "all_gather":
        return {"bytes": world * n * size * (1 + world), "flops": 0}
    if kind == "reduce_scatter":
        return {"bytes": world * n * (world * size + 4), "flops": 0}
    return {"bytes": 2 * world * n * size, "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "all_gather":
        return "exact"
    if kind == "optimizer":
        # fp32 state; the order of the norm's partial sums is free, and it can move a bf16 weight over a rounding boundary
        return {"rel": 1e-4, "max": 1e-2}
    if kind in ("reduce_scatter", "all_reduce"):
        # one rounding to the type for the direct forms, one per hop where partial sums travel in 16 bits
        if case["dtype"] == "fp32":
            return {"rel": 1e-6, "max": 1e-5}
        return {"rel": 1e-2, "max": 5e-2}
    # bf16 results of fp32 sums: one rounding (2^-9) each way in single layers, several layers deep in the block and the head
    return {"rel": 1e-2, "max": 0.1} if kind in ("linear", "linear_gelu", "norm") else {"rel": 2e-2, "max": 0.5}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _norm64(x, w, b, eps=1e-5):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, eps)


def exact(case, seed):
    kind = case["kind"]
    if kind == "all_gather":
        return None
    s = prepare(case, seed)
    f = {k: v.double() for k, v in s.items() if isinstance(v, torch.Tensor) and v.is_floating_point()}
    if kind == "linear":
        return {"y": f["x"] @ f["w"].t() + f["b"], "dx": f["dy"] @ f["w"], "dw": f["dy"].t() @ f["x"]}
    if kind == "linear_gelu":
        u = f["x"] @ f["w"].t() + f["b"]
        return {"u": u, "a": torch.nn.functional.gelu(u, approximate="tanh")}
    if kind == "norm":
        # the stream is held in bf16; everything after it is taken from there
        v = (f["x"] + f["branch"]).to(BF16).double().requires_grad_()
        w, b = f["w"].requires_grad_(), f["b"].requires_grad_()
        y = _norm64(v, w, b)
        dx, gw, gb = torch.autograd.grad(y, (v, w, b), f["dy"])
        dx = dx + f["resid"]
        mean = v.detach().mean(1)
        rstd = (v.detach().var(1, unbiased=False) + 1e-5).rsqrt()
        return {"y": y, "mean": mean, "rstd": rstd, "stream": v, "dx": dx, "gw": gw, "gb": gb, "sum": dx.sum(0)}
    if kind == "head":
        p = {k: v.double().requires_grad_() for k, v in s["p"].items()}
        x = f["x"].requires_grad_()
        logits = _norm64(x, p["lnf_w"], p["lnf_b"]) @ p["wte"].t()
        loss = torch.nn.functional.cross_entropy(logits, s["targets"], reduction="sum")
        dx, wte, gw, gb = torch.autograd.grad(loss / case["tokens"], (x, p["wte"], p["lnf_w"], p["lnf_b"]))
        return {"loss": loss.detach().view(1), "dx": dx, "wte": wte, "lnf_w": gw, "lnf_b": gb}
    if kind == "optimizer":
        norm = f["grad"].square().sum().view(1)
        g = f["grad"] * torch.clamp(1.0 / (norm.sqrt() + 1e-6), max=1.0)
        m = 0.9 * f["m"] + 0.1 * g
        v = 0.95 * f["v"] + 0.05 * g * g
        step = (m / (1 - 0.9 ** 10)) / ((v / (1 - 0.95 ** 10)).sqrt() + 1e-8)
        master = f["master"] * (1 - 1e-4 * 0.1) - 1e-4 * step
        return {"norm": norm, "master": master, "m": m, "v": v, "param": master}
    if kind == "block":
        p = {k: v.double().requires_grad_() for k, v in s["p"].items()}
        x, lin = f["x"].requires_grad_(), torch.nn.functional.linear
        b, t, d, h = case["batch"], case["seq"], case["width"], case["heads"]
        qkv = lin(_norm64(x, p["ln1_w"], p["ln1_b"]), p["qkv_w"], p["qkv_b"]).view(b, t, 3, h, d // h)
        q, k, v = (z.transpose(1, 2) for z in qkv.unbind(2))
        score = (q @ k.transpose(-1, -2)) / math.sqrt(d // h)
        mask = torch.ones(t, t, dtype=torch.bool, device=DEV).triu(1)
        a = (score.masked_fill(mask, float("-inf")).softmax(-1) @ v).transpose(1, 2).reshape(b * t, d)
        x2 = x + lin(a, p["proj_w"], p["proj_b"])
        u = lin(_norm64(x2, p["ln2_w"], p["ln2_b"]), p["fc1_w"], p["fc1_b"])
        y = x2 + lin(torch.nn.functional.gelu(u, approximate="tanh"), p["fc2_w"], p["fc2_b"])
        names = list(p)
        grads = torch.autograd.grad(y, [x] + [p[n] for n in names], f["dy"])
        return {"y": y, "dx": grads[0], "gr": dict(zip(names, grads[1:]))}
    n, world = case["count"], case["world"]
    tensors = s["ins"] if kind == "reduce_scatter" else s["outs"]
    total = sum(t.double() for t in tensors) / world
    return [total[r * n:(r + 1) * n].clone() for r in range(world)] if kind == "reduce_scatter" else [total] * world
