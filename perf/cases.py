"""The work a program has this library do on one GPU, as cases that can be timed and compared.

The collectives run on ``mintccl_b200.emulated(n)``: n ranks on one GPU, the kernels of the multi-GPU paths in one
cooperative launch, so "peer" memory is this GPU's own and the floor is the HBM.  The compute ops are what one rank of
a tensor-parallel Llama-3-8B MLP (hidden 4096, ffn 14336, TP = 8) does, plus the fused kernels on two emulated ranks.
"""
from __future__ import annotations

import math

import torch

import mintccl_b200
from mintccl_b200 import Config
from mintccl_b200.ops import mxfp8 as mx
from mintccl_b200.ops.gemm import AllGatherGemm, GemmReduceScatter, gemm
from mintccl_b200.parallel.rendezvous import SingleControl

_DT = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
_SIZE = {"fp32": 4, "fp16": 2, "bf16": 2}
_MIB = 1 << 20


def listed():
    return [
        # the 8-byte all-reduce: a loss or a flag; latency and nothing else
        {"name": "allreduce_8B", "kind": "allreduce", "n": 8, "dtype": "fp32", "numel": 2},
        # one gradient bucket of data-parallel training
        {"name": "allreduce_bf16_64MiB", "kind": "allreduce", "n": 8, "dtype": "bf16", "numel": 32 * _MIB},
        # shards whose size is no multiple of a vector (unpadded parameter shards)
        {"name": "allgather_fp16_ragged", "kind": "allgather", "n": 4, "dtype": "fp16", "numel": 1_000_003},
        # 16-bit gradients summed into fp32 shards for a sharded optimiser
        {"name": "reducescatter_bf16_to_fp32", "kind": "reducescatter", "n": 8, "dtype": "bf16", "out": "fp32",
         "numel": 1_048_576},
        # parameters sent out from rank 0 and a metric buffer summed on it: 64 MiB fp16 each
        {"name": "broadcast_reduce_fp16_64MiB", "kind": "rooted", "n": 8, "dtype": "fp16", "numel": 32 * _MIB},
        # pipeline activations forwarded over ring neighbours, rank 0 -> 4 through 1, 2, 3
        {"name": "multihop_ll128_16MiB", "kind": "multihop", "n": 8, "hops": 4, "proto": "ll128", "nbytes": 16 * _MIB},
        # block-scaled fp8 gradients
        {"name": "mxfp8_allreduce_16Mi", "kind": "mxfp8_allreduce", "n": 8, "numel": 16 * _MIB},
        # a linear layer in MXFP8: activations are quantised on the way in, weights are quantised and tiled once
        {"name": "mxfp8_linear_8192", "kind": "mxfp8_linear", "m": 8192, "nn": 1792, "k": 4096},
        # the up projection of a prefill or training step
        {"name": "gemm_8192x1792x4096", "kind": "gemm", "m": 8192, "nn": 1792, "k": 4096},
        # the down projection of a decode step with a batch of 128
        {"name": "gemm_128x4096x1792", "kind": "gemm", "m": 128, "nn": 4096, "k": 1792},
        # one training step of the MLP block: forward and backward
        {"name": "mlp_train_8192", "kind": "mlp", "tokens": 8192, "hidden": 4096, "ffn": 1792, "train": True},
        # forward of the MLP block on two ranks: all-gather -> GEMM, activation, GEMM -> reduce-scatter
        {"name": "fused_tp2_4096", "kind": "fused_tp", "n": 2, "tokens": 4096, "hidden": 4096, "ffn": 1792},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mult(rng, lo, hi, step):
    return max(lo, min(hi, _log(rng, lo, hi) // step * step))


def draw(rng):
    kind = rng.choice(["allreduce", "allgather", "reducescatter", "rooted", "multihop", "mxfp8_allreduce", "mxfp8_linear",
                       "gemm", "mlp", "fused_tp"])
    n = rng.choice([2, 4, 8])
    dtype = rng.choice(["fp32", "fp16", "bf16"])
    most = 64 * _MIB // _SIZE[dtype]
    if kind == "allreduce":
        return {"kind": kind, "n": n, "dtype": dtype, "numel": _log(rng, 2, most)}
    if kind == "allgather":
        return {"kind": kind, "n": n, "dtype": dtype, "numel": _log(rng, 1000, 1_000_003)}
    if kind == "reducescatter":
        numel = _log(rng, 1000, 1_048_576)
        return {"kind": kind, "n": n, "dtype": dtype, "numel": numel,
                "out": rng.choice([dtype, "fp32" if dtype != "fp32" else "bf16"])}
    if kind == "rooted":
        return {"kind": kind, "n": n, "dtype": dtype, "numel": _log(rng, 1000, most)}
    if kind == "multihop":
        return {"kind": kind, "n": 8, "hops": rng.choice([1, 2, 4, 7]), "proto": rng.choice(["ll128", "auto"]),
                "nbytes": _log(rng, 4096, 16 * _MIB)}
    if kind == "mxfp8_allreduce":
        return {"kind": kind, "n": n, "numel": _mult(rng, 8192, 16 * _MIB, 32)}
    if kind == "fused_tp":
        return {"kind": kind, "n": 2, "tokens": _mult(rng, 256, 4096, 256), "hidden": _mult(rng, 512, 4096, 256),
                "ffn": _mult(rng, 512, 1792, 256)}
    m = _mult(rng, 128, 8192, 128)
    if kind == "mlp":
        return {"kind": kind, "tokens": m, "hidden": _mult(rng, 512, 4096, 256), "ffn": _mult(rng, 512, 1792, 256),
                "train": rng.random() < 0.6}
    nn, k = _mult(rng, 256, 14336, 256), _mult(rng, 256, 8192, 128)
    while m * nn * k > 2 * 8192 * 1792 * 4096:
        m = max(128, m // 256 * 128)
    return {"kind": kind, "m": m, "nn": nn, "k": k}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, shape, dtype, scale=1.0):
    return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * scale).to(dtype)


def _ranks(c, seed):
    """The contributions of all ranks of a collective."""
    g = _gen(seed)
    shape = (c["n"], c["numel"]) if c["kind"] == "reducescatter" else (c["numel"],)
    return [_randn(g, shape, _DT[c["dtype"]]) for _ in range(c["n"])]


def _world(n, user_bytes):
    cfg = Config.from_env(max_channels=16, num_blocks=16, buff_size=1 << 20, scratch_bytes=1 << 20, wait_timeout_ms=3000,
                          heap_bytes=(32 + 26 * n) * _MIB + user_bytes)
    return mintccl_b200.emulated(n, 0, cfg)


def _symm_empty(w, shape, dtype):
    """Heap tensors that keep their world: the heap goes with it, and results outlive the state they came from."""
    ts = w.symm_empty(shape, dtype)
    for t in ts:
        t.world = w
    return ts


def _symm(w, values):
    ts = _symm_empty(w, tuple(values[0].shape), values[0].dtype)
    for t, v in zip(ts, values):
        t.copy_(v)
    return ts


def _linear_inputs(c, seed):
    g = _gen(seed)
    return _randn(g, (c["m"], c["k"]), torch.bfloat16), _randn(g, (c["nn"], c["k"]), torch.bfloat16, 0.02)


def _mlp_inputs(c, seed):
    g = _gen(seed)
    t, h, f = c["tokens"], c["hidden"], c["ffn"]
    return (_randn(g, (t, h), torch.bfloat16), _randn(g, (f, h), torch.bfloat16, 0.02),
            _randn(g, (h, f), torch.bfloat16, 0.02), _randn(g, (t, h), torch.bfloat16))


def _tp_inputs(c, seed):
    g = _gen(seed)
    n, t, h, f = c["n"], c["tokens"], c["hidden"], c["ffn"]
    return ([_randn(g, (t // n, h), torch.bfloat16) for _ in range(n)], [_randn(g, (f, h), torch.bfloat16, 0.02) for _ in range(n)],
            [_randn(g, (h, f), torch.bfloat16, 0.02) for _ in range(n)])


def _mx_inputs(c, seed):
    g = _gen(seed)
    return [torch.randn(c["numel"], generator=g, device="cuda") for _ in range(c["n"])]


def prepare(case, seed):
    c, k, n = case, case["kind"], case.get("n", 1)
    s = {"c": c}
    if k in ("allreduce", "allgather", "reducescatter", "rooted"):
        xs = _ranks(c, seed)
        dt = xs[0].dtype
        one = xs[0].numel() * xs[0].element_size()
        w = s["w"] = _world(n, (n + 1) * one + _MIB if k == "allgather" else 3 * one + _MIB)
        s["x"] = _symm(w, xs)
        if k == "allreduce":
            s["out"] = _symm_empty(w, (c["numel"],), dt)
        elif k == "allgather":
            s["out"] = _symm_empty(w, (n, c["numel"]), dt)
        elif k == "reducescatter":
            s["out"] = [torch.empty(c["numel"], dtype=_DT[c["out"]], device="cuda") for _ in range(n)]
        else:
            s["y"], s["out"] = _symm(w, xs), _symm_empty(w, (c["numel"],), dt)
    elif k == "multihop":
        s["w"] = _world(n, 0)
        g = _gen(seed)
        s["src"] = [torch.randint(0, 256, (c["nbytes"],), generator=g, device="cuda", dtype=torch.uint8)] * n
        s["dst"] = [torch.zeros(c["nbytes"], device="cuda", dtype=torch.uint8) for _ in range(n)]
    elif k == "mxfp8_allreduce":
        w = s["w"] = _world(n, 3 * c["numel"] + 4 * _MIB)
        q = [mx.quantize_mxfp8(x) for x in _mx_inputs(c, seed)]
        s["d"], s["s"] = _symm(w, [a for a, _ in q]), _symm(w, [b for _, b in q])
        s["od"], s["os"] = _symm_empty(w, (c["numel"],), torch.uint8), _symm_empty(w, (c["numel"] // 32,), torch.uint8)
    elif k == "mxfp8_linear":
        s["x"], w = _linear_inputs(c, seed)
        s["wd"], ws = mx.quantize_rows_mxfp8(w)
        s["ws"] = mx.tile_scales(ws)
    elif k == "gemm":
        s["x"], s["w"] = _linear_inputs(c, seed)
    elif k == "mlp":
        x, up, down, dy = _mlp_inputs(c, seed)
        t, h, f = c["tokens"], c["hidden"], c["ffn"]
        from mintccl_b200.models.tp_mlp import TensorParallelMLP
        cfg = Config.from_env(max_channels=2, num_blocks=2, buff_size=1 << 20, scratch_bytes=1 << 20, wait_timeout_ms=4000,
                              heap_bytes=64 * _MIB + 12 * t * h)
        comm = s["w"] = mintccl_b200.Communicator(control=SingleControl(), device=0, config=cfg)
        mlp = s["mlp"] = TensorParallelMLP(comm, t, h, f)
        with torch.no_grad():
            mlp.w_up.copy_(up)
            mlp.w_down.copy_(down)
        s["x"], s["dy"] = x.requires_grad_(c["train"]), dy
    elif k == "fused_tp":
        t, h, f = c["tokens"], c["hidden"], c["ffn"]
        w = s["w"] = _world(n, 2 * t * h + 4 * t * h + 4 * _MIB)
        s["x"], s["up"], s["down"] = _tp_inputs(c, seed)
        s["ag"], s["rs"] = AllGatherGemm(w, t, f, h), GemmReduceScatter(w, t, h, f)
    else:
        raise ValueError(k)
    return s


def run(s):
    c = s["c"]
    k = c["kind"]
    if k == "allreduce":
        s["w"].allreduce(s["x"], out=s["out"])
        return s["out"]
    if k == "allgather":
        s["w"].allgather(s["out"], inp=s["x"])
        return s["out"]
    if k == "reducescatter":
        s["w"].reducescatter(s["x"], out=s["out"])
        return s["out"]
    if k == "rooted":
        s["w"].broadcast(s["x"], root=0)
        s["w"].reduce(s["y"], root=0, out=s["out"])
        return {"broadcast": s["x"], "reduce": s["out"][0]}
    if k == "multihop":
        s["w"].sendrecv_route(list(range(c["hops"] + 1)), s["src"], s["dst"], proto=None if c["proto"] == "auto" else c["proto"])
        return s["dst"][c["hops"]]
    if k == "mxfp8_allreduce":
        mx.allreduce_mxfp8(s["w"], s["d"], s["s"], s["od"], s["os"])
        return s["od"], s["os"]
    if k == "mxfp8_linear":
        xd, xs = mx.quantize_rows_mxfp8(s["x"])
        y = mx.gemm_mxfp8(xd, mx.tile_scales(xs), s["wd"], s["ws"], scales_tiled=True)
        return {"payload": xd, "scale": xs, "y": y}
    if k == "gemm":
        return gemm(s["x"], s["w"])
    if k == "mlp":
        mlp = s["mlp"]
        if not c["train"]:
            with torch.no_grad():
                return mlp(s["x"])
        y = mlp(s["x"])
        return (y.detach(), *torch.autograd.grad(y, [s["x"], mlp.w_up, mlp.w_down], s["dy"]))
    hs = s["ag"](s["x"], s["up"])
    ys = s["rs"]([torch.nn.functional.silu(h) for h in hs], s["down"])
    return {"h": hs, "y": ys}


def work(case):
    c, k, n = case, case["kind"], case.get("n", 1)
    if k == "allreduce":
        b = c["numel"] * _SIZE[c["dtype"]]
        return {"bytes": 2 * n * b, "flops": (n - 1) * c["numel"]}
    if k == "allgather":
        b = c["numel"] * _SIZE[c["dtype"]]
        return {"bytes": n * b + n * n * b, "flops": 0}
    if k == "reducescatter":
        return {"bytes": n * n * c["numel"] * _SIZE[c["dtype"]] + n * c["numel"] * _SIZE[c["out"]], "flops": n * (n - 1) * c["numel"]}
    if k == "rooted":
        b = c["numel"] * _SIZE[c["dtype"]]
        return {"bytes": n * b + (n + 1) * b, "flops": (n - 1) * c["numel"]}
    if k == "multihop":
        return {"bytes": 2 * c["nbytes"], "flops": 0}
    if k == "mxfp8_allreduce":
        return {"bytes": 2 * n * c["numel"] * 33 / 32, "flops": 2 * n * c["numel"]}
    if k == "fused_tp":
        t, h, f = c["tokens"], c["hidden"], c["ffn"]
        return {"bytes": 2 * (2 * t * h + n * (2 * t * f + 2 * f * h)), "flops": 4.0 * n * t * h * f}
    if k == "mlp":
        t, h, f = c["tokens"], c["hidden"], c["ffn"]
        if not c["train"]:
            return {"bytes": 2 * (2 * t * h + 2 * h * f), "flops": 4.0 * t * h * f}
        return {"bytes": 2 * (4 * t * h + 4 * h * f), "flops": 12.0 * t * h * f}
    m, nn, kk = c["m"], c["nn"], c["k"]
    if k == "mxfp8_linear":
        return {"bytes": 2 * m * kk + (m + nn) * kk * 33 / 32 + 2 * m * nn, "flops": 2.0 * m * nn * kk}
    return {"bytes": 2 * (m * kk + nn * kk + m * nn), "flops": 2.0 * m * nn * kk}


def tolerance(case):
    k = case["kind"]
    if k in ("allgather", "multihop", "mxfp8_allreduce"):
        return "exact"
    if k in ("allreduce", "reducescatter", "rooted"):
        # sums in fp32; one or two roundings into the output type
        out = case.get("out", case["dtype"])
        return {"rel": {"fp32": 1e-6, "fp16": 1e-3, "bf16": 8e-3}[out]}
    if k in ("gemm", "mxfp8_linear"):
        return {"rel": 7e-3, "differ": 0.0}     # one rounding into bf16; the quantised bytes are the same
    return {"rel": 1.5e-2}                      # bf16 intermediates feed the next product


def _exact_mx(x):
    """MXFP8 quantisation and its value in 64 bits: blocks of 32 along the last dimension."""
    b = x.double().reshape(-1, 32)
    amax = b.abs().amax(1)
    m, e = torch.frexp(amax)
    p = (e - 9 + (m * 2 > 1.75).to(e.dtype)).clamp(-126, 127).double()
    p = torch.where(amax > 0, p, torch.full_like(p, -8.0))
    q = torch.ldexp(b, -p[:, None]).float().to(torch.float8_e4m3fn)
    return torch.ldexp(q.double(), p[:, None]).reshape(x.shape)


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("multihop", "mxfp8_allreduce"):
        return None
    if k in ("allreduce", "allgather", "reducescatter", "rooted"):
        xs = _ranks(c, seed)
        if k == "allgather":
            return [torch.stack(xs).double()] * c["n"]
        total = sum(x.double() for x in xs)
        if k == "reducescatter":
            return [total[r] for r in range(c["n"])]
        if k == "allreduce":
            return [total] * c["n"]
        return {"broadcast": [xs[0].double()] * c["n"], "reduce": total}
    if k in ("gemm", "mxfp8_linear"):
        x, w = _linear_inputs(c, seed)
        if k == "gemm":
            return x.double() @ w.double().t()
        return {"payload": None, "scale": None, "y": _exact_mx(x) @ _exact_mx(w).t()}
    if k == "mlp":
        x, up, down, dy = (t.double() for t in _mlp_inputs(c, seed))
        h = x @ up.t()
        sig = torch.sigmoid(h)
        a = h * sig
        y = a @ down.t()
        if not c["train"]:
            return y
        dh = (dy @ down) * (sig * (1 + h * (1 - sig)))
        return y, dh @ up, dh.t() @ x, dy.t() @ a
    xs, ups, downs = _tp_inputs(c, seed)
    x = torch.cat(xs).double()
    hs = [x @ u.double().t() for u in ups]
    y = sum((h * torch.sigmoid(h)) @ d.double().t() for h, d in zip(hs, downs))
    return {"h": hs, "y": list(y.chunk(c["n"]))}
