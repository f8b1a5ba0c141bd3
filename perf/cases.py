"""What a program that uses this framework on one GPU has it do, as measurable cases.

A case is a dict of plain values; ``kind`` says which part of the framework it goes through:

    collective   ``Communicator``: all-reduce, all-gather, reduce-scatter, all-to-all, broadcast
    moe          ``ExpertParallel``: dispatch of a batch of tokens to experts and combine of their rows
    linear       ``TensorParallel.gemm``: bf16 linear layer
    linear_fp8   ``TensorParallel.quantize_fp8`` + ``gemm_fp8``: block-scaled e4m3 linear layer
    ar_rmsnorm   ``DeviceComm.ar_rmsnorm``: all-reduce, residual add and RMSNorm in one kernel
    train        ``FSDPEngine.step``: one ZeRO-3 training step (forward, backward, optimizer)

The communicator has one rank, so the cases cover what each rank does on its own GPU: the same calls, kernels and
buffers as with more ranks, without the traffic between GPUs.
"""
import math

import torch

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16, "i32": torch.int32, "u8": torch.uint8, "f64": torch.float64}
E4M3_MAX = 448.0


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a scalar-like statistic reduced between steps: the smallest call, where only the call itself costs anything
        {"name": "allreduce_small", "kind": "collective", "func": "all_reduce", "dtype": "f32", "count": 1013, "op": "sum", "send_off": 0, "recv_off": 0},
        # a large bf16 message, the end of the size sweep that bandwidth is quoted on
        {"name": "allreduce_large", "kind": "collective", "func": "all_reduce", "dtype": "bf16", "count": 1 << 28, "op": "sum", "send_off": 0, "recv_off": 0},
        # gradients averaged by a pre-multiplied sum, a bucket with a ragged end
        {"name": "reduce_scatter_premul", "kind": "collective", "func": "reduce_scatter", "dtype": "bf16", "count": 12582917, "op": "premul", "send_off": 0, "recv_off": 0},
        # a parameter gathered into its place inside a flat buffer: neither end is aligned to anything but its type
        {"name": "allgather_view", "kind": "collective", "func": "all_gather", "dtype": "bf16", "count": 16777259, "op": "sum", "send_off": 3, "recv_off": 7},
        # decoding: few tokens, fp8 payload, experts of one GPU out of a large mixture
        {"name": "moe_decode_fp8", "kind": "moe", "layout": "expert_major", "fp8": True, "tokens": 64, "max_tokens": 64, "hidden": 7168, "experts": 32, "topk": 8, "drop": 0.0},
        # prefill: a full batch, bf16 payload, one row per selected expert
        {"name": "moe_prefill_bf16", "kind": "moe", "layout": "expert_major", "fp8": False, "tokens": 4096, "max_tokens": 4096, "hidden": 7168, "experts": 32, "topk": 8, "drop": 0.0},
        # one copy of a token per rank, fp8 payload, the token count below the capacity, some entries unused
        {"name": "moe_rank_major_fp8", "kind": "moe", "layout": "rank_major", "fp8": True, "tokens": 2000, "max_tokens": 2048, "hidden": 4096, "experts": 64, "topk": 6, "drop": 0.05},
        # a linear layer while decoding: one row block, the weights are the traffic
        {"name": "linear_decode", "kind": "linear", "m": 128, "n": 8192, "k": 8192},
        # a linear layer while prefilling or training: this rank's share of a large layer
        {"name": "linear_prefill", "kind": "linear", "m": 8192, "n": 8192, "k": 3584},
        # the same with activations quantised on the way, weights quantised once; a row count that does not split into large tiles
        {"name": "linear_fp8", "kind": "linear_fp8", "m": 1920, "n": 4096, "k": 7168},
        # the seam between two tensor-parallel layers of a decoder
        {"name": "ar_rmsnorm", "kind": "ar_rmsnorm", "tokens": 2048, "hidden": 8192, "mode": 0},
        # a training step of a two-layer model with the layer shape of the 8B configuration
        {"name": "train_step", "kind": "train", "layers": 2, "hidden": 4096, "heads": 32, "kv_heads": 8, "ffn": 14336, "vocab": 16384, "batch": 1, "seq": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["collective", "collective", "collective", "moe", "moe", "moe", "linear", "linear", "linear_fp8", "linear_fp8", "ar_rmsnorm", "train"])
    if kind == "collective":
        dtype = rng.choice(["f32", "bf16", "bf16", "f16", "i32", "u8", "f64"])
        func = rng.choice(["all_reduce", "reduce_scatter", "all_gather", "all_to_all", "broadcast"])
        op = rng.choice(["sum", "avg", "premul", "premul"]) if func in ("all_reduce", "reduce_scatter") and dtype in ("f32", "bf16", "f16", "f64") else "sum"
        size = DTYPES[dtype].itemsize
        return {"kind": kind, "func": func, "dtype": dtype, "count": _log(rng, 1, (1 << 27) // size), "op": op,
                "send_off": rng.choice([0, 0, rng.randrange(16)]), "recv_off": rng.choice([0, 0, rng.randrange(16)])}
    if kind == "moe":
        experts = rng.choice([8, 16, 32, 48, 64, 128, 256])
        layout, fp8 = rng.choice(["expert_major", "expert_major", "rank_major"]), rng.random() < 0.5
        # a decoding batch where the rows of the whole capacity are scaled back, else up to a prefill batch
        tokens = _log(rng, 1, 128 if fp8 and layout == "expert_major" else min(4096, 131072 // experts))
        return {"kind": kind, "layout": layout, "fp8": fp8, "tokens": tokens,
                "max_tokens": tokens + rng.choice([0, 0, rng.randrange(1 + tokens // 4)]), "hidden": 128 * rng.randint(8, 56), "experts": experts,
                "topk": rng.randint(1, 8), "drop": rng.choice([0.0, 0.0, 0.1])}
    if kind == "linear":
        return {"kind": kind, "m": 128 * _log(rng, 1, 64), "n": 256 * _log(rng, 4, 32), "k": 64 * _log(rng, 8, 112)}
    if kind == "linear_fp8":
        return {"kind": kind, "m": 128 * _log(rng, 1, 64), "n": 256 * _log(rng, 4, 32), "k": 128 * _log(rng, 4, 56)}
    if kind == "ar_rmsnorm":
        return {"kind": kind, "tokens": _log(rng, 1, 4096), "hidden": 8 * _log(rng, 64, 1024), "mode": rng.choice([0, 0, 2])}
    heads = rng.choice([4, 8, 16])
    return {"kind": kind, "layers": rng.randint(1, 3), "hidden": 128 * heads, "heads": heads, "kv_heads": rng.choice([2, 4]), "ffn": 256 * rng.randint(4, 28),
            "vocab": 1024 * rng.randint(2, 16), "batch": rng.randint(1, 2), "seq": _log(rng, 65, 1024)}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _values(count, dtype, gen):
    t = DTYPES[dtype]
    if t == torch.uint8:
        return torch.randint(0, 256, (count,), dtype=t, device="cuda", generator=gen)
    if t == torch.int32:
        return torch.randint(-(1 << 20), 1 << 20, (count,), dtype=t, device="cuda", generator=gen)
    return torch.randn(count, device="cuda", dtype=torch.float64 if t == torch.float64 else torch.float32, generator=gen).to(t)


def _collective_inputs(c, seed):
    return _values(c["count"], c["dtype"], _gen(seed))


def _scale(c, seed):
    return 0.25 + 0.0625 * (seed % 8)   # a factor that every floating type holds exactly


def _moe_inputs(c, seed):
    """Tokens like normalised hidden states; routing by the top-k of logits with popular and unpopular experts."""
    g = _gen(seed)
    T, H, E, K = c["tokens"], c["hidden"], c["experts"], c["topk"]
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    logits = torch.randn(T, E, device="cuda", generator=g) + 0.5 * torch.randn(1, E, device="cuda", generator=g)
    top = logits.topk(K, dim=1)
    w = torch.softmax(top.values, dim=1).contiguous()
    idx = top.indices.long()
    if c["drop"]:
        idx = torch.where(torch.rand(T, K, device="cuda", generator=g) < c["drop"], torch.full_like(idx, -1), idx)
    y = torch.randn(1, c["max_tokens"], H, device="cuda", generator=g).bfloat16() if c["layout"] == "rank_major" else None
    return x, idx.contiguous(), w, y


def _linear_inputs(c, seed):
    g = _gen(seed)
    x = torch.randn(c["m"], c["k"], device="cuda", generator=g).bfloat16()
    w = (torch.randn(c["n"], c["k"], device="cuda", generator=g) / math.sqrt(c["k"])).bfloat16()
    return x, w


def _rmsnorm_inputs(c, seed):
    g = _gen(seed)
    t, h = c["tokens"], c["hidden"]
    partial = torch.randn(t, h, device="cuda", generator=g).bfloat16()
    residual = (2 * torch.randn(t, h, device="cuda", generator=g)).bfloat16()
    weight = (1 + 0.1 * torch.randn(h, device="cuda", generator=g)).bfloat16()
    return partial, residual, weight


def _train_shapes(c):
    h, kv, f = c["hidden"], c["kv_heads"] * (c["hidden"] // c["heads"]), c["ffn"]
    layer = [("norm1", (h,)), ("wq", (h, h)), ("wk", (kv, h)), ("wv", (kv, h)), ("wo", (h, h)), ("norm2", (h,)), ("w_gate", (f, h)), ("w_up", (f, h)), ("w_down", (h, f))]
    return [[("tok", (c["vocab"], h))]] + [layer] * c["layers"] + [[("norm", (h,)), ("out", (c["vocab"], h))]]


def _train_inputs(c, seed):
    """Weights of every unit as one flat bf16 vector, and a batch of token ids in pinned host memory."""
    g = _gen(seed)
    flats = [torch.cat([torch.ones(s, device="cuda") if len(s) == 1 else 0.02 * torch.randn(math.prod(s), device="cuda", generator=g) for _, s in shapes]).bfloat16()
             for shapes in _train_shapes(c)]
    hg = torch.Generator().manual_seed(int(seed) + 5)
    ids = torch.randint(0, c["vocab"], (c["batch"], c["seq"] + 1), generator=hg)
    return flats, ids[:, :-1].contiguous().pin_memory(), ids[:, 1:].contiguous().pin_memory()


# ------------------------------------------------------------------------------------------------ state
class _Owned(dict):
    """A state that gives back what the framework allocated for it when it goes."""
    close = None

    def __del__(self):
        if self.close is not None:
            self.close()


class _Outputs(dict):
    """Outputs that lie in memory of a state: they keep the state (and with it that memory) alive."""

    def __init__(self, owner, **outputs):
        super().__init__(**outputs)
        self.owner = owner


_process = {}


def _comm():
    if "comm" not in _process:
        from nccl_b200 import Communicator, get_unique_id
        torch.cuda.set_device(0)
        _process["comm"] = Communicator(1, 0, get_unique_id())
    return _process["comm"]


def _tp():
    if "tp" not in _process:
        from nccl_b200.ops.tp import TensorParallel
        _process["tp"] = TensorParallel(_comm(), 8192, 8192)
    return _process["tp"]


def prepare(case, seed):
    c, s = case, _Owned()
    s["case"] = c
    kind = c["kind"]
    if kind == "collective":
        from nccl_b200.core import BF16, FP16, FP32, FP64
        s["comm"] = _comm()
        x = _collective_inputs(c, seed)
        s["send"] = torch.empty(c["count"] + c["send_off"], dtype=x.dtype, device="cuda")[c["send_off"]:].copy_(x)
        s["recv"] = torch.zeros(c["count"] + c["recv_off"], dtype=x.dtype, device="cuda")[c["recv_off"]:]
        s["op"] = c["op"]
        if c["op"] == "premul":
            code = {"f32": FP32, "bf16": BF16, "f16": FP16, "f64": FP64}[c["dtype"]]
            comm, op = s["comm"], s["comm"].premul_sum(_scale(c, seed), code)
            s["op"], s.close = op, lambda: comm.destroy_op(op)
    elif kind == "moe":
        from nccl_b200.ops.ep import ExpertParallel
        s["x"], s["idx"], s["w"], s["y"] = _moe_inputs(c, seed)
        ep = s["ep"] = ExpertParallel(_comm(), c["experts"], c["max_tokens"], c["hidden"], layout=c["layout"])
        lead = (ep.El, ep.cap) if c["layout"] == "expert_major" else (1, c["max_tokens"])
        s["toks"] = torch.zeros(*lead, c["hidden"], dtype=torch.uint8 if c["fp8"] else torch.bfloat16, device="cuda")
        s["scales"] = torch.zeros(*lead, c["hidden"] // 128, device="cuda") if c["fp8"] else None
        s["counts"] = torch.zeros(ep.El, dtype=torch.int32, device="cuda")
        s["out"] = torch.empty(c["tokens"], c["hidden"], dtype=torch.bfloat16, device="cuda")
        s.close = ep.destroy
    elif kind == "linear":
        s["tp"] = _tp()
        s["x"], s["w"] = _linear_inputs(c, seed)
    elif kind == "linear_fp8":
        s["tp"] = _tp()
        s["x"], w = _linear_inputs(c, seed)
        s["wq"], s["ws"] = s["tp"].quantize_fp8(w, 128)
    elif kind == "ar_rmsnorm":
        from nccl_b200.ops.devapi import DeviceComm
        dc = s["dc"] = DeviceComm(_comm())
        partial, residual, s["weight"] = _rmsnorm_inputs(c, seed)
        for name in ("partial", "residual", "out"):
            s[name] = dc.symmetric(partial.numel(), torch.bfloat16).view(partial.shape)
        s["partial"].copy_(partial)
        s["residual"].copy_(residual)
        s.close = dc.destroy
    else:
        from nccl_b200.models.llama import LlamaConfig
        from nccl_b200.parallel.fsdp import FSDPEngine
        cfg = LlamaConfig(layers=c["layers"], hidden=c["hidden"], heads=c["heads"], kv_heads=c["kv_heads"], ffn=c["ffn"], vocab=c["vocab"])
        eng = s["engine"] = FSDPEngine(_comm(), cfg, device="cuda", seed=0, lr=1e-4, init_on_device=True)
        flats, s["tokens"], s["targets"] = _train_inputs(c, seed)
        for u, f in zip(eng.units, flats):   # the weights of a checkpoint
            u.param[:f.numel()].copy_(f)
            u.master[:f.numel()].copy_(f)
        s.close = eng.close
    return s


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "collective":
        comm, f = s["comm"], c["func"]
        if f == "all_reduce":
            return comm.all_reduce(s["send"], s["recv"], op=s["op"])
        if f == "reduce_scatter":
            return comm.reduce_scatter(s["send"], s["recv"], op=s["op"])
        if f == "all_gather":
            return comm.all_gather(s["send"], s["recv"])
        if f == "all_to_all":
            return comm.all_to_all(s["send"], s["recv"])
        return comm.broadcast(s["send"], s["recv"], 0)
    if kind == "moe":
        ep = s["ep"]
        toks, scales, counts = ep.dispatch(s["x"], s["idx"], s["w"], fp8=c["fp8"], toks=s["toks"], scales=s["scales"], counts=s["counts"])
        if c["layout"] == "rank_major":
            # the caller's experts give one row per received token
            out = ep.combine(s["y"], out=s["out"])
            return {"out": out, "counts": counts, "toks": toks, "scales": scales, "recv_idx": ep.recv_topk_idx, "recv_w": ep.recv_topk_weights} if c["fp8"] else \
                {"out": out, "counts": counts, "toks": toks, "recv_idx": ep.recv_topk_idx, "recv_w": ep.recv_topk_weights}
        # the order of the rows of one expert is not defined, so what stands for the experts keeps each row's value
        # (identity); with an fp8 payload that means to scale the rows back
        y = toks
        if c["fp8"]:
            y = toks.view(torch.float8_e4m3fn).to(torch.bfloat16)
            y.view(ep.El, ep.cap, -1, 128).mul_(scales.to(torch.bfloat16).unsqueeze(-1))
        return {"out": ep.combine(y, out=s["out"]), "counts": counts}
    if kind == "linear":
        return s["tp"].gemm(s["x"], s["w"])
    if kind == "linear_fp8":
        q, scales = s["tp"].quantize_fp8(s["x"])
        return {"out": s["tp"].gemm_fp8(q, scales, s["wq"], s["ws"]), "q": q.view(torch.uint8), "scales": scales}
    if kind == "ar_rmsnorm":
        s["dc"].ar_rmsnorm(s["partial"], s["residual"], s["out"], s["weight"], mode=c["mode"])
        return _Outputs(s, out=s["out"], residual=s["residual"])
    loss = s["engine"].step(s["tokens"], s["targets"])
    return _Outputs(s, loss=loss, units=[{"param": u.param, "master": u.master, "m": u.m, "v": u.v} for u in s["engine"].units])


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c, kind = case, case["kind"]
    if kind == "collective":
        return {"bytes": 2 * c["count"] * DTYPES[c["dtype"]].itemsize, "flops": c["count"] if c["op"] == "premul" else 0}
    if kind == "moe":
        T, H, K = c["tokens"], c["hidden"], c["topk"]
        payload = H + H // 128 * 4 if c["fp8"] else 2 * H
        routing = T * K * 12
        if c["layout"] == "rank_major":
            # tokens in, one payload row out per token, the experts' rows in, the result out, the routing rows out
            return {"bytes": T * (2 * H + payload) + T * 4 * H + 2 * routing, "flops": 0}
        rows = T * K * (1 - c["drop"])
        back = rows * (payload + 2 * H) if c["fp8"] else 0
        return {"bytes": T * 2 * H + rows * payload + back + rows * 2 * H + T * 2 * H + routing, "flops": 2 * rows * H}
    if kind == "linear":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if kind == "linear_fp8":
        m, n, k = c["m"], c["n"], c["k"]
        return {"bytes": 2 * m * k + 2 * (m * k + m * k // 32) + n * k + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "ar_rmsnorm":
        return {"bytes": c["tokens"] * c["hidden"] * 8 + 2 * c["hidden"], "flops": 6 * c["tokens"] * c["hidden"]}
    units = [sum(math.prod(s) for _, s in shapes) for shapes in _train_shapes(c)]
    tok = c["batch"] * c["seq"]
    attention = 4 * tok * c["seq"] * c["hidden"] / 2
    layers = c["layers"] * (2 * tok * units[1] + attention)
    # forward, the forward again for the checkpointed layers, backward; the optimizer's pass over every parameter
    return {"bytes": 28 * sum(units), "flops": 4 * layers + 3 * 2 * tok * c["vocab"] * c["hidden"]}


def tolerance(case):
    c, kind = case, case["kind"]
    if kind == "collective":
        if c["op"] != "premul":
            return "exact"   # a sum of one rank's values, or a copy
        # one rounding of one product
        return {"rel": {"f64": 1e-15, "f32": 1e-7, "f16": 1e-3, "bf16": 8e-3}[c["dtype"]], "max": {"f64": 1e-14, "f32": 1e-6, "f16": 4e-3, "bf16": 1.6e-2}[c["dtype"]]}
    if kind == "moe":
        return {"rel": 4e-3, "max": 4e-2}        # one bf16 rounding of a sum held in fp32; bytes and counts are the same
    if kind in ("linear", "linear_fp8"):
        return {"rel": 4e-3, "max": 4e-2}        # one bf16 rounding of a sum held in fp32
    if kind == "ar_rmsnorm":
        return {"rel": 4e-3, "max": 4e-2}        # one bf16 rounding of each output
    # bf16 through a whole model, forward and backward, and squares of gradients
    return {"rel": 2e-2, "max": 0.9}


# ------------------------------------------------------------------------------------------------ 64-bit results
def _quantised(x, clamp, by_division):
    """Values of e4m3 blocks of 128 channels and their scales, each step rounded to fp32 as the format defines it (torch
    divides by a number with a rounded reciprocal, so the quotients are taken in 64 bits)."""
    v = x.float().view(x.shape[0], -1, 128)
    amax = v.abs().amax(-1, keepdim=True).clamp_min(clamp)
    if by_division:
        scale = (amax.double() / E4M3_MAX).float()
        q = v * (1.0 / scale.double()).float()
    else:
        scale = amax * (1.0 / E4M3_MAX)
        q = v * (E4M3_MAX / amax.double()).float()
    return q.clamp(-E4M3_MAX, E4M3_MAX).to(torch.float8_e4m3fn), scale.squeeze(-1)


def _exact_train(c, seed):
    flats, tokens, targets = _train_inputs(c, seed)
    flats = [f.double().requires_grad_(True) for f in flats]
    tokens, targets = tokens.cuda(), targets.cuda()
    heads, kv, D, eps = c["heads"], c["kv_heads"], c["hidden"] // c["heads"], 1e-5
    B, S = tokens.shape

    def cut(flat, shapes):
        off, got = 0, {}
        for name, shape in shapes:
            got[name] = flat[off:off + math.prod(shape)].view(shape)
            off += math.prod(shape)
        return got

    def norm(x, gain):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * gain

    freq = 500000.0 ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
    angle = torch.arange(S, device="cuda", dtype=torch.float64)[:, None] * freq
    cos, sin = angle.cos()[:, None, :], angle.sin()[:, None, :]

    def turn(x):
        a, b = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    hidden_above = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
    shapes = _train_shapes(c)
    x = cut(flats[0], shapes[0])["tok"][tokens]
    for i in range(c["layers"]):
        p = cut(flats[1 + i], shapes[1 + i])
        h = norm(x, p["norm1"])
        q, k, v = (h @ p[n].T for n in ("wq", "wk", "wv"))
        q = turn(q.view(B, S, heads, D)).transpose(1, 2)
        k = turn(k.view(B, S, kv, D)).transpose(1, 2).repeat_interleave(heads // kv, 1)
        v = v.view(B, S, kv, D).transpose(1, 2).repeat_interleave(heads // kv, 1)
        att = (q @ k.transpose(-1, -2) / math.sqrt(D)).masked_fill(hidden_above, -math.inf).softmax(-1) @ v
        x = x + att.transpose(1, 2).reshape(B, S, -1) @ p["wo"].T
        h = norm(x, p["norm2"])
        gate = h @ p["w_gate"].T
        x = x + (gate * torch.sigmoid(gate) * (h @ p["w_up"].T)) @ p["w_down"].T
    p = cut(flats[-1], shapes[-1])
    logits = (norm(x, p["norm"]) @ p["out"].T).view(-1, c["vocab"])
    loss = (torch.logsumexp(logits, -1) - logits.gather(1, targets.view(-1, 1)).squeeze(1)).mean()
    units = []
    for f, g in zip(flats, torch.autograd.grad(loss, flats)):
        # the first optimizer step; vectors are padded to a multiple of 128
        pad = (-f.numel()) % 128
        w, g = (torch.nn.functional.pad(t.detach(), (0, pad)) for t in (f, g))
        w = w * (1 - 1e-4 * 0.1) - 1e-4 * g / (g.abs() + 1e-8)
        units.append({"param": w, "master": w, "m": 0.1 * g, "v": 0.05 * g * g})
    return {"loss": loss.detach(), "units": units}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "collective":
        if not DTYPES[c["dtype"]].is_floating_point:
            return None
        x = _collective_inputs(c, seed).double()
        return x * _scale(c, seed) if c["op"] == "premul" else x
    if kind == "moe":
        x, idx, w, y = _moe_inputs(c, seed)
        T = c["tokens"]
        if c["fp8"]:
            q, scale = _quantised(x, 1e-4, False)
        if c["layout"] == "rank_major":
            pad, used = c["max_tokens"] - T, (idx >= 0).any(1)
            grow = torch.nn.functional.pad
            got = {"out": y[0, :T].double() * used[:, None], "counts": None, "recv_idx": None, "recv_w": grow((w * used[:, None]).double(), (0, 0, 0, pad))[None]}
            if c["fp8"]:
                got["toks"], got["scales"] = None, grow((scale * used[:, None]).double(), (0, 0, 0, pad))[None]
            else:
                got["toks"] = grow((x * used[:, None]).double(), (0, 0, 0, pad))[None]
            return got
        rows = (q.double() * scale.bfloat16().double()[..., None]).view(T, -1) if c["fp8"] else x.double()
        return {"out": rows * (w.double() * (idx >= 0)).sum(1, keepdim=True), "counts": None}
    if kind == "linear":
        x, w = _linear_inputs(c, seed)
        return x.double() @ w.double().T
    if kind == "linear_fp8":
        x, w = _linear_inputs(c, seed)
        q, s = _quantised(x, 1e-10, True)
        n, k = w.shape
        blocks = w.float().view(n // 128, 128, k // 128, 128)
        ws = (blocks.abs().amax((1, 3), keepdim=True).clamp_min(1e-10).double() / E4M3_MAX).float()
        wq = (blocks * (1.0 / ws.double()).float()).clamp(-E4M3_MAX, E4M3_MAX).to(torch.float8_e4m3fn)
        xd = (q.double() * s.double()[..., None]).view(c["m"], k)
        wd = (wq.double() * ws.double()).view(n, k)
        return {"out": xd @ wd.T, "q": None, "scales": s.double().T}
    if kind == "ar_rmsnorm":
        partial, residual, weight = _rmsnorm_inputs(c, seed)
        x = partial.double() + residual.double()
        return {"out": x * torch.rsqrt(x.square().mean(1, keepdim=True) + 1e-6) * weight.double(), "residual": x}
    return _exact_train(c, seed)
