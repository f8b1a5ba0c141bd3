"""Row kernels of the training step (src/contrib/train_ops.cu) against the same formulas in 64 bits on the same bf16 inputs, and the
units built from them against autograd.

A result that is rounded once to bf16 is off by at most 2**-9 of its value; twice that is allowed, and for results that are
sums an absolute part: 2**-20 of the sum of the magnitudes (fp32 sums of up to 16384 terms in a tree)."""
import math

import pytest

torch = pytest.importorskip("torch")

from nccl_b200.models import llama as M  # noqa: E402
from nccl_b200.models import llama_fused  # noqa: E402

gpu = pytest.mark.gpu
ROUND = 2.0 ** -8


def _units(**kw):
    from nccl_b200 import _lib
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return llama_fused.FusedUnits(M.LlamaConfig(**kw), _lib.load())


def _rand(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).bfloat16()


def _close(got, ref, spread=0.0, roundings=1):
    err = (got.double() - ref).abs() - (roundings * ROUND * ref.abs() + 2.0 ** -20 * spread + 1e-30)
    assert bool(torch.isfinite(got.double()).all()) and float(err.max()) <= 0, float(err.max())


@gpu
@pytest.mark.parametrize("rows,hidden", [(1, 8), (3, 264), (301, 512), (2, 4096), (5, 4104), (700, 8192), (3, 8200), (2, 16384)])
@pytest.mark.parametrize("with_add", [False, True])
def test_norm_both_ways(rows, hidden, with_add):
    u = _units(eps=1e-5)
    x, add, gain = _rand(rows, hidden, seed=1), _rand(rows, hidden, seed=2, scale=0.3), (1 + 0.1 * _rand(hidden, seed=3).float()).bfloat16()
    dh, res, dgain = _rand(rows, hidden, seed=4), _rand(rows, hidden, seed=5), torch.empty(hidden, dtype=torch.bfloat16, device="cuda")
    total, h, rstd = u.norm(x, gain, add=add if with_add else None, need_rstd=True)
    if with_add:
        assert torch.equal(total, x + add)
    xd = total.double().requires_grad_(True)
    gd = gain.double().requires_grad_(True)
    ref = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * gd
    _close(h, ref.detach(), roundings=2)   # normalised, then times the gain
    dx = u.norm_backward(total, gain, rstd, dh, res if with_add else None, dgain)
    gx, gg = torch.autograd.grad(ref, (xd, gd), dh.double())
    xn = (xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5)).detach()
    r = res.double() if with_add else torch.zeros_like(gx)
    scale = torch.rsqrt(xd.detach().square().mean(-1, keepdim=True) + 1e-5)
    dn = (dh.double() * gain.double())
    _close(dx, gx + r, spread=r.abs() + scale * (dn.abs() + xn.abs() * (dn * xn).abs().mean(-1, keepdim=True)))
    _close(dgain, gg, spread=(dh.double() * xn).abs().sum(0))


@gpu
@pytest.mark.parametrize("B,S,heads,kv,d", [(1, 1, 1, 1, 16), (2, 65, 4, 2, 64), (1, 7, 3, 1, 48), (2, 33, 16, 8, 128), (1, 5, 2, 2, 256)])
def test_rope_both_ways(B, S, heads, kv, d):
    u = _units(hidden=heads * d, heads=heads, kv_heads=kv)
    rope = M.rope_tables(u.cfg, S, "cuda")
    qkv = _rand(B * S, (heads + 2 * kv) * d, seed=1)
    src = qkv.clone().view(B, S, heads + 2 * kv, d)
    u.rope(qkv, rope, S)
    out = qkv.view(B, S, heads + 2 * kv, d)
    c, s = (t.double()[None, :, None, :] for t in rope)

    def turned(x, sign):
        a, b = x[..., :d // 2].double(), x[..., d // 2:].double()
        return torch.cat([a * c - sign * b * s, b * c + sign * a * s], -1), torch.cat([(a * c).abs() + (b * s).abs(), (b * c).abs() + (a * s).abs()], -1)

    assert torch.equal(out[:, :, heads + kv:], src[:, :, heads + kv:])
    _close(out[:, :, :heads + kv], *turned(src[:, :, :heads + kv], 1))
    # gradients as [B, heads, S, D] in memory, as [B, S, heads, D], and at an odd offset
    grads = [_rand(B, n, S, d, seed=2 + i) for i, n in enumerate((heads, kv, kv))]
    for form in ("heads", "tokens", "offset"):
        if form == "tokens":
            got = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in grads]
        elif form == "offset":
            got = [torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")[1:].view(t.shape).copy_(t) for t in grads]
        else:
            got = grads
        back = u.rope_backward(*got, rope, B * S, S).view(B, S, heads + 2 * kv, d)
        for t, at in zip(grads[:2], (slice(0, heads), slice(heads, heads + kv))):
            _close(back[:, :, at], *turned(t.transpose(1, 2), -1))
        assert torch.equal(back[:, :, heads + kv:], grads[2].transpose(1, 2))


@gpu
@pytest.mark.parametrize("rows,ffn", [(1, 8), (3, 2040), (17, 2056), (260, 14336)])
def test_swiglu_both_ways(rows, ffn):
    u = _units()
    gu = _rand(rows, 2 * ffn, seed=1, scale=4.0)
    gu[0, :4] = torch.tensor([-80.0, 300.0, 0.0, -30.0], device="cuda")
    gate, up = (t.double() for t in gu.split(ffn, 1))
    sig = torch.sigmoid(gate)
    act = u.swiglu(gu)
    _close(act, gate * sig * up, roundings=2)   # silu, then times up
    dact = _rand(rows, ffn, seed=2)
    d = dact.double()
    u.swiglu_backward(gu, dact)
    _close(dact, gate * sig * up)
    dgate, dup = gu.split(ffn, 1)
    _close(dgate, d * up * sig * (1 + gate * (1 - sig)), spread=(d * up).abs() * (1 + gate.abs()))
    _close(dup, d * gate * sig)


@gpu
@pytest.mark.parametrize("rows,vocab", [(1, 8), (3, 264), (65, 1024), (130, 16384), (2, 128256)])
def test_cross_entropy(rows, vocab):
    u = _units()
    logits = _rand(rows, vocab, seed=1, scale=5.0)
    logits[0, 1:4] = -math.inf
    targets = torch.randint(0, vocab, (rows,), generator=torch.Generator().manual_seed(1)).cuda()
    targets[0] = vocab - 1
    if rows > 2:
        targets[rows // 2] = -100
    x = logits.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(x, targets)
    g, = torch.autograd.grad(ref, x)
    loss = u.cross_entropy(logits, targets)
    assert abs(float(loss) - float(ref)) <= 2e-6 * abs(float(ref)) + 1e-6
    # the exponent, a difference of numbers up to about 50, is off by a few 2**-24 of that: 1e-5 of the softmax (at the target, where 1
    # is taken off, of 1)
    soft = torch.softmax(x.detach(), -1) / max(int((targets != -100).sum()), 1)
    _close(logits, g, spread=2.0 ** 20 * 1e-5 * soft)


@gpu
def test_cross_entropy_without_a_row_that_counts():
    u = _units()
    logits = _rand(3, 64, seed=1)
    loss = u.cross_entropy(logits, torch.full((3,), -100, device="cuda"))
    assert math.isnan(float(loss)) and not logits.any()   # as the framework's own


@gpu
@pytest.mark.parametrize("bad", [[], [-1], [64], [1 << 40, -101, -(1 << 62)]])
def test_cross_entropy_reports_targets_out_of_range(bad):
    """The entry itself (its caller asserts on what it reports): rows of such targets get no gradient and add nothing to the loss, but count in its mean."""
    import ctypes
    u = _units()
    rows, vocab = 8, 64
    logits = _rand(rows, vocab, seed=1)
    targets = torch.tensor([3, -100, 0, 63, 9, 10, 11, 12], device="cuda")
    targets[5:5 + len(bad)] = torch.tensor(bad, dtype=torch.int64, device="cuda")
    good = (targets >= 0) & (targets < vocab)
    count = int((targets != -100).sum())
    x = logits.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(x[good], targets[good], reduction="sum") / count
    g, = torch.autograd.grad(ref, x)
    loss, work, ok = torch.empty((), device="cuda"), torch.empty(rows + 1, device="cuda"), torch.empty((), dtype=torch.bool, device="cuda")
    fn = u.lib.b200CrossEntropy
    assert fn(*[ctypes.c_void_p(t.data_ptr()) for t in (logits, targets, loss, work, ok)], rows, vocab, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert bool(ok) == (not bad)
    assert abs(float(loss) - float(ref)) <= 2e-6 * abs(float(ref)) + 1e-6
    assert not logits[~good].any()
    _close(logits, g, spread=2.0 ** 20 * 1e-5 * torch.softmax(x.detach(), -1) / count)


@gpu
def test_cross_entropy_of_infinite_and_nan_logits():
    u = _units()
    logits = _rand(4, 64, seed=1)
    logits[0], logits[1, 5], logits[2, 7] = -math.inf, math.inf, math.nan
    targets = torch.tensor([0, 1, 2, 3], device="cuda")
    x = logits.double().requires_grad_(True)
    ref = torch.nn.functional.cross_entropy(x, targets, reduction="none")
    g, = torch.autograd.grad(ref.sum() / 4, x)
    u.cross_entropy(logits, targets)
    assert torch.equal(logits.isnan(), g.isnan())
    _close(logits[3:], g[3:], spread=2.0 ** 20 * 1e-5)


@gpu
@pytest.mark.parametrize("B,S,hidden,heads,kv,ffn,vocab", [(1, 65, 128, 8, 2, 264, 512), (2, 130, 512, 4, 2, 1024, 1032), (1, 1, 64, 1, 1, 8, 8), (2, 257, 1024, 8, 8, 2816, 2048)])
def test_units_are_as_close_to_64_bits_as_autograd_in_bf16(B, S, hidden, heads, kv, ffn, vocab):
    u = _units(layers=1, hidden=hidden, heads=heads, kv_heads=kv, ffn=ffn, vocab=vocab)
    cfg = u.cfg
    rope = M.rope_tables(cfg, S, "cuda")
    gen = torch.Generator().manual_seed(0)
    layer, head = (M.init_flat(s, gen, std=0.05).cuda() for s in (M.layer_shapes(cfg), M.head_shapes(cfg)))
    x, gy = _rand(B, S, hidden, seed=1), _rand(B, S, hidden, seed=2)
    targets = torch.randint(0, vocab, (B, S), generator=gen).cuda()

    def by_autograd(dtype):
        xs, fl, fh = (t.to(dtype, copy=True).requires_grad_(True) for t in (x, layer, head))
        p = M.views(fl, M.layer_shapes(cfg))
        if dtype == torch.float64:
            def norm(v, gain):
                return v * torch.rsqrt(v.square().mean(-1, keepdim=True) + cfg.eps) * gain
            c, s = (t.double()[None, :, None, :] for t in rope)

            def turn(v):
                a, b = v.chunk(2, -1)
                return torch.cat([a * c - b * s, b * c + a * s], -1)
            h = norm(xs, p["norm1"])
            q, k, v = ((h @ p[n].T).view(B, S, -1, cfg.head_dim) for n in ("wq", "wk", "wv"))
            q, k, v = (t.transpose(1, 2) for t in (turn(q), turn(k).repeat_interleave(heads // kv, 2), v.repeat_interleave(heads // kv, 2)))
            mask = torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1)
            a = (q @ k.transpose(-1, -2) / math.sqrt(cfg.head_dim)).masked_fill(mask, -math.inf).softmax(-1) @ v
            y = xs + a.transpose(1, 2).reshape(B, S, -1) @ p["wo"].T
            h = norm(y, p["norm2"])
            gate = h @ p["w_gate"].T
            y = y + (gate * torch.sigmoid(gate) * (h @ p["w_up"].T)) @ p["w_down"].T
            ph = M.views(fh, M.head_shapes(cfg))
            loss = torch.nn.functional.cross_entropy((norm(xs, ph["norm"]) @ ph["out"].T).view(-1, vocab), targets.view(-1))
        else:
            y = M.decoder_layer(xs, p, cfg, rope)
            loss = M.head_loss(xs, M.views(fh, M.head_shapes(cfg)), cfg, targets)
        return [y.detach(), *torch.autograd.grad(y, (xs, fl), gy.to(dtype)), loss.detach(), *torch.autograd.grad(loss, (xs, fh))]

    exact, general = by_autograd(torch.float64), by_autograd(torch.bfloat16)
    glayer, ghead = torch.full_like(layer, 7.0), torch.full_like(head, 7.0)
    flat = x.view(-1, hidden)
    with torch.no_grad():
        xin, *y = u.layer(flat, None, layer, rope, (B, S))
        assert xin is flat
        y = y[0] + y[1]
        for t, again in zip(u.layer(flat - y, y, layer, rope, (B, S)), u.layer(flat - y + y, None, layer, rope, (B, S))):
            assert torch.equal(t, again)   # an input in two terms
    got = [y, u.layer_backward(flat, layer, glayer, rope, (B, S), gy.view(-1, hidden)), glayer]
    loss, gx = u.head(flat, None, head, ghead, targets.view(-1))
    got += [loss, gx, ghead]
    for name, e, a, b in zip(("y", "dx", "dw", "loss", "head dx", "head dw"), exact, general, got):
        scale = float(e.norm()) + 1e-30
        old, new = float((a.double() - e).norm()) / scale, float((b.double().view(e.shape) - e).norm()) / scale
        # the loss is one number, whose error is the luck of the logits' rounding: two roundings to bf16 at most
        assert new <= (2 ** -8 if name == "loss" else 1.05 * old + 1e-5), (name, old, new)


def test_what_stays_with_autograd():
    tok = torch.zeros(2, 8, dtype=torch.int64)
    good = dict(hidden=256, heads=4, kv_heads=2, ffn=512, vocab=1024)
    assert llama_fused.applies(M.LlamaConfig(**good), tok, tok)
    for change in ({"heads": 32}, {"hidden": 260}, {"ffn": 516}, {"vocab": 1001}, {"hidden": 32768}, {"kv_heads": 3}):
        assert not llama_fused.applies(M.LlamaConfig(**{**good, **change}), tok, tok)
    cfg = M.LlamaConfig(**good)
    assert not llama_fused.applies(cfg, tok, tok[:1]) and not llama_fused.applies(cfg, tok, tok.int()) and not llama_fused.applies(cfg, tok[:, :0], tok[:, :0])
    with torch.no_grad():
        assert not llama_fused.applies(cfg, tok, tok)
    with torch.autograd.detect_anomaly(check_nan=False):
        assert not llama_fused.applies(cfg, tok, tok)


def test_modes_that_watch_operations_stay_with_autograd():
    from torch.overrides import TorchFunctionMode
    from torch.utils.flop_counter import FlopCounterMode
    tok = torch.zeros(2, 8, dtype=torch.int64)
    cfg = M.LlamaConfig(hidden=256, heads=4, kv_heads=2, ffn=512, vocab=1024)
    ident = lambda t: t  # noqa: E731

    class Functions(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    for mode in (FlopCounterMode(display=False), Functions(), torch.autograd.graph.saved_tensors_hooks(ident, ident)):
        with mode:
            assert not llama_fused.applies(cfg, tok, tok), mode
    seen = []
    torch.func.vmap(lambda x: seen.append(llama_fused.applies(cfg, tok, tok)) or x)(torch.zeros(2))
    assert seen == [False]
    with torch.device("cpu"):   # a default device changes no operation
        assert llama_fused.applies(cfg, tok, tok)
    assert llama_fused.applies(cfg, tok, tok)


def test_gradient_buffers_are_waited_for_behind_the_recomputation():
    """On the CPU, with kernels that do nothing: what is called before the first write stands right in front of that product."""
    from torch.utils._python_dispatch import TorchDispatchMode

    from nccl_b200 import _lib

    class NoKernels(llama_fused.FusedUnits):
        def _run(self, name, *args):
            log.append(name)

    class Products(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func.overloadpacket == torch.ops.aten.mm:
                log.append("into" if "out" in (kwargs or {}) else "mm")
            return func(*args, **(kwargs or {}))

    u = NoKernels(M.LlamaConfig(hidden=64, heads=4, kv_heads=2, ffn=128, vocab=64), _lib.load())
    rope = M.rope_tables(u.cfg, 8, "cpu")
    x, gy = (torch.zeros(16, 64, dtype=torch.bfloat16) for _ in range(2))
    for unit in ("layer", "head"):
        log = []
        shapes = M.layer_shapes(u.cfg) if unit == "layer" else M.head_shapes(u.cfg)
        flat, gflat = (torch.zeros(M.numel(shapes), dtype=torch.bfloat16) for _ in range(2))
        with Products():
            if unit == "layer":
                u.layer_backward(x, flat, gflat, rope, (2, 8), gy, before=lambda: log.append("before"))
            else:
                u.cross_entropy = lambda logits, targets: log.append("loss")
                u.head(x, None, flat, gflat, torch.zeros(16, dtype=torch.int64), before=lambda: log.append("before"))
        at = log.index("before")
        assert log.count("before") == 1 and log.index("into") == at + 1 and log[:at].count("mm") == (4 if unit == "layer" else 2)


@gpu
@pytest.mark.parametrize("shape,hidden,vocab", [((1, 1), 8, 8), ((2, 65), 64, 16), ((1, 700), 2056, 1000), ((3, 257), 4096, 5), ((2, 1024), 128, 50000)])
def test_embedding_backward(shape, hidden, vocab):
    u = _units(hidden=hidden, vocab=vocab)
    tokens = torch.randint(0, vocab, shape, generator=torch.Generator().manual_seed(2)).cuda()
    gx = _rand(*shape, hidden, seed=1)
    out = torch.full((vocab * hidden,), 7.0, dtype=torch.bfloat16, device="cuda")
    u.embedding_backward(tokens, gx, out)
    ref, spread = (torch.zeros(vocab, hidden, dtype=torch.float64, device="cuda").index_add_(0, tokens.view(-1), t.view(-1, hidden)) for t in (gx.double(), gx.double().abs()))
    _close(out.view(vocab, hidden), ref, spread)


@gpu
@pytest.mark.parametrize("tokens", [31, 32, 33, 64, 65, 1000, 8192])
@pytest.mark.parametrize("ids", ["one", "two", "half", "runs"])
def test_embedding_backward_of_repeated_ids(tokens, ids):
    """Ids that reach over the rows one CTA adds, up to all of them; the first and last id of the table; the same bits again; time that does not grow with
    the repetition."""
    hidden, vocab = 1032, 600
    u = _units(hidden=hidden, vocab=vocab)
    g = torch.Generator().manual_seed(tokens)
    tok = torch.randint(0, vocab, (1, tokens), generator=g)
    if ids == "one":
        tok[:] = 7
    elif ids == "two":
        tok[:] = torch.where(torch.arange(tokens) % 3 == 0, 0, vocab - 1)
    elif ids == "half":
        tok[0, torch.randperm(tokens, generator=g)[:tokens // 2]] = 300
    else:
        tok[0] = torch.arange(tokens) // 47 % vocab
    tok = tok.cuda()
    gx = _rand(1, tokens, hidden, seed=1)
    out, again = (torch.full((vocab * hidden,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    u.embedding_backward(tok, gx, out)
    u.embedding_backward(tok, gx, again)
    ref, spread = (torch.zeros(vocab, hidden, dtype=torch.float64, device="cuda").index_add_(0, tok.view(-1), t.view(-1, hidden)) for t in (gx.double(), gx.double().abs()))
    _close(out.view(vocab, hidden), ref, spread)
    assert torch.equal(out, again)
    if tokens == 8192:
        def ms(t):
            at = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            u.embedding_backward(t, gx, out)
            at[0].record()
            for _ in range(5):
                u.embedding_backward(t, gx, out)
            at[1].record()
            at[1].synchronize()
            return at[0].elapsed_time(at[1])
        # one CTA that adds all rows of an id took 30 times as long for one id as for uniform ones
        assert ms(tok) <= 3 * ms(torch.randint(0, vocab, (1, tokens), generator=g).cuda()) + 0.2


@gpu
def test_embedding_backward_leaves_out_ids_behind_the_table():
    u = _units(hidden=64, vocab=10)
    ids = torch.tensor([3, -1, 10, 3, 1 << 40, -(1 << 62), 9] * 20, device="cuda")
    gx = _rand(ids.numel(), 64, seed=1)
    out = torch.full((640,), 7.0, dtype=torch.bfloat16, device="cuda")
    u.embedding_backward(ids.view(1, -1), gx, out)
    valid = (ids >= 0) & (ids < 10)
    ref, spread = (torch.zeros(10, 64, dtype=torch.float64, device="cuda").index_add_(0, ids[valid], t[valid]) for t in (gx.double(), gx.double().abs()))
    _close(out.view(10, 64), ref, spread)
