"""Steps of the sharded engine on one GPU that do not, or not wholly, take the row kernels: shapes they do not fit, autocast, and fused layers whose
embedding goes by autograd; the optimizer's state after three steps against plain autograd over the same weights.

Gradients are bf16 results of chains of some 30 operations (two layers forward, again and backward), each rounded to 2**-9 of its value at
most, so two correct orders of them differ by about sqrt(30) * 2**-10, half a percent; with eps far above the gradients the weights follow
them smoothly. 3 % are allowed; a gradient that is missing, stale or of another tensor is off by about its own size."""
import contextlib

import pytest

torch = pytest.importorskip("torch")

from nccl_b200.models import llama as M  # noqa: E402
from nccl_b200.models import llama_fused  # noqa: E402

pytestmark = pytest.mark.gpu

GOOD = dict(layers=2, hidden=256, heads=4, kv_heads=2, ffn=512, vocab=1024)


def _off(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("case", ["vocab", "ffn", "autocast", "int32 ids", "many ids", "row kernels"])
def test_step_against_autograd(case, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.parallel.fsdp import FSDPEngine
    torch.cuda.set_device(0)
    cfg = M.LlamaConfig(**{**GOOD, **{"vocab": {"vocab": 1001}, "ffn": {"ffn": 516}}.get(case, {})})
    mode = (lambda: torch.autocast("cuda", torch.bfloat16)) if case == "autocast" else contextlib.nullcontext
    if case == "many ids":
        monkeypatch.setattr(llama_fused, "embedding_applies", lambda tokens: False)
    comm = Communicator(1, 0, get_unique_id())
    eps = 1.0
    eng = FSDPEngine(comm, cfg, device="cuda", seed=1, lr=1e-2, eps=eps, weight_decay=0.1, init_on_device=True)
    calls = {"layer_backward": 0, "head": 0, "embedding_backward": 0}
    for name in calls:
        def counted(*args, fn=getattr(eng.fused, name), name=name, **kw):
            calls[name] += 1
            return fn(*args, **kw)
        setattr(eng.fused, name, counted)
    master = [u.master[:u.numel].clone() for u in eng.units]
    m, v = ([torch.zeros_like(f) for f in master] for _ in range(2))
    b1, b2 = eng.betas
    gen = torch.Generator().manual_seed(5)
    for step in (1, 2, 3):
        tok, tgt = (torch.randint(0, cfg.vocab, (2, 70), generator=gen).cuda() for _ in range(2))
        tok = tok.int() if case == "int32 ids" else tok
        with mode():
            loss = eng.step(tok, tgt)
            ps = [f.bfloat16().requires_grad_(True) for f in master]
            ref = M.reference_loss(ps, cfg, tok, tgt)
        assert abs(float(loss) - float(ref.detach())) <= 2 ** -7 * abs(float(ref.detach()))
        for i, g in enumerate(torch.autograd.grad(ref, ps)):
            g = g.float()
            m[i] = b1 * m[i] + (1 - b1) * g
            v[i] = b2 * v[i] + (1 - b2) * g * g
            master[i] = master[i] * (1 - 1e-2 * 0.1) - 1e-2 * (m[i] / (1 - b1 ** step)) / (v[i].sqrt() / (1 - b2 ** step) ** 0.5 + eps)
    fused = case in ("int32 ids", "many ids", "row kernels")
    assert calls == {"layer_backward": 6 * fused, "head": 3 * fused, "embedding_backward": 3 * (case == "row kernels")}
    for u, want_m, want_v, want in zip(eng.units, m, v, master):
        n = u.numel
        assert _off(u.m[:n], want_m) <= 0.03 and _off(u.v[:n], want_v) <= 0.06, (u.name, _off(u.m[:n], want_m), _off(u.v[:n], want_v))
        assert _off(u.master[:n], want) <= 1e-4 and torch.equal(u.param[:n], u.master[:n].bfloat16())
        assert not u.m[n:].any() and not u.master[n:].any()
    eng.close()
    comm.destroy()
