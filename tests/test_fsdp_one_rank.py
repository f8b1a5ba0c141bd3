"""The sharded engine with one rank, whose shards are the whole units: against plain autograd on the CPU; on the GPU the optimizer taken
piece by piece during the backward against one call per unit, over steps on changing streams."""
import pytest

torch = pytest.importorskip("torch")

from mp_util import run_ranks  # noqa: E402


def _cpu_rank(rank, nranks, uid):
    import torch
    torch.set_num_threads(2)
    from nccl_b200 import Communicator
    from nccl_b200.models import llama as M
    from nccl_b200.parallel.fsdp import FSDPEngine
    comm = Communicator(nranks, rank, uid)
    cfg = M.LlamaConfig.tiny(layers=2)
    lr = 1e-2
    eng = FSDPEngine(comm, cfg, device="cpu", seed=1, lr=lr, weight_decay=0.0)
    g = torch.Generator().manual_seed(50)
    tok, tgt = (torch.randint(0, cfg.vocab, (2, 16), generator=g) for _ in range(2))
    gen = torch.Generator().manual_seed(1)
    ps = [M.init_flat(s, gen).requires_grad_(True) for _, s in M.unit_specs(cfg)]
    ref = M.reference_loss(ps, cfg, tok, tgt)
    grads = torch.autograd.grad(ref, ps)
    loss = eng.step(tok, tgt)
    # the first step of AdamW moves every weight by lr against the sign of its gradient
    bad = [float(((p.master[:f.numel()] - (f.detach().float() - lr * q.float() / (q.float().abs() + 1e-8))).abs() > 0.5 * lr).float().mean())
           for p, f, q in zip(eng.units, ps, grads)]
    same = all(torch.equal(a, u.param[:u.numel].float()) for a, u in zip(eng.full_params(), eng.units))
    comm.destroy()
    return abs(float(loss) - float(ref.detach())), max(bad), same


def test_against_autograd_on_the_cpu():
    off, bad, same = run_ranks(_cpu_rank, 1, env={"NCCL_B200_HOST_ONLY": "1", "NCCL_SOCKET_IFNAME": "lo"}, timeout=300)[0]
    assert off < 2e-2 and bad < 0.03 and same


@pytest.mark.gpu
def test_pieces_of_a_unit_are_updated_like_the_whole():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.models import llama as M
    from nccl_b200.parallel import fsdp
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    cfg = M.LlamaConfig(layers=3, hidden=512, heads=8, kv_heads=2, ffn=1032, vocab=1000)
    least = fsdp.kEarlyUpdate
    got = []
    try:
        for early in (0, 1 << 62):
            fsdp.kEarlyUpdate = early
            eng = fsdp.FSDPEngine(comm, cfg, device="cuda", seed=1, lr=1e-2)
            gen = torch.Generator().manual_seed(3)
            outs = []
            for s in (torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()):
                tok, tgt = (torch.randint(0, cfg.vocab, (2, 96), generator=gen).pin_memory() for _ in range(2))
                with torch.cuda.stream(s):
                    outs.append(eng.step(tok, tgt))
            torch.cuda.synchronize()
            got.append([float(o) for o in outs] + [t.clone() for u in eng.units for t in (u.param, u.master, u.m, u.v, u.grad)])
            eng.close()
    finally:
        fsdp.kEarlyUpdate = least
    for a, b in zip(*got):
        assert a == b if isinstance(a, float) else torch.equal(a, b)
    comm.destroy()


@pytest.mark.gpu
def test_small_pieces_wait_for_the_next():
    """wo and norm2 of this shape are a million elements, far below what is worth a launch of its own."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.models import llama as M
    from nccl_b200.parallel import fsdp
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    cfg = M.LlamaConfig(layers=2, hidden=1024, heads=8, kv_heads=2, ffn=4864, vocab=512)
    eng = fsdp.FSDPEngine(comm, cfg, device="cuda", seed=1, init_on_device=True)
    assert eng.units[1].numel >= fsdp.kEarlyUpdate
    pieces, update = [], eng._update_early

    def record(idx, lo, hi):
        pieces.append((idx, lo, hi))
        update(idx, lo, hi)

    eng._update_early = record
    tok = torch.randint(0, cfg.vocab, (1, 32))
    eng.step(tok, tok)
    w_down, w_gu = cfg.hidden * cfg.ffn, 2 * cfg.hidden * cfg.ffn
    end = eng.units[1].shard
    assert pieces == [(idx, lo, hi) for idx in (2, 1) for lo, hi in ((end - w_down, end), (end - w_down - w_gu, end - w_down))]
    assert all(hi - lo >= 1 << 22 for _, lo, hi in pieces)
    eng.close()
    comm.destroy()


def test_a_step_runs_on_the_device_of_its_engine(monkeypatch):
    """Kernels are launched into the current device's stream: a step under another current device would give them the wrong one. No GPU is
    touched here."""
    import contextlib

    from nccl_b200.parallel.fsdp import FSDPEngine
    entered = []

    @contextlib.contextmanager
    def device(d):
        entered.append(d)
        yield
        entered.append("left")

    monkeypatch.setattr(torch.cuda, "device", device)
    eng = FSDPEngine.__new__(FSDPEngine)
    eng.cuda, eng.device = True, torch.device("cuda", 1)
    eng._step = lambda tokens, targets: entered.append("step") or "loss"
    assert eng.step(None, None) == "loss" and entered == [torch.device("cuda", 1), "step", "left"]
