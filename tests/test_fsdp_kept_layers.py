"""How many layers of a step keep their activations: decided from what the allocator and the driver say, which these tests say for them (no GPU is
touched)."""
import pytest

torch = pytest.importorskip("torch")

from nccl_b200.models import llama as M  # noqa: E402
from nccl_b200.models.llama_fused import FusedUnits  # noqa: E402
from nccl_b200.parallel.fsdp import FSDPEngine, _Kept  # noqa: E402

GB = 1 << 30
CFG = M.LlamaConfig(layers=8, hidden=4096, heads=32, kv_heads=8, ffn=14336, vocab=128256)


class Memory:
    """One GPU's memory as torch.cuda tells of it."""

    def __init__(self, monkeypatch, total=180 * GB, free=150 * GB, reserved=10 * GB, used=9 * GB, fraction=1.0):
        self.total, self.free, self.reserved, self.used, self.fraction, self.asked = total, free, reserved, used, fraction, 0
        monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
        monkeypatch.setattr(torch.cuda, "mem_get_info", self.info)
        monkeypatch.setattr(torch.cuda, "get_per_process_memory_fraction", lambda device=None: self.fraction)
        monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda device=None: {
            "reserved_bytes": {"all": {"current": self.reserved}}, "allocated_bytes": {"all": {"current": self.used}}})

    def info(self, device=None):
        self.asked += 1
        return self.free, self.total


def _engine(keep_layers=None):
    eng = FSDPEngine.__new__(FSDPEngine)
    eng.keep_layers = keep_layers
    eng.cfg, eng.units, eng.device, eng._kept_for = CFG, [None] * (CFG.layers + 2), torch.device("cuda", 0), None
    eng.fused = FusedUnits.__new__(FusedUnits)
    eng.fused.cfg = CFG
    return eng


def test_memory_fraction(monkeypatch):
    """Free memory beyond the process's share is none that a step can have."""
    m, eng = Memory(monkeypatch), _engine()
    each = eng.fused.activation_bytes(4096)
    assert eng._layers_kept(4096) == CFG.layers
    m.fraction = 10.5 / 180
    assert eng._layers_kept(4096) == 0        # another share is another decision
    for gb in (12, 15, 20, 30, 60):
        m.fraction = gb / 180
        kept = eng._layers_kept(4096)
        assert kept * each <= (gb * GB - m.used) // 2
    assert kept == CFG.layers


def test_asked_once(monkeypatch):
    m, eng = Memory(monkeypatch), _engine()
    assert [eng._layers_kept(4096) for _ in range(3)] == [CFG.layers] * 3 and m.asked == 1
    m.used += 8 << 20
    eng._layers_kept(4096)
    assert m.asked == 1
    m.reserved += GB
    eng._layers_kept(4096)
    assert m.asked == 2


def test_at_most_as_many_as_the_caller_says(monkeypatch):
    m = Memory(monkeypatch)
    for most in (0, 1, 5, CFG.layers, 100, None):
        eng = _engine(most)
        assert eng._layers_kept(4096) == (CFG.layers if most is None else min(most, CFG.layers))
    assert m.asked == 5                       # nothing to ask for none
    eng.keep_layers = 3                       # and from then on
    assert eng._layers_kept(4096) == 3


def test_out_of_memory_costs_what_was_kept_only():
    kept = _Kept(3, 6)
    kept.acts[3] = kept.acts[4] = "activations"
    tried = []

    def fn():
        tried.append((kept.first, dict(kept.acts)))
        if kept.acts:
            raise torch.OutOfMemoryError("no memory")
        return "done"
    assert kept.spare(fn) == "done" and kept.ran_out and len(tried) == 2 and tried[1] == (6, {})

    def full():
        tried.append(None)
        raise torch.OutOfMemoryError("no memory at all")
    with pytest.raises(torch.OutOfMemoryError):   # nothing is left to give up: once
        kept.spare(full)
    assert len(tried) == 3
    with pytest.raises(ValueError):
        _Kept(3, 6).spare(lambda: [].index(1))


def test_activations_go_as_they_are_used():
    """On the CPU, with kernels that do nothing: by the gradient of the second norm, gate and up and that norm's output are gone, by the last product
    all but the first norm's output, for a kept layer as for one that is computed again."""
    import weakref

    from nccl_b200 import _lib

    class NoKernels(FusedUnits):
        def _run(self, name, *args):
            pass

        def norm_backward(self, *a):
            alive.append([r() is not None for r in refs])
            return super().norm_backward(*a)

    u = NoKernels(M.LlamaConfig(hidden=64, heads=4, kv_heads=2, ffn=128, vocab=64), _lib.load())
    rope = M.rope_tables(u.cfg, 8, "cpu")
    x, gy = (torch.zeros(16, 64, dtype=torch.bfloat16) for _ in range(2))
    shapes = M.layer_shapes(u.cfg)
    flat, gflat = (torch.zeros(M.numel(shapes), dtype=torch.bfloat16) for _ in range(2))
    alive = []
    with torch.no_grad():
        x, y, add, acts = u.layer(x, None, flat, rope, (2, 8), keep=True)
    h1, _, (q, _, _), a, x2, h2, _, gu = acts
    refs = [weakref.ref(t) for t in (h1, q, a, x2, h2, gu)]
    held = [acts]
    del h1, q, _, a, x2, h2, gu, acts, y, add
    u.layer_backward(x, flat, gflat, rope, (2, 8), gy, kept=held)
    assert held == [] and alive == [[True, True, True, True, False, False], [True, False, False, True, False, False]]
