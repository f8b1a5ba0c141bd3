"""The sharded engine with the activations of none, some and all layers kept for the backward: the same gradients as computing them again."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 65), (2, 128)])
def test_kept_layers(shape, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.models import llama as M
    from nccl_b200.parallel.fsdp import FSDPEngine
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    cfg = M.LlamaConfig(layers=3, hidden=256, heads=4, kv_heads=2, ffn=512, vocab=1024)
    g = torch.Generator().manual_seed(3)
    tok, tgt = (torch.randint(0, cfg.vocab, shape, generator=g) for _ in range(2))
    got = []
    for layers in (0, 2, 3, None):
        eng = FSDPEngine(comm, cfg, device="cuda", seed=1, lr=1e-3, eps=1.0, init_on_device=True)
        used = []
        again = eng.fused._to_product
        monkeypatch.setattr(eng.fused, "_to_product", lambda *a: used.append(a[-1]) or again(*a))
        if layers is None:   # by what is free: a small model has room for all
            assert eng._layers_kept(tok.numel()) == cfg.layers
            monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (0, 0))
            monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda *a: {k: {"all": {"current": 0}} for k in ("reserved_bytes", "allocated_bytes")})
            assert eng._layers_kept(tok.numel()) == 0   # nothing free: none
            monkeypatch.undo()
            asked = []
            real = torch.cuda.mem_get_info
            monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: asked.append(1) or real(*a))
            for _ in range(3):   # the second step finds what the first one left in the allocator, the third finds no change
                eng.step(tok, tgt)
            n = len(asked)
            eng.step(tok, tgt)
            assert 1 <= n <= 3 and len(asked) == n
            held = torch.empty(1 << 26, dtype=torch.uint8, device="cuda")
            eng.step(tok, tgt)
            assert len(asked) == n + 1
            del held
            eng.close()
            continue
        else:
            monkeypatch.setattr(eng, "_layers_kept", lambda tokens: layers)
        losses = [eng.step(tok, tgt) for _ in range(2)]
        torch.cuda.synchronize()
        # forward passes with and without what the backward needs, then the layers computed again, for each step
        assert used == ([False] * (3 - layers) + [True] * layers + [True] * (3 - layers)) * 2
        got.append((torch.stack(losses), [u.m.clone() for u in eng.units]))
        eng.close()
    for losses, ms in got[1:3]:
        # the same operations on the same values; attention alone may pick another kernel where no gradient is wanted, and adds its gradients up
        # in no fixed order: both within bf16's rounding of one of some 30 chained results (2**-9)
        assert torch.allclose(losses, got[0][0], rtol=2 ** -9)
        for a, b in zip(ms, got[0][1]):
            assert float((a.double() - b.double()).norm() / b.double().norm()) < 3e-2
    comm.destroy()


@pytest.mark.parametrize("where", ["first layer kept", "last layer", "head", "backward", "declined"])
def test_memory_that_runs_out(where, monkeypatch):
    """A step that runs out of memory with activations kept is one that computes them again, and the next steps keep fewer."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.models import llama as M
    from nccl_b200.parallel.fsdp import FSDPEngine
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    cfg = M.LlamaConfig(layers=4, hidden=256, heads=4, kv_heads=2, ffn=512, vocab=1024)
    g = torch.Generator().manual_seed(3)
    tok, tgt = (torch.randint(0, cfg.vocab, (1, 65), generator=g) for _ in range(2))
    eng = FSDPEngine(comm, cfg, device="cuda", seed=1, lr=1e-3, eps=1.0, init_on_device=True, keep_layers=0 if where == "declined" else None)
    ref = FSDPEngine(comm, cfg, device="cuda", seed=1, lr=1e-3, eps=1.0, init_on_device=True, keep_layers=0)
    used, failed = [], []
    product, head, backward_bytes = eng.fused._to_product, eng.fused.head, eng._backward_bytes

    def fail(now):
        if now and not failed:
            failed.append(1)
            raise torch.OutOfMemoryError("no memory")

    def counted(*a):
        fail(a[-1] and where in ("first layer kept", "last layer") and len(used) == (0 if where == "first layer kept" else 3))
        used.append(a[-1])
        return product(*a)

    def failing_head(*a, **kw):
        fail(where == "head")
        return head(*a, **kw)

    def failing_bytes(tokens):   # of the check ahead of the backward, not of the decision ahead of the forward
        if where == "backward" and len(used) == cfg.layers and not failed:
            failed.append(1)
            return 1 << 50
        return backward_bytes(tokens)
    monkeypatch.setattr(eng.fused, "_to_product", counted)
    monkeypatch.setattr(eng.fused, "head", failing_head)
    monkeypatch.setattr(eng, "_backward_bytes", failing_bytes)
    losses = [eng.step(tok, tgt)]
    first = {"first layer kept": [False] * 4, "last layer": [True] * 3 + [False], "head": [True] * 4, "backward": [True] * 4, "declined": [False] * 4}[where]
    assert used == first + [True] * 4 and bool(failed) == (where != "declined") and eng.layers_kept == 0
    assert eng.keep_layers == (0 if where == "declined" else 2)
    used.clear()
    losses.append(eng.step(tok, tgt))
    assert used == ([False] * 4 + [True] * 4 if where == "declined" else [False] * 2 + [True] * 2 + [True] * 2)
    assert eng.layers_kept == eng.keep_layers
    want = [ref.step(tok, tgt) for _ in range(2)]
    torch.cuda.synchronize()
    # the bounds of the test above: attention may pick another kernel where no gradient is wanted
    assert torch.allclose(torch.stack(losses), torch.stack(want), rtol=2 ** -9)
    for a, b in zip(eng.units, ref.units):
        assert float((a.m.double() - b.m.double()).norm() / b.m.double().norm()) < 3e-2
    eng.close()
    ref.close()
    comm.destroy()


def test_step_within_a_share_of_the_memory():
    """A step of a model whose layers would keep more than the process may have."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.models import llama as M
    from nccl_b200.parallel.fsdp import FSDPEngine
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    cfg = M.LlamaConfig(layers=12, hidden=1024, heads=8, kv_heads=2, ffn=3584, vocab=1024)
    eng = FSDPEngine(comm, cfg, device="cuda", seed=1, init_on_device=True)
    tok = torch.randint(0, cfg.vocab, (1, 8192))
    each, total = eng.fused.activation_bytes(tok.numel()), torch.cuda.mem_get_info()[1]
    torch.cuda.empty_cache()
    try:
        for layers in (6, 12, 40):
            torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + layers * each) / total)
            loss = eng.step(tok, tok)
            torch.cuda.synchronize()
            assert torch.isfinite(loss) and torch.cuda.memory_reserved() <= (torch.cuda.get_per_process_memory_fraction() + 1e-6) * total
            kept = eng._kept_for[2] if eng._kept_for else 0
            assert kept < cfg.layers or layers > 12
            torch.cuda.empty_cache()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    eng.close()
    comm.destroy()


@pytest.mark.parametrize("fused_attention", [True, False])
def test_attention_that_saves_probabilities(fused_attention, monkeypatch):
    """Attention by single operations saves S x S values per head for its backward: layers that run it are computed again, and a step takes no more
    memory than one that keeps none."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.models import llama as M
    from nccl_b200.parallel.fsdp import FSDPEngine
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    cfg = M.LlamaConfig(layers=4, hidden=512, heads=8, kv_heads=2, ffn=512, vocab=512)
    g = torch.Generator().manual_seed(3)
    tok, tgt = (torch.randint(0, cfg.vocab, (1, 1024), generator=g) for _ in range(2))
    peaks, losses = [], []
    for most in (0, None):
        eng = FSDPEngine(comm, cfg, device="cuda", seed=1, lr=1e-3, init_on_device=True, keep_layers=most)
        used, product = [], eng.fused._to_product
        monkeypatch.setattr(eng.fused, "_to_product", lambda *a: used.append(a[-1]) or product(*a))
        with sdpa_kernel([SDPBackend.FLASH_ATTENTION, SDPBackend.CUDNN_ATTENTION] if fused_attention else SDPBackend.MATH):
            eng.step(tok, tgt)
            torch.cuda.synchronize()
            used.clear()
            before = torch.cuda.memory_allocated()
            torch.cuda.reset_peak_memory_stats()
            losses.append(float(eng.step(tok, tgt)))
            torch.cuda.synchronize()
            peaks.append(torch.cuda.max_memory_allocated() - before)
        again = 0 if most is None and fused_attention else cfg.layers
        assert used == [most is None] * cfg.layers + [True] * again
        eng.close()
    assert abs(losses[1] - losses[0]) <= 2 ** -9 * losses[0]
    if not fused_attention:
        # a block may be up to 1 MiB larger than what it was taken for, by what the allocator had at hand; one layer that keeps its probabilities
        # in bf16 takes 16 MiB
        assert peaks[1] - peaks[0] < 2 * cfg.heads * tok.numel() ** 2
    comm.destroy()
