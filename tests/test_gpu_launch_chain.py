"""Kernels that are launched while the one before them still runs (programmatic stream serialisation): chains in which every call reads
what the call before wrote and overwrites what it read, issued without waiting, against the same calls one at a time; then the
chain captured into a CUDA graph and replayed."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROUNDS = 6


def _chain(env, wait):
    """Outputs of every round, each made from buffers that the rounds before have used too."""
    comm, tp, ep, dc, op, b = (env[k] for k in ("comm", "tp", "ep", "dc", "op", "buf"))
    got = []

    def done():
        if wait:
            torch.cuda.synchronize()

    for r in range(ROUNDS):
        comm.all_gather(b["x"].view(-1), b["y"].view(-1))            # aligned copy
        done()
        comm.all_reduce(b["y"].view(-1)[1:], b["z"][3:2 + b["y"].numel()], op=op)   # scaled, at odd offsets
        done()
        q, s = tp.quantize_fp8(b["y"], q=b["q"], scales=b["s"])
        done()
        tp.gemm_fp8(q, s, b["wq"], b["ws"], out=b["big"])
        done()
        tp.gemm(b["big"][:128].contiguous(), b["w"], out=b["small"])  # K shared by a cluster
        done()
        tp.gemm(b["big"], b["w"], out=b["tall"])
        done()
        b["partial"].copy_(b["tall"][:b["partial"].shape[0]])
        dc.ar_rmsnorm(b["partial"], b["residual"], b["normed"], b["gain"])
        done()
        x = b["normed"]
        toks, _, counts = ep.dispatch(x, b["idx"], b["prob"], fp8=False, toks=b["toks"], counts=b["counts"])
        done()
        ep.combine(toks, out=b["back"])
        done()
        b["x"][:b["back"].shape[0]].copy_(b["back"])                  # the next round's input
        got += [b[k].clone() for k in ("z", "q", "s", "small", "tall", "normed", "residual", "back", "counts")]
        done()
    return got


@pytest.fixture(scope="module")
def env():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.core import BF16
    from nccl_b200.ops.devapi import DeviceComm
    from nccl_b200.ops.ep import ExpertParallel
    from nccl_b200.ops.tp import TensorParallel
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    tp, dc = TensorParallel(comm, 1024, 2048), DeviceComm(comm)
    T, H, E, K = 384, 2048, 16, 4
    ep = ExpertParallel(comm, E, T, H, layout="expert_major")
    dev = dict(device="cuda", dtype=torch.bfloat16)
    b = {"x": torch.empty(640, H, **dev), "y": torch.empty(640, H, **dev), "z": torch.empty(640 * H + 8, **dev), "big": torch.empty(640, H, **dev),
         "q": torch.empty(640, H, dtype=torch.float8_e4m3fn, device="cuda"), "s": torch.empty(H // 128, 640, device="cuda"),
         "small": torch.empty(128, H, **dev), "tall": torch.empty(640, H, **dev), "gain": torch.ones(H, **dev), "back": torch.empty(T, H, **dev),
         "toks": torch.empty(E, T, H, **dev), "counts": torch.empty(E, dtype=torch.int32, device="cuda")}
    for name in ("partial", "residual", "normed"):
        b[name] = dc.symmetric(T * H, torch.bfloat16).view(T, H)
    g = torch.Generator(device="cuda").manual_seed(3)
    w = (torch.randn(H, H, device="cuda", generator=g) / H ** 0.5).bfloat16()
    b["w"] = w
    b["wq"], b["ws"] = tp.quantize_fp8(w.flip(0).contiguous(), 128)
    b["idx"] = torch.rand(T, E, device="cuda", generator=g).topk(K, dim=1).indices
    b["prob"] = torch.rand(T, K, device="cuda", generator=g)
    start = torch.randn(640, H, device="cuda", generator=g).bfloat16()

    def reset():
        for t in b.values():
            if t is not b["w"] and t is not b["wq"] and t is not b["ws"] and t is not b["idx"] and t is not b["prob"] and t is not b["gain"]:
                t.zero_()
        b["x"].copy_(start)

    op = comm.premul_sum(0.3125, BF16)
    yield {"comm": comm, "tp": tp, "ep": ep, "dc": dc, "op": op, "buf": b, "reset": reset}
    comm.destroy_op(op)
    ep.destroy()
    dc.destroy()
    tp.destroy()
    comm.destroy()


def test_chain_without_waiting(env):
    env["reset"]()
    torch.cuda.synchronize()
    ref = _chain(env, wait=True)
    for _ in range(3):
        env["reset"]()
        got = _chain(env, wait=False)
        torch.cuda.synchronize()
        assert len(got) == len(ref) and all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, ref))
    assert env["dc"].status() == 0


def test_chain_captured(env):
    env["reset"]()
    torch.cuda.synchronize()
    ref = _chain(env, wait=True)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        env["reset"]()
        _chain(env, wait=False)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = _chain(env, wait=False)
    for _ in range(2):
        env["reset"]()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, ref))
    graph.reset()
