"""The fused all-reduce + residual + RMSNorm kernel on one rank: row lengths around the limits of a group of threads, fewer
and more rows than groups, against fp32 PyTorch."""
import ctypes
import sys
import threading

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [8, 1016, 1024, 1032, 2048, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("tokens,ctas", [(1, 64), (7, 3), (65, 1), (200, 5), (300, 64)])
def test_rows(hidden, tokens, ctas):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.devapi import DeviceComm
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    dc = DeviceComm(comm)
    part, resid, out = (dc.symmetric((tokens + 1) * hidden, torch.bfloat16).view(tokens + 1, hidden) for _ in range(3))
    g = torch.Generator(device="cuda").manual_seed(hidden + tokens)
    w = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).bfloat16()
    for mode in (0, 2):
        part.copy_(torch.randn(tokens + 1, hidden, device="cuda", generator=g))
        resid.copy_(torch.randn(tokens + 1, hidden, device="cuda", generator=g))
        out.fill_(9)
        x = (part.float() + resid.float()).bfloat16()
        ref = x.float() * torch.rsqrt(x.float().square().mean(1, keepdim=True) + 1e-5) * w.float()
        guard = resid[tokens].clone()
        torch.cuda.synchronize()
        dc.ar_rmsnorm(part[:tokens], resid[:tokens], out[:tokens], w, eps=1e-5, mode=mode, ctas=ctas)
        assert dc.status() == 0
        assert torch.equal(resid[:tokens], x[:tokens]) and torch.equal(resid[tokens], guard) and (out[tokens] == 9).all()
        # one bf16 rounding (2^-9) of a value that fp32 has to about 1e-6
        torch.testing.assert_close(out[:tokens].float(), ref[:tokens], rtol=2 ** -8, atol=1e-6)
    dc.destroy()
    comm.destroy()


@pytest.mark.parametrize("hidden", [6144, 6152, 7168, 8104, 8184])
@pytest.mark.parametrize("tokens,ctas", [(35, 3), (36, 3), (77, 5), (770, 64)])
def test_long_rows(hidden, tokens, ctas):
    """Both sides of the line behind which a CTA has six rows under way: rows longer than 6144, twelve to a CTA."""
    test_rows(hidden, tokens, ctas)


@pytest.mark.parametrize("tokens,hidden", [(5, 0), (5, -8), (0, 1024)])
def test_empty_calls(tokens, hidden):
    """No rows, or rows without channels, are an empty call of the C entry point: nothing is divided by their size, nothing is
    launched or written."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.devapi import DeviceComm
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    dc = DeviceComm(comm)
    bufs = [dc.symmetric(1024, torch.bfloat16).fill_(9) for _ in range(3)]
    w = torch.ones(1024, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    for mode in (0, 2):
        places = [v for b in bufs for v in dc._locate(b)]
        assert dc.lib.b200DevApiArRmsNorm(ctypes.byref(dc.dc), *places, w.data_ptr(), 1e-6, tokens, hidden, mode, 4, 0) == 0
    assert dc.status() == 0 and all((b == 9).all() for b in bufs)
    dc.destroy()
    comm.destroy()


def test_threads_with_rings_of_different_sizes():
    """Threads launch the same kernel (32 threads to a row) with rings of 32 KiB and of 128 KiB: none takes the limit of shared
    memory away from another."""
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.devapi import DeviceComm
    torch.cuda.set_device(0)
    failed, work = [], []
    for tokens, hidden in ((40, 64), (16, 2048)) * 2:
        comm = Communicator(1, 0, get_unique_id())
        dc = DeviceComm(comm)
        bufs = [dc.symmetric(tokens * hidden, torch.bfloat16).view(tokens, hidden).zero_() for _ in range(3)]
        work.append((comm, dc, bufs, torch.ones(hidden, dtype=torch.bfloat16, device="cuda"), torch.cuda.Stream()))
    torch.cuda.synchronize()

    def calls(dc, bufs, w, stream):
        torch.cuda.set_device(0)
        places = [v for b in bufs for v in dc._locate(b)]
        args = (ctypes.byref(dc.dc), *places, w.data_ptr(), 1e-6, *bufs[0].shape, 0, 1, stream.cuda_stream)
        call = dc.lib.b200DevApiArRmsNorm   # without the interpreter's lock
        failed.extend(r for r in (call(*args) for _ in range(20000)) if r)

    interval = sys.getswitchinterval()
    sys.setswitchinterval(1e-6)
    threads = [threading.Thread(target=calls, args=w[1:]) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    sys.setswitchinterval(interval)
    torch.cuda.synchronize()
    assert not failed
    for comm, dc, *_ in work:
        dc.destroy()
        comm.destroy()
