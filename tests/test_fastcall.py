"""The native host path of the wrappers (bindings/python/fastcall.c): what reaches an entry point is what ctypes hands over, and what the wrappers
refuse stays refused."""
import ctypes
import functools
import os
import shutil

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from mp_util import run_ranks  # noqa: E402
from nccl_b200 import _lib, core  # noqa: E402

P, I, Z = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
_lib.load()   # builds library and module where they are not
needs_module = pytest.mark.skipif(_lib.fastcall() is None, reason="built without the interpreter's headers")


def _recorder(types):
    calls = []

    def fn(*a):
        calls.append(a)
        return 7 if len(calls) > 1 else 0
    cb = ctypes.CFUNCTYPE(I, *types)(fn)
    return calls, cb, ctypes.cast(cb, P).value


@needs_module
def test_collectives():
    fast = _lib.fastcall()
    a, b = torch.zeros(3, 4, dtype=torch.bfloat16), torch.zeros(6)
    types, handle = core._torch_types(), ctypes.c_void_p(0x1234)
    for lead, n, t in ((0, 12, core.BF16), (1, 6, core.FP32), (2, 12, core.BF16), (3, 6, core.FP32)):
        calls, keep, at = _recorder([P, P, Z, I, I, P, P])
        assert fast.collective(at, types, None, a, b, lead, 1, -2, handle, None) == 0
        assert fast.collective(at, types, None, a, b, lead, 3, 4, handle, 77) == 7
        assert calls == [(a.data_ptr(), b.data_ptr(), n, t, -2, 0x1234, None), (a.data_ptr(), b.data_ptr(), n // 3, t, 4, 0x1234, 77)]
    calls, keep, at = _recorder([P, P, Z, I, P, P])

    class Stream:
        cuda_stream = 1 << 40
    assert fast.collective(at, types, None, None, b, 3, 1, None, None, Stream()) == 0
    assert calls == [(None, b.data_ptr(), 6, core.FP32, None, 1 << 40)]


@needs_module
def test_refused():
    fast, types = _lib.fastcall(), core._torch_types()
    calls, keep, at = _recorder([P, P, Z, I, P, P])
    ok = torch.zeros(4)
    for bad, error in ((torch.zeros(4, 4).t(), ValueError), (torch.zeros(4, dtype=torch.complex64), KeyError)):
        for pair in ((ok, bad), (bad, ok)):
            with pytest.raises(error):
                fast.collective(at, types, None, *pair, 0, 1, None, 0, None)
    for other in (np.zeros(4, np.float32), [1, 2], object()):
        assert fast.collective(at, types, None, ok, other, 0, 1, None, 0, None) is NotImplemented
    for args in ((at, 1.5), (at, "x"), (at, *range(33)), (0, 1), ()):
        with pytest.raises((TypeError, AttributeError)):
            fast.invoke(*args)
    with pytest.raises(TypeError):
        fast.collective(at, types, None, None, ok, 0, 1, None, 0, None)   # nothing to count
    assert not calls


@needs_module
@pytest.mark.parametrize("n", [1, 8, 9, 16, 17, 32])
def test_words(n):
    """Words on both sides of the forms that a call takes; shapes are four of them."""
    calls, keep, at = _recorder([ctypes.c_uint64] * n)
    args = [(1 << 64) - 1 - k if k % 3 else k - 5 for k in range(n)]
    assert _lib.fastcall().invoke(at, *args) == 0
    assert calls == [tuple(v % (1 << 64) for v in args)]
    if n == 16:   # words behind the last are whatever the registers and the stack hold
        calls, keep, at = _recorder([ctypes.c_uint64] * n)
        _lib.fastcall().invoke(at, torch.Size((2, 3)), (4, 5, 6), (9,), torch.Size((1, 2, 3, 4)))
        assert calls == [(2, 2, 3, 0, 3, 4, 5, 6, 1, 0, 0, 0, 4, 0, 0, 0)]


def _rank(rank, nranks, uid):
    import torch
    from nccl_b200 import Communicator
    comm = Communicator(nranks, rank, uid)
    got, took = [], []
    real = comm._native
    comm._native = lambda *a: took.append(real(*a)) or took[-1]
    for native in (True, False):
        if not native:
            comm._entries = dict.fromkeys(("ncclAllReduce", "ncclBroadcast", "ncclReduceScatter", "ncclAllGather", "ncclAlltoAll"))
        x = torch.arange(8, dtype=torch.float32) * (rank + 1)
        out = [comm.all_reduce(x, torch.zeros(8)), comm.all_reduce(x.clone(), op="max"), comm.broadcast(x if rank == 1 else None, torch.zeros(8), 1),
               comm.reduce_scatter(x, torch.zeros(4), op="avg"), comm.all_gather(x, torch.zeros(16)), comm.all_to_all(x, torch.zeros(8))]
        got.append([t.tolist() for t in out])
        assert took == [native] * 6   # neither path stands in for the other
        took.clear()
        with pytest.raises(ValueError):
            comm.all_reduce(torch.zeros(4, 4).t())
        with pytest.raises(TypeError):
            comm.all_reduce([1, 2])
        assert comm.all_reduce(np.ones(3, np.float32), np.zeros(3, np.float32)).tolist() == [nranks] * 3
        assert not any(took)
        took.clear()
    comm.destroy()
    return got


@needs_module
def test_communicator_either_way():
    got = run_ranks(_rank, 2, env={"NCCL_B200_HOST_ONLY": "1", "NCCL_SOCKET_IFNAME": "lo"}, timeout=300)
    for rank in range(2):
        native, through_ctypes = got[rank]
        assert native == through_ctypes and native[0] == [3.0 * i for i in range(8)]


@needs_module
def test_no_integer_where_one_is_due():
    """Whether an entry point takes an operator or a root is not told by the caller's value: None reaches none of them."""
    fast, types = _lib.fastcall(), core._torch_types()
    calls, keep, at = _recorder([P, P, Z, I, I, P, P])
    a, b = torch.zeros(4), torch.zeros(4)
    for lead in (4, 5, 7):
        assert fast.collective(at, types, None, a, b, lead, 1, None, 0x1234, 0x77) is NotImplemented
    assert not calls
    assert fast.collective(at, types, None, a, b, 7, 1, 3, 0x1234, 0x77) == 0
    assert calls == [(a.data_ptr(), b.data_ptr(), 4, core.FP32, 3, 0x1234, 0x77)]


class _CallsOnly:
    """A library of which the wrappers' methods see the entry points alone: each call is recorded."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        fn = ctypes.CFUNCTYPE(I, *_lib._PROTOS[name])(lambda *a: self.calls.append((name, *a)) or 0)
        fn.argtypes = _lib._PROTOS[name]
        setattr(self, name, fn)
        return fn


def _wrapper(monkeypatch):
    """A communicator over recorded entry points that takes the native path where that is built."""
    lib = _CallsOnly()
    comm = core.Communicator(2, 0, None, lib=lib, _handle=ctypes.c_void_p(0x1234))
    monkeypatch.setattr(_lib, "address", lambda lib, name: ctypes.cast(getattr(lib, name), P).value)
    return lib, comm


def test_broadcast_without_a_root(monkeypatch):
    lib, comm = _wrapper(monkeypatch)
    x, y = torch.zeros(4), torch.zeros(4)
    with pytest.raises(ctypes.ArgumentError):
        comm.broadcast(x, y, None, stream=0x77)
    assert not lib.calls
    comm.broadcast(x, y, 1, stream=0x77)
    assert lib.calls == [("ncclBroadcast", x.data_ptr(), y.data_ptr(), 4, core.FP32, 1, 0x1234, 0x77)]


def test_integers_that_are_no_int(monkeypatch):
    """What ctypes takes for an integer or a stream, either path takes; what it refuses, both refuse."""
    lib, comm = _wrapper(monkeypatch)
    x, y = torch.zeros(4), torch.zeros(4)

    class Stream:
        cuda_stream = P(0x77)
    for root in (np.int64(1), np.uint8(1), torch.tensor(1), True):
        comm.broadcast(x, y, root, stream=Stream())
    Stream.cuda_stream = None
    comm.broadcast(x, y, 1, stream=Stream())
    at = ("ncclBroadcast", x.data_ptr(), y.data_ptr(), 4, core.FP32, 1, 0x1234)
    assert lib.calls == [(*at, 0x77)] * 4 + [(*at, None)]
    lib.calls.clear()
    for root in (1.0, "1", object(), torch.zeros(2)):
        with pytest.raises(ctypes.ArgumentError):
            comm.broadcast(x, y, root)
    comm.nranks = np.int64(2)
    comm.all_to_all(x, y, stream=0x77)
    assert lib.calls == [("ncclAlltoAll", x.data_ptr(), y.data_ptr(), 2, core.FP32, 0x1234, 0x77)]


def test_block_rows(monkeypatch):
    """The rows of a block of fp8 scales are the one integer that a caller hands to a call of words."""
    from nccl_b200.ops.tp import TensorParallel
    calls = []
    types = [P, P, P, P, I, I, I, P]
    fn = ctypes.CFUNCTYPE(I, *types)(lambda *a: calls.append(a) or 0)
    fn.argtypes = types
    fast = _lib.fastcall()
    tp = TensorParallel.__new__(TensorParallel)
    tp.lib, tp.handle, tp._fp8_ready = type("Lib", (), {"ncclTpQuantizeFp8": fn}), P(0x1234), True
    tp._ncclTpQuantizeFp8 = functools.partial(fast.invoke, ctypes.cast(fn, P).value) if fast else fn
    monkeypatch.setattr(tp, "_stream", lambda stream: 0x77, raising=False)
    x = torch.zeros(256, 128, dtype=torch.bfloat16)
    for rows in (128, np.int64(128), torch.tensor(128)):
        q, scales = tp.quantize_fp8(x, rows)
        assert tuple(scales.shape) == (1, 2) and calls.pop() == (0x1234, x.data_ptr(), q.data_ptr(), scales.data_ptr(), 256, 128, 128, 0x77)
    for rows in (None, 128.0, "128"):
        with pytest.raises(ctypes.ArgumentError):
            tp.quantize_fp8(x, rows, q=q, scales=scales)
    assert not calls


@needs_module
def test_module_built_after_it_was_asked_for(monkeypatch, tmp_path):
    """What is not there yet is looked for again: loading the library builds it."""
    built = os.path.join(_lib._HERE, "lib", "_fastcall.so")
    monkeypatch.setattr(_lib, "_HERE", str(tmp_path))
    assert _lib.fastcall() is None
    (tmp_path / "lib").mkdir()
    shutil.copy(built, tmp_path / "lib")
    assert _lib.fastcall() is not None
