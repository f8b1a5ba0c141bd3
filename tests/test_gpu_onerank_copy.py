"""One-rank collectives move data with the local copy and scale kernels: every alignment of source and destination, sizes
around the 16-byte packs and the tiles of a CTA, against plain tensor arithmetic, with guard bands around the result."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    from nccl_b200 import Communicator, get_unique_id
    torch.cuda.set_device(0)
    c = Communicator(1, 0, get_unique_id())
    yield c
    c.destroy()


def _between_bands(count, off, dtype):
    raw = torch.full((count + off + 64,), 77, device="cuda").to(dtype)
    return raw, raw[off:off + count]


# one below, at and above: a pack, what is moved byte by byte (up to 2048), a tile (4 x 512 packs), several tiles; from 2049 on
# with ends of 1, 8, 15 and 16 bytes behind the packs
@pytest.mark.parametrize("nbytes", [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 2047, 2048, 2049, 2056, 2064, 2079, 2080, 2081, 4095, 32767, 32768, 32769,
                                    32768 * 3 + 21, (1 << 20) + 13])
@pytest.mark.parametrize("soff,doff", [(0, 0), (1, 1), (0, 1), (3, 0), (15, 14), (7, 9), (8, 4), (16, 5)])
def test_copy_at_any_alignment(comm, nbytes, soff, doff):
    sraw, src = _between_bands(nbytes, soff, torch.uint8)
    src.copy_(torch.randint(0, 256, (nbytes,), dtype=torch.uint8, device="cuda"))
    draw, dst = _between_bands(nbytes, doff, torch.uint8)
    comm.all_gather(src, dst)
    torch.cuda.synchronize()
    assert torch.equal(src, dst)
    assert (draw[:doff] == 77).all() and (draw[doff + nbytes:] == 77).all()


@pytest.mark.parametrize("nbytes", [2049, 2111, 2112, 2113, 65536 + 31, 3 * 32768 + 77])
def test_copy_at_every_shift(comm, nbytes):
    """Packs of 32 bytes from two words each: every distance of source and destination, from both ends of a word."""
    for shift in range(32):
        for doff in (0, 1, 31):
            test_copy_at_any_alignment(comm, nbytes, doff + shift, doff)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16", "float64", "int32", "int64"])
@pytest.mark.parametrize("count,soff,doff", [(1, 0, 0), (7, 0, 0), (9, 1, 0), (40, 1, 1), (256, 1, 0), (257, 0, 1), (513, 1, 2), (1025, 3, 1), (2047, 0, 3), (16384, 0, 0), (16391, 3, 2), (100003, 1, 0)])
def test_scale_at_any_element_offset(comm, dtype, count, soff, doff):
    from nccl_b200 import core
    dt = getattr(torch, dtype)
    code = {"float32": core.FP32, "bfloat16": core.BF16, "float16": core.FP16, "float64": core.FP64, "int32": core.INT32, "int64": core.INT64}[dtype]
    factor = 3 if dt in (torch.int32, torch.int64) else 0.3125
    sraw, src = _between_bands(count, soff, dt)
    src.copy_((torch.randn(count, device="cuda", dtype=torch.float64) * 50).to(dt))
    draw, dst = _between_bands(count, doff, dt)
    op = comm.premul_sum(factor, code)
    for buf in (dst, src):   # out of place, then in place
        ref = src * factor   # one rounding of one product, like the kernel
        comm.all_reduce(src, buf, op=op)
        torch.cuda.synchronize()
        assert torch.equal(buf, ref)
    assert (draw[:doff] == 77).all() and (draw[doff + count:] == 77).all()
    comm.destroy_op(op)
