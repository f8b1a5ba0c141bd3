"""Block-scaled fp8: the GEMM at the edges of its pipeline (one K block, odd and even numbers of them, one tile, more tiles than
CTAs) against a 64-bit product, and the quantiser of activations at the edges of its tiles."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPES = [(128, 256, 128), (256, 256, 128), (384, 512, 256), (640, 256, 640), (1920, 1024, 384), (4224, 2304, 1152)]


def test_fp8_tiles():
    if not torch.cuda.is_available() or torch.cuda.get_device_capability()[0] < 10:
        pytest.skip("needs sm_100")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.tp import TensorParallel
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    tp = TensorParallel(comm, 4096, 4096)
    for M, N, K in SHAPES:
        g = torch.Generator(device="cuda").manual_seed(M + N + K)
        xq, xs = tp.quantize_fp8((torch.randn(M, K, device="cuda", generator=g) * torch.rand(M, 1, device="cuda", generator=g) * 4).bfloat16())
        wq, ws = tp.quantize_fp8((torch.randn(N, K, device="cuda", generator=g) * 0.05).bfloat16(), 128)
        xd = (xq.double().view(M, -1, 128) * xs.t().double().unsqueeze(-1)).view(M, K)
        wd = (wq.double().view(N // 128, 128, -1, 128) * ws.t().double()[:, None, :, None]).view(N, K)
        ref = xd @ wd.t()
        out = torch.full((M + 1, N), 9.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):
            tp.gemm_fp8(xq, xs, wq, ws, out=out[:M])
            torch.cuda.synchronize()
            # bf16 rounds to 2^-9 of the value; the sums are fp32 over K terms of at most the row's and column's size
            bound = 2 ** -8 * ref.abs() + 2 ** -20 * (xd.abs() @ wd.abs().t())
            assert ((out[:M].double() - ref).abs() <= bound).all(), (M, N, K)
            assert (out[M] == 9).all()
    assert comm.async_error() == 0
    tp.destroy()
    comm.destroy()


@pytest.mark.parametrize("rows,K", [(1, 128), (7, 384), (9, 512), (3, 2048), (4, 2176), (5, 896), (129, 4224)])
@pytest.mark.parametrize("off", [0, 4])   # 4 elements: too little alignment for the wide loads, which rows from 512 channels on take
def test_quantise_rows(rows, K, off):
    if not torch.cuda.is_available() or torch.cuda.get_device_capability()[0] < 10:
        pytest.skip("needs sm_100")
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.tp import TensorParallel
    comm = Communicator(1, 0, get_unique_id())
    tp = TensorParallel(comm, 256, 256)
    x = torch.empty(rows * K + off, dtype=torch.bfloat16, device="cuda")[off:].view(rows, K)
    x.copy_(torch.randn(rows, K, device="cuda") * torch.rand(rows, 1, device="cuda"))
    x[0, :128] = 0
    q = torch.full((rows + 1, K), 1.0, device="cuda").to(torch.float8_e4m3fn)
    q, s = tp.quantize_fp8(x, q=q)
    amax = x.float().view(rows, -1, 128).abs().amax(-1).clamp_min(1e-10)
    scale = (amax.double() / 448).float()
    want = (x.float().view(rows, -1, 128) * (1 / scale.double()).float().unsqueeze(-1)).view(rows, K).to(torch.float8_e4m3fn)
    assert torch.equal(s.t(), scale)
    assert torch.equal(q[:rows].view(torch.uint8), want.view(torch.uint8)) and (q[rows].float() == 1).all()
    tp.destroy()
    comm.destroy()
