"""Block-scaled fp8 GEMM in both tile widths and with the K blocks shared by clusters of 2 to 8 CTAs, against a 64-bit product: uneven
shares, fewer K blocks than CTAs, more tiles than CTAs."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPES = [(128, 256, 128), (256, 256, 1152), (128, 768, 640), (384, 1280, 2176), (128, 2048, 7168), (640, 2304, 1024), (2048, 2560, 384), (1920, 4096, 512),
          (1152, 3328, 896)]


def _run(width, split):
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.tp import TensorParallel
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    tp = TensorParallel(comm, 4096, 4096)
    for M, N, K in SHAPES:
        g = torch.Generator(device="cuda").manual_seed(M + N + K)
        xq, xs = tp.quantize_fp8((torch.randn(M, K, device="cuda", generator=g) * torch.rand(M, 1, device="cuda", generator=g) * 4).bfloat16())
        w = torch.randn(N, K, device="cuda", generator=g) * 0.05
        # the scale of W differs from block to block
        w *= 2.0 ** torch.randint(-3, 4, (N // 128, 1, K // 128, 1), device="cuda", generator=g).expand(-1, 128, -1, 128).reshape(N, K)
        wq, ws = tp.quantize_fp8(w.bfloat16(), 128)
        xd = (xq.double().view(M, -1, 128) * xs.t().double().unsqueeze(-1)).view(M, K)
        wd = (wq.double().view(N // 128, 128, -1, 128) * ws.t().double()[:, None, :, None]).view(N, K)
        ref = xd @ wd.t()
        # bf16 rounds to 2^-9 of the value; the sums are fp32 over K terms of at most the row's and column's size
        bound = 2 ** -8 * ref.abs() + 2 ** -20 * (xd.abs() @ wd.abs().t())
        out = torch.full((M + 1, N), 9.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):
            out[:M].zero_()
            tp.gemm_fp8(xq, xs, wq, ws, out=out[:M])
            torch.cuda.synchronize()
            assert ((out[:M].double() - ref).abs() <= bound).all(), (M, N, K, width, split)
            assert (out[M] == 9).all()
    assert comm.async_error() == 0
    tp.destroy()
    comm.destroy()
    print("shapes ok")


# width 0 and split 0: what the rule takes
@pytest.mark.parametrize("width,split", [(0, 0), (256, 1), (128, 1), (256, 2), (256, 8), (128, 2), (128, 3), (128, 4), (128, 7)])
def test_fp8_forms(width, split):
    if not torch.cuda.is_available() or torch.cuda.get_device_capability()[0] < 10:
        pytest.skip("needs sm_100")
    env = dict(os.environ, NCCL_B200_TP_FP8_WIDTH=str(width), NCCL_B200_TP_FP8_SPLIT=str(split))
    r = subprocess.run([sys.executable, os.path.abspath(__file__), str(width), str(split)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "shapes ok" in r.stdout, r.stdout + r.stderr


if __name__ == "__main__":
    _run(int(sys.argv[1]), int(sys.argv[2]))
