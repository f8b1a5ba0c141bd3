"""Plain bf16 GEMMs in every tile width, on one CTA and on pairs, against a 64-bit product: last tiles that hang over N by all but 32 columns
and by few, half empty row tiles, more tiles than CTAs, one K step; and the shapes that the rule gives each width and to clusters on narrow
tiles."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPES = [(128, 256, 64), (256, 256, 128), (384, 1280, 192), (512, 2304, 320), (2048, 4096, 64), (2176, 2304, 1024), (128, 512, 448),
          # by rule: 128 columns with 4 shares of K on 4 CTAs, 8 on 8, 6 on 4, 4 on 2 and 2 on one; 160; pairs of 192; pairs of 224; 192
          (128, 1024, 2048), (128, 1024, 7168), (128, 4096, 4096), (128, 8192, 2112), (512, 4096, 1024), (2048, 2560, 1024), (768, 8192, 1024),
          (2560, 3072, 1024), (1792, 3328, 512), (1152, 2304, 1600)]


def _run():
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    from nccl_b200 import Communicator, get_unique_id
    from nccl_b200.ops.tp import TensorParallel
    torch.cuda.set_device(0)
    comm = Communicator(1, 0, get_unique_id())
    tp = TensorParallel(comm, 4096, 4096)
    for M, N, K in SHAPES:
        g = torch.Generator(device="cuda").manual_seed(M + N + K)
        x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
        ref = x.double() @ w.double().t()
        # bf16 rounds to 2^-9 of the value; the sums are fp32 over K terms of at most the row's and column's size
        bound = 2 ** -8 * ref.abs() + 2 ** -20 * (x.double().abs() @ w.double().abs().t())
        out = torch.full((M + 1, N), 9.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):
            out[:M].zero_()
            tp.gemm(x, w, out=out[:M])
            torch.cuda.synchronize()
            assert ((out[:M].double() - ref).abs() <= bound).all(), (M, N, K)
            assert (out[M] == 9).all()
    assert comm.async_error() == 0
    tp.destroy()
    comm.destroy()
    print("shapes ok")


@pytest.mark.parametrize("width,split,pair", [("0", "8", "1"), ("0", "3", "1"), ("0", "8", "0")] + [(w, "1", p) for w in ("256", "224", "192", "160", "128") for p in "01"])
def test_gemm_widths(width, split, pair):
    if not torch.cuda.is_available() or torch.cuda.get_device_capability()[0] < 10:
        pytest.skip("needs sm_100")
    env = dict(os.environ, NCCL_B200_TP_WIDTH=width, NCCL_B200_TP_SPLIT=split, NCCL_B200_TP_PAIR=pair)
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "shapes ok" in r.stdout, r.stdout + r.stderr


if __name__ == "__main__":
    _run()
