"""Plain bf16 GEMMs off the beaten tile counts: the K dimension shared by clusters of 2 to 8 CTAs (uneven shares, column chunks
that do not divide evenly over the cluster), and pairs of CTAs whose last row tile is half empty; against a 64-bit product."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# with the largest cluster: tiles x shares 2x8 (K 66 blocks), 1x7 (61 blocks), 5x3, 22x6, 29x5, 32x4, 40x3; where the split begins 1x1 (23
# blocks) and 1x3 (24 blocks) instead of one CTA, 64x1 (15 blocks) and 64x2 (16 blocks) instead of pairs; 1x1 further below;
# without clusters: the one-CTA and the pair kernel, the latter also where the rows end inside a tile (the last three)
SHAPES = [(256, 256, 4224), (128, 256, 3904), (128, 256, 960), (128, 256, 1024), (128, 256, 1472), (128, 256, 1536), (128, 1280, 1664), (128, 5632, 3200),
          (128, 7424, 2752), (128, 8192, 2048), (640, 2048, 1600), (256, 8192, 960), (256, 8192, 1024), (256, 8192, 1088), (1920, 5120, 320),
          (4224, 4096, 192), (1920, 5120, 1536), (4224, 4096, 1024), (384, 8192, 4096)]


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
        out = torch.full((M + 1, N), 9.0, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):
            out[:M].zero_()
            tp.gemm(x, w, out=out[:M])
            torch.cuda.synchronize()
            # bf16 rounds to 2^-9 of the value; the sums are fp32 over K terms of at most the row's and column's size
            bound = 2 ** -8 * ref.abs() + 2 ** -20 * (x.double().abs() @ w.double().abs().t())
            assert ((out[:M].double() - ref).abs() <= bound).all(), (M, N, K)
            assert (out[M] == 9).all()
    assert comm.async_error() == 0
    tp.destroy()
    comm.destroy()
    print("shapes ok")


@pytest.mark.parametrize("split,pair", [("8", "1"), ("1", "1"), ("1", "0"), ("3", "1")])
def test_gemm_shapes(split, pair):
    if not torch.cuda.is_available() or torch.cuda.get_device_capability()[0] < 10:
        pytest.skip("needs sm_100")
    env = dict(os.environ, NCCL_B200_TP_SPLIT=split, NCCL_B200_TP_PAIR=pair)
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "shapes ok" in r.stdout, r.stdout + r.stderr


if __name__ == "__main__":
    _run()
