"""The tile width of a plain bf16 GEMM changes neither its sums nor their order: what the rule takes gives the same bits as tiles of 256
columns, where K is one sum and where it is summed in shares (more, as many and fewer CTAs to a tile than shares, one CTA with all of them;
shares of unequal length)."""
import hashlib
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

SHAPES = [(128, 8192, 8192), (128, 4096, 4096), (128, 1024, 2048), (128, 1024, 7168), (128, 1280, 3904), (128, 2048, 6144), (256, 4352, 3200), (128, 5632, 3200),
          (128, 7424, 2752), (640, 2048, 1600), (512, 4096, 1024), (256, 8192, 1088), (768, 2560, 4160), (384, 4096, 7168), (128, 256, 4224),
          (1152, 2304, 1600), (2048, 2560, 1024), (1280, 4096, 3584), (2560, 3072, 1024)]


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
        outs = [tp.gemm(x, w) for _ in range(3)]
        assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2]), (M, N, K)
        print("sums", M, N, K, hashlib.sha1(outs[0].view(torch.int16).cpu().numpy().tobytes()).hexdigest())
    tp.destroy()
    comm.destroy()


def test_width_leaves_the_sums_alone():
    if not torch.cuda.is_available() or torch.cuda.get_device_capability()[0] < 10:
        pytest.skip("needs sm_100")
    got = []
    for width in ("0", "256"):
        r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, NCCL_B200_TP_WIDTH=width), capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        got.append([line for line in r.stdout.splitlines() if line.startswith("sums")])
    assert len(got[0]) == len(SHAPES) and got[0] == got[1]


if __name__ == "__main__":
    _run()
