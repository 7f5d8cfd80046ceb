"""Every tile form of the BF16 GEMM (csrc/mixed_ops.cu), forced for all three stages
of the local matvec, against the fused matvec: the same MMA steps in the same K
order, so the same bits.  The forms differ in their output types too: stages 1
and 2 write BF16, stage 3 FP32."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# one tile; fewer tiles than SMs; tile counts that no grid divides, with row and
# column remainders; packed stores and not; one K step and many
SHAPES = [(1, 1, 1, 1, 1), (4, 4, 4, 1, 1), (7, 12, 4, 3, 1), (64, 64, 2, 3, 3),
          (33, 17, 65, 3, 2), (61, 64, 59, 3, 3), (130, 16, 129, 2, 3), (256, 64, 260, 3, 3),
          (258, 62, 255, 3, 2), (401, 36, 300, 2, 2), (300, 64, 200, 3, 3), (512, 8, 512, 5, 5)]

CHILD = r"""
import os, sys
import numpy as np
sys.path[:0] = [os.path.join(os.environ["ROOT"], "tt-toolbox_b200")]
import ttgpu
ctx = ttgpu.Context(int(os.environ.get("TTG_DEVICE", "0")))
out = []
for (rx1, n, rx2, ra1, ra2) in eval(os.environ["SHAPES"]):
    rng = np.random.default_rng(rx1 + 7 * rx2 + n)
    Phi1 = rng.standard_normal((rx1, rx1, ra1)); A = rng.standard_normal((ra1, n, n, ra2))
    Phi2 = rng.standard_normal((rx2, ra2, rx2)); x = rng.standard_normal(rx1 * n * rx2)
    out.append(ttgpu.bfun3(Phi1, A, Phi2, x, ctx=ctx, precision="mixed"))
# the kernels of one more matvec, by name
import torch
from torch.profiler import ProfilerActivity, profile
torch.cuda.synchronize()
with profile(activities=[ProfilerActivity.CUDA]) as prof:
    ttgpu.bfun3(Phi1, A, Phi2, x, ctx=ctx, precision="mixed")
    torch.cuda.synchronize()
print("\n".join(e.key for e in prof.key_averages()))
np.savez(os.environ["OUT"], *out)
"""


def _run(path, **env):
    env = dict(os.environ, ROOT=ROOT, SHAPES=repr(SHAPES), OUT=str(path), **env)
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    with np.load(path) as f:
        return [f[k] for k in f.files], r.stdout


@pytest.fixture(scope="module")
def fused(tmp_path_factory):
    return _run(tmp_path_factory.mktemp("fused") / "out.npz", TTG_FUSED_MV="1")[0]


@pytest.mark.parametrize("tile,kernel", [
    ("64", "k_umma_gemm<64"), ("128", "k_umma_gemm<128"), ("256", "k_umma_gemm<256"),
    ("p192", "k_umma_pers<192"), ("p256", "k_umma_pers<256")])
def test_forced_tile_gives_the_same_bits(fused, tmp_path, tile, kernel):
    got, kernels = _run(tmp_path / "out.npz", TTG_FUSED_MV="0", TTG_AUTOTUNE=tile)
    ran = {k.split("k_umma")[1].split(",")[0] for k in kernels.splitlines() if "k_umma" in k}
    assert ran == {kernel[len("k_umma"):]}, kernels
    for shape, a, b in zip(SHAPES, fused, got):
        assert np.array_equal(a, b), shape
