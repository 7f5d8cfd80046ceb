"""The BF16 GEMM's persistent form and packed stores (csrc/mixed_ops.cu) against
the fused matvec, which keeps one 2-byte store per element and tiles of at most
128 columns: the same MMA steps in the same K order, so the same bits.  Shapes
of many tiles, for which the tile autotuner weighs the persistent form: rows
that come in aligned fours (packed) and not, column remainders, few K steps."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHAPES = [(256, 64, 260, 3, 3), (258, 62, 255, 3, 2), (96, 128, 512, 2, 3), (401, 36, 300, 2, 2),
          (512, 8, 512, 5, 5), (64, 64, 2, 3, 3), (4, 4, 4, 1, 1), (7, 12, 4, 3, 1)]

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
np.savez(os.environ["OUT"], *out)
"""


def _run(fused, path):
    env = dict(os.environ, ROOT=ROOT, SHAPES=repr(SHAPES), OUT=str(path),
               TTG_FUSED_MV="1" if fused else "0")
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    with np.load(path) as f:
        return [f[k] for k in f.files]


def test_same_bits_as_the_fused_form(tmp_path):
    for shape, a, b in zip(SHAPES, _run(True, tmp_path / "f.npz"), _run(False, tmp_path / "s.npz")):
        assert np.array_equal(a, b), shape
