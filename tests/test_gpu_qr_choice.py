"""Which one-CTA Householder QR a shape takes (csrc/small_dense.cu): a few
reflectors go one at a time, more in panels of eight columns; LAPACK's factors
from both, on either side of the line."""
import os
import subprocess
import sys

import numpy as np
import pytest

import ttgpu

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SINGLE = [(1, 1), (64, 1), (512, 1), (1, 64), (1, 512), (2, 2), (2, 300), (2000, 2), (3, 3),
          (3, 4), (4, 3), (3, 256), (256, 3)]
BLOCKED = [(257, 3), (1000, 3), (4, 4), (4, 64), (64, 4), (9, 9)]

CHILD = r"""
import os, sys
import numpy as np
sys.path[:0] = [os.path.join(os.environ["ROOT"], "tt-toolbox_b200")]
import ttgpu, torch
from torch.profiler import ProfilerActivity, profile
ctx = ttgpu.Context(int(os.environ.get("TTG_DEVICE", "0")))
for group in eval(os.environ["SHAPES"]):
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for m, n in group:
            ttgpu.dense_qr(np.ones((m, n)) + np.eye(m, n), ctx=ctx)
        torch.cuda.synchronize()
    keys = [e.key for e in prof.key_averages()]
    print("single", sum("k_house_qr_body" in k for k in keys),
          "blocked", sum("k_house_qr_blk_body" in k for k in keys))
"""


def test_kernel_of_each_shape():
    env = dict(os.environ, ROOT=ROOT, SHAPES=repr([SINGLE, BLOCKED]))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    lines = [q for q in r.stdout.splitlines() if q.startswith("single")]
    assert lines == ["single 1 blocked 0", "single 0 blocked 1"]


@pytest.mark.parametrize("m,n", SINGLE + BLOCKED)
def test_matches_lapack(ctx, m, n):
    A = np.random.default_rng(m + 1000 * n).standard_normal((m, n))
    Q, R = ttgpu.dense_qr(A, ctx=ctx)
    Rr = np.linalg.qr(A)[1]
    k = min(m, n)
    assert np.linalg.norm(Q @ R - A) <= 1e-14 * np.linalg.norm(A)
    assert np.linalg.norm(Q.T @ Q - np.eye(k)) <= 1e-15 * (k + 10)
    assert np.linalg.norm(R - Rr) <= 1e-11 * np.linalg.norm(Rr)
