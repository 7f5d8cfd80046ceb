"""The one-CTA block Jacobi SVD (csrc/small_dense.cu) over the sizes that a lone call
gives to the cluster form: 48 to 96 columns, three to six block pairs, some with
idle warps, up to the largest shared memory.  A grouped batch runs them."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = [47, 48, 49, 63, 64, 65, 79, 80, 81, 95, 96]

CHILD = r"""
import os, sys
import numpy as np
sys.path[:0] = [os.path.join(os.environ["ROOT"], "tt-toolbox_b200")]
import ttgpu
ctx = ttgpu.Context(int(os.environ.get("TTG_DEVICE", "0")))
inp = np.load(os.environ["IN"])
out = {}
for k in inp.files:
    for f, v in zip("usv", ttgpu.dense_svd(inp[k], ctx=ctx)):
        out[k + "." + f] = v
np.savez(os.environ["OUT"], **out)
"""


def _inputs():
    out = {}
    for n in SIZES:
        g = np.random.default_rng(n)
        G = g.standard_normal((n, n))
        out["gauss%d" % n] = G
        Q1, _ = np.linalg.qr(g.standard_normal((n, n)))
        Q2, _ = np.linalg.qr(g.standard_normal((n, n)))
        out["graded%d" % n] = (Q1 * 10.0 ** -np.linspace(0, 12, n)) @ Q2
        C = G * 10.0 ** -np.linspace(0, 60, n)  # columns over 60 decades, two almost parallel
        C[:, 3] = C[:, 2] * (1.0 + 1e-9) + 1e-12 * C[:, 5]
        out["columns%d" % n] = C
        out["small%d" % n] = G * 1e-60
        out["large%d" % n] = G * 1e60
    return out


def test_sizes_of_the_cluster_form(tmp_path):
    inp = _inputs()
    np.savez(tmp_path / "in.npz", **inp)
    env = dict(os.environ, ROOT=ROOT, IN=str(tmp_path / "in.npz"), OUT=str(tmp_path / "out.npz"),
               TTG_JACOBI_CLUSTER_MIN_N="1000")
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    with np.load(tmp_path / "out.npz") as out:
        for k, A in inp.items():
            n = A.shape[0]
            U, s, VT = (out[k + "." + f] for f in "usv")
            # a one-sided Jacobi SVD with n columns: backward error n eps,
            # orthogonality eps n^1.5
            tol, orth = max(1e-13, 4e-16 * n), max(1e-12, 4e-16 * n ** 1.5)
            sr = np.linalg.svd(A, compute_uv=False)
            assert np.allclose(s, sr, rtol=0, atol=tol * sr[0]), k
            assert np.all(np.diff(s) <= 0), k
            assert np.linalg.norm(U * s @ VT - A) <= tol * np.linalg.norm(A), k
            assert np.linalg.norm(VT @ VT.T - np.eye(n)) < orth, k
            keep = s > 0
            assert np.linalg.norm(U[:, keep].T @ U[:, keep] - np.eye(int(keep.sum()))) < orth, k
