"""<x, A x> gradients whose products are too long to gain from sharing a launch
(csrc/kernels_f64.cu): they run one by one, shorter ones beside them in pairs."""
import numpy as np
import pytest

import ttgpu
from oracle import grad as og

pytestmark = pytest.mark.gpu


def _problem(n, r, ra):
    rng = np.random.default_rng(sum(n) + sum(r))
    xs = [np.asfortranarray(rng.standard_normal((r[k], n[k], r[k + 1]))) / np.sqrt(r[k] * n[k])
          for k in range(len(n))]
    As = [np.asfortranarray(rng.standard_normal((ra[k], n[k], n[k], ra[k + 1])))
          for k in range(len(n))]
    return xs, As


def _launches(ctx, n, r, ra):
    xs, As = _problem(n, r, ra)
    x, A = ttgpu.TensorTrain.from_cores(xs), ttgpu.TTMatrix.from_cores(As)
    ttgpu.grad_xAx(x, A, ctx=ctx)
    before = ctx.launch_count()
    ttgpu.grad_xAx(x, A, ctx=ctx)
    return ctx.launch_count() - before


def test_long_products_run_one_by_one(ctx):
    """Four cores: of 16, rank 16, every pair shares; the six products of two
    inner cores of 48 and rank 128 (1.2 GFLOP a pair and more) do not."""
    short = _launches(ctx, [16] * 4, [1, 16, 16, 16, 1], [1, 2, 2, 2, 1])
    long_ = _launches(ctx, [48] * 4, [1, 128, 128, 128, 1], [1, 3, 3, 3, 1])
    assert long_ >= short + 4


# the work of the inner core's pairs on either side of the limit
@pytest.mark.parametrize("n,r,ra", [
    ([20, 32, 20], [1, 79, 80, 1], [1, 3, 3, 1]),
    ([20, 32, 20], [1, 90, 88, 1], [1, 3, 3, 1]),
    ([24, 33, 24], [1, 97, 101, 1], [1, 3, 3, 1]),
    ([40, 48, 40], [1, 128, 130, 1], [1, 2, 3, 1])])
def test_matches_the_oracle(ctx, n, r, ra):
    xs, As = _problem(n, r, ra)
    v, G = ttgpu.grad_xAx(ttgpu.TensorTrain.from_cores(xs), ttgpu.TTMatrix.from_cores(As), ctx=ctx)
    vref, Gref = og.xAx(xs, As)
    ref = np.concatenate([g.ravel(order="F") for g in Gref])
    # the bounds of tests/test_gpu_grad.py
    assert np.linalg.norm(G.core - ref) <= 1e-11 * np.linalg.norm(ref)
    scale = np.linalg.norm(xs[0]) * np.linalg.norm(Gref[0])
    assert abs(v - vref) <= 1e-12 * max(abs(vref), scale)
