"""Grouped batches of local systems whose cooperative Krylov grids fill the device
(csrc/group.cu, gmres.cu, mixed.cu): two systems in the same phase go out as one
launch whose CTAs are all resident, and each gets what it gets alone."""
import numpy as np
import pytest

import ttgpu
from ttgpu import workloads

pytestmark = pytest.mark.gpu


def _solve(ctx, n, precision, count=2, sms=0):
    """Equal systems of n^3 unknowns in the middle core, one sweep; and one alone."""
    A, y, _, z0 = workloads.aniso(d=3, n=n, rhs_rank=n, seed=5, react_scale=50.0)
    x0 = ttgpu.TensorTrain.from_cores(
        workloads.randn_cores(n, 3, n, np.random.default_rng(6), scale=0.1))
    opts = dict(nswp=1, rmax=n, precision=precision)
    ctx.set_option(ttgpu.Context.OPT_GROUP_SMS, sms)
    stats, gs = [], {}
    try:
        xs = ttgpu.amen_solve2_batch([A] * count, [y] * count, 1e-6, x0s=[x0] * count,
                                     z0s=[z0] * count, ctx=ctx, stats=stats, grouped=True,
                                     group_stats=gs, **opts)
    finally:
        ctx.set_option(ttgpu.Context.OPT_GROUP_SMS, 0)
    assert all(s["status"] == 0 for s in stats)
    lone = ttgpu.amen_solve2(A, y, 1e-6, x0=x0, z0=z0, ctx=ctx, **opts)
    return xs, lone, gs


# FP64 grids take a CTA per 256 unknowns (141 and, at the limit of a share, 148),
# mixed ones a CTA per 1024 (148).
CASES = [("fp64", 33), ("fp64", 40), ("mixed", 56)]


@pytest.mark.parametrize("precision,n", CASES)
def test_two_large_systems_share_every_launch(ctx, precision, n):
    """Both systems record the same kernels, so every grouped step has two
    members, and one launch when their grids fit together."""
    xs, _, gs = _solve(ctx, n, precision)
    assert np.array_equal(xs[0].core, xs[1].core)
    assert max(xs[0].r) >= n - 1  # the middle system was as large as meant
    steps = gs["launches"] - (gs["records"] - gs["grouped_records"])
    assert gs["grouped_records"] > 0 and 2 * steps == gs["grouped_records"], gs


@pytest.mark.parametrize("precision,n", CASES)
def test_large_systems_as_alone(ctx, precision, n):
    """With grids sized from the whole device (up to two CTAs per SM each, more
    than fit side by side) the systems still get the bits of a batch of one,
    and of a lone solve where that takes the same SVDs (ranks below 48)."""
    xs, lone, _ = _solve(ctx, n, precision, sms=4096)
    (one,), _, _ = _solve(ctx, n, precision, count=1, sms=4096)
    for x in xs:
        for ref in [one] + ([lone] if n < 48 else []):
            assert list(x.r) == list(ref.r)
            assert np.array_equal(x.core, ref.core)
