"""<x, A x> where the device has no room for the intermediates that its two sweeps
keep (csrc/grad.cu): the sweeps then follow one another in two buffers of the
largest core, and the call succeeds with the same gradient."""
import os

import numpy as np
import pytest
import torch

import ttgpu

pytestmark = pytest.mark.gpu


def _cores(rng, shapes, scale):
    return [np.asfortranarray(rng.standard_normal(s) * scale(s)) for s in shapes]


def test_nearly_full_device():
    """The middle core's intermediates are 0.61 GB each: four are kept (0.67 GB
    each in the pool's size classes), two suffice; 2.1 GB are free."""
    rng = np.random.default_rng(11)
    n, r, ra = [4, 172, 4], [1, 384, 384, 1], [1, 3, 3, 1]
    x = ttgpu.TensorTrain.from_cores(_cores(
        rng, [(r[k], n[k], r[k + 1]) for k in range(3)], lambda s: (s[0] * s[1]) ** -0.5))
    A = ttgpu.TTMatrix.from_cores(_cores(
        rng, [(ra[k], n[k], n[k], ra[k + 1]) for k in range(3)], lambda s: 1.0))
    dev = int(os.environ.get("TTG_DEVICE", "0"))
    c = ttgpu.Context(dev)
    vref, ref = ttgpu.grad_xAx(x, A, ctx=c)
    c.close()
    c = ttgpu.Context(dev)
    dx, dA = ttgpu.DeviceTT.upload(c, x), ttgpu.DeviceTT.upload(c, A)
    free = torch.cuda.mem_get_info(dev)[0]
    ballast = torch.empty(free - int(2.1 * 1e9), dtype=torch.uint8, device="cuda:%d" % dev)
    try:
        v, g = ttgpu.grad_xAx(dx, dA, ctx=c)
    finally:
        del ballast
        torch.cuda.empty_cache()
        dx.free()
        dA.free()
        c.close()
    # the same sums in another split of their terms
    assert np.linalg.norm(g.core - ref.core) <= 1e-11 * np.linalg.norm(ref.core)
    assert abs(v - vref) <= 1e-11 * np.linalg.norm(ref.core) * np.linalg.norm(x.core)
