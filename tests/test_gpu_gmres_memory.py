"""Device memory of the FP64 Householder GMRES (csrc/gmres.cu) at a long restart:
the basis and one square array of the restart's size (the triangular factor of
the least-squares problem and the WY factor share it), as with reflectors
applied one by one."""
import os

import numpy as np
import pytest
import torch

import ttgpu
from oracle import amen as oamen

pytestmark = pytest.mark.gpu


def test_long_restart_holds_one_square():
    rx1, n, rx2, nrestart = 14, 20, 15, 4096
    rng = np.random.default_rng(2)
    Phi1 = 1e-3 * rng.standard_normal((rx1, rx1, 1)) + np.eye(rx1)[:, :, None]
    A = 1e-3 * rng.standard_normal((1, n, n, 1)) + np.eye(n)[None, :, :, None]
    Phi2 = 1e-3 * rng.standard_normal((rx2, 1, rx2)) + np.eye(rx2)[:, None, :]
    sz = rx1 * n * rx2
    rhs, prev = rng.standard_normal(sz), np.zeros(sz)
    dev = int(os.environ.get("TTG_DEVICE", "0"))
    c = ttgpu.Context(dev)
    try:
        # kernels and small pools first
        ttgpu.solve3d_2(Phi1, A, Phi2, rhs, 1e-10, 1, prev, 0, 8, 4, 0, ctx=c)
        free = torch.cuda.mem_get_info(dev)[0]
        x = ttgpu.solve3d_2(Phi1, A, Phi2, rhs, 1e-10, 1, prev, 0, nrestart, 1, 0, ctx=c)
        grown = free - torch.cuda.mem_get_info(dev)[0]
    finally:
        c.close()
    assert np.linalg.norm(rhs - oamen.bfun3(Phi1, A, Phi2, x)) <= 1e-9 * np.linalg.norm(rhs)
    # two blocks, each at most a quarter above its request, and 128 MB of slabs
    basis, square = 8 * sz * (nrestart + 1), 8 * (nrestart + 1) ** 2
    assert grown <= 1.25 * (basis + square) + 128e6
