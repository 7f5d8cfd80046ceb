"""Householder GMRES in compact WY form (csrc/gmres.cu) at the edges of its row
and column splits, against the oracle's reflector-by-reflector dgmresr_hh."""
import numpy as np
import pytest

import ttgpu
from oracle import amen as oamen

pytestmark = pytest.mark.gpu


# sizes: a 1 x 1 system; restarts that exhaust the space; one row past a
# block's least share (256 rows) and past two of them; more columns than warps
# take at once; restarts beyond the staged back-substitution (64); uneven
# splits of the rows over more than one block per SM
@pytest.mark.parametrize("rx1,n,rx2,nrestart,niters", [
    (1, 1, 1, 40, 2), (1, 2, 1, 1, 1), (2, 4, 2, 40, 2), (1, 257, 1, 3, 2), (3, 19, 9, 7, 2),
    (5, 6, 7, 210, 1), (9, 11, 10, 65, 1), (4, 33, 5, 130, 1), (37, 61, 41, 12, 2)])
def test_gmres_matches_oracle(ctx, rx1, n, rx2, nrestart, niters):
    rng = np.random.default_rng(rx1 + 7 * n + 31 * rx2)
    ra = 2
    Phi1 = rng.standard_normal((rx1, rx1, ra)) / max(rx1, 2)
    A = rng.standard_normal((ra, n, n, ra)) / max(n, 2)
    Phi2 = rng.standard_normal((rx2, ra, rx2)) / max(rx2, 2)
    # a dominant identity term keeps the system well conditioned, so that both
    # solvers' rounding stays far below the bound
    Phi1[:, :, 0] += 2.0 * np.eye(rx1)
    A[0, :, :, 0] += 2.0 * np.eye(n)
    Phi2[:, 0, :] += 2.0 * np.eye(rx2)
    sz = rx1 * n * rx2
    rhs = rng.standard_normal(sz)
    prev = 0.01 * rng.standard_normal(sz)
    st, info = {}, {}
    ref = oamen.solve3d_2(Phi1, A, Phi2, rhs, 1e-12, prev, nrestart, niters, st)
    got = ttgpu.solve3d_2(Phi1, A, Phi2, rhs, 1e-12, 1, prev, 0, nrestart, niters, 0, ctx=ctx,
                          info=info)
    assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref)
