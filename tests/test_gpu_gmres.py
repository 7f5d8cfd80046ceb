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


# row counts of every remainder by the four-row groups, below and above one
# group; systems smaller than the restart; more than one block (1024 rows);
# a two-eigenvalue operator, whose Krylov space ends after two steps
@pytest.mark.parametrize("rx1,n,rx2,spread", [
    (1, 1, 1, 0.2), (1, 3, 1, 0.2), (1, 5, 1, 0.2), (2, 3, 1, 0.2), (3, 5, 9, 0.2),
    (11, 10, 11, 0.2), (13, 17, 15, 0.2), (29, 21, 31, 0.2), (8, 8, 17, 0.0)])
def test_mixed_solve_meets_its_tolerance(ctx, rx1, n, rx2, spread):
    rng = np.random.default_rng(rx1 + 7 * n + 31 * rx2)
    Phi1 = np.zeros((rx1, rx1, 1))
    Phi1[:, :, 0] = np.diag(np.where(np.arange(rx1) % 2, 1.0, 2.0))
    A = np.zeros((1, n, n, 1))
    A[0, :, :, 0] = np.eye(n) + spread * rng.standard_normal((n, n)) / max(n, 2)
    Phi2 = np.zeros((rx2, 1, rx2))
    Phi2[:, 0, :] = np.eye(rx2) + spread * rng.standard_normal((rx2, rx2)) / max(rx2, 2)
    sz = rx1 * n * rx2
    rhs, tol = rng.standard_normal(sz), 1e-9
    x = ttgpu.solve3d_2(Phi1, A, Phi2, rhs, tol, 1, np.zeros(sz), 0, 40, 2, 0, ctx=ctx,
                        precision="mixed")
    r = rhs - oamen.bfun3(Phi1, A, Phi2, x)
    # the solver stops on its own FP64 residual, which rounds at 1e-13 at most
    assert np.linalg.norm(r) <= (tol + 1e-12) * np.linalg.norm(rhs)
