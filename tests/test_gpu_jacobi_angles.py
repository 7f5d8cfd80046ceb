"""Angles of the block Jacobi SVDs (csrc/small_dense.cu): a pair of columns that
no other column meets takes one rotation, so a matrix of such pairs is done in
one sweep, and the second finds nothing above the stopping threshold (4 eps of
the column norms; the rounding of one rotation is about one eps)."""
import numpy as np
import pytest

import ttgpu

pytestmark = pytest.mark.gpu


@pytest.fixture
def two_sweeps(ctx):
    ctx.set_option(ttgpu.Context.OPT_JACOBI_MAX_SWEEPS, 2)
    yield ctx
    ctx.set_option(ttgpu.Context.OPT_JACOBI_MAX_SWEEPS, 40)


# one CTA (up to 47 columns outside a batch) and cluster; pairs within a block
# of 8 columns and across the matrix's blocks
@pytest.mark.parametrize("n", [10, 16, 40, 46, 64, 96, 128, 250, 256])
@pytest.mark.parametrize("across", [False, True])
@pytest.mark.parametrize("ratio", [1.0, 1e-3])
def test_disjoint_pairs_take_one_rotation(two_sweeps, n, across, ratio):
    g = np.random.default_rng(n)
    A = np.zeros((n, n))
    h = n // 2
    for i in range(h):
        p, q = (i, i + h) if across else (2 * i, 2 * i + 1)
        A[p, p] = 1.0 + g.random()
        A[p, q] = ratio * (0.1 + g.random())
        A[q, q] = ratio * (1.0 + g.random())
    U, s, VT = ttgpu.dense_svd(A, ctx=two_sweeps)
    assert np.linalg.norm(U * s @ VT - A) <= 1e-15 * n * np.linalg.norm(A)
    assert np.allclose(s, np.linalg.svd(A, compute_uv=False), rtol=0, atol=1e-15 * n * s[0])
