"""Cholesky QR (csrc/linalg.cu on k_chol_inv) at the edges of its 8-column
steps and 96-column blocks, through the SVD of tall matrices that take it."""
import numpy as np
import pytest

import ttgpu

pytestmark = pytest.mark.gpu


# (m, n): m n above what one CTA's Householder QR holds, m >= 4 n
@pytest.mark.parametrize("m,n", [(3000, 9), (2000, 15), (2000, 16), (1601, 17), (700, 63),
                                 (640, 64), (500, 65), (383, 95), (384, 96), (400, 97),
                                 (450, 104), (1000, 193), (900, 200)])
@pytest.mark.parametrize("decades", [0, 9])
def test_tall_svd(ctx, m, n, decades):
    g = np.random.default_rng(m + n)
    A = g.standard_normal((m, n))
    if decades:
        A = (np.linalg.qr(A)[0] * 10.0 ** -np.linspace(0, decades, n)) @ np.linalg.qr(
            g.standard_normal((n, n)))[0]
    U, s, VT = ttgpu.dense_svd(A, ctx=ctx)
    tol, orth = max(1e-13, 4e-16 * n), max(1e-12, 4e-16 * n ** 1.5)
    assert np.linalg.norm(U * s @ VT - A) <= tol * np.linalg.norm(A)
    assert np.linalg.norm(U.T @ U - np.eye(n)) < orth
    assert np.linalg.norm(VT @ VT.T - np.eye(n)) < orth


@pytest.mark.parametrize("scale", [1e-40, 1e40])
def test_scale_beyond_single_precision(ctx, scale):
    """Pivots of 1e-80 and 1e80: the reciprocal roots leave single precision."""
    A = np.random.default_rng(1).standard_normal((1200, 40)) * scale
    U, s, VT = ttgpu.dense_svd(A, ctx=ctx)
    assert np.linalg.norm(U * s @ VT - A) <= 1e-13 * np.linalg.norm(A)
    assert np.linalg.norm(U.T @ U - np.eye(40)) < 1e-12


def test_rank_deficient_falls_back(ctx):
    """Exactly dependent columns break the unshifted passes: the orthogonality
    check sends them to the Householder path."""
    g = np.random.default_rng(2)
    B = g.standard_normal((1500, 20))
    A = np.hstack([B, B[:, :7] @ g.standard_normal((7, 10))])
    U, s, VT = ttgpu.dense_svd(A, ctx=ctx)
    assert np.linalg.norm(U * s @ VT - A) <= 1e-13 * np.linalg.norm(A)
    assert np.linalg.norm(VT @ VT.T - np.eye(30)) < 1e-12
