"""Block Jacobi SVDs (csrc/small_dense.cu: one CTA, and a cluster) at the edges of
their blocks of 8 columns, pairs of 16 and cluster sizes, on spectra and
scales that their single-precision angles have to stand."""
import numpy as np
import pytest

import ttgpu

pytestmark = pytest.mark.gpu

SIZES = [9, 15, 16, 17, 24, 31, 32, 33, 47, 48, 49, 57, 64, 65, 112, 113, 127, 128, 129, 240,
         241, 255, 256]


def _check(A, U, s, VT):
    n = A.shape[0]
    sr = np.linalg.svd(A, compute_uv=False)
    # the bounds of a one-sided Jacobi SVD with n columns: backward error n eps,
    # orthogonality eps n^1.5
    tol, orth = max(1e-13, 4e-16 * n), max(1e-12, 4e-16 * n ** 1.5)
    assert np.allclose(s, sr, rtol=0, atol=tol * sr[0])
    assert np.all(np.diff(s) <= 0)
    assert np.linalg.norm(U * s @ VT - A) <= tol * np.linalg.norm(A)
    assert np.linalg.norm(VT @ VT.T - np.eye(n)) < orth
    keep = s > 0
    assert np.linalg.norm(U[:, keep].T @ U[:, keep] - np.eye(int(keep.sum()))) < orth


@pytest.mark.parametrize("n", SIZES)
def test_gaussian(ctx, n):
    A = np.random.default_rng(n).standard_normal((n, n))
    _check(A, *ttgpu.dense_svd(A, ctx=ctx))


@pytest.mark.parametrize("n", [12, 48, 100, 200])
def test_tall_and_wide(ctx, n):
    g = np.random.default_rng(n)
    A = g.standard_normal((5 * n + 3, n))
    for B in (A, A.T):
        U, s, VT = ttgpu.dense_svd(B, ctx=ctx)
        assert np.linalg.norm(U * s @ VT - B) <= 1e-13 * np.linalg.norm(B)


@pytest.mark.parametrize("scale", [1e-60, 1e60])
@pytest.mark.parametrize("n", [20, 50, 130])
def test_scales(ctx, n, scale):
    A = np.random.default_rng(n).standard_normal((n, n)) * scale
    _check(A, *ttgpu.dense_svd(A, ctx=ctx))


@pytest.mark.parametrize("n,decades", [(24, 14), (40, 12), (64, 12), (96, 14), (160, 8)])
def test_graded(ctx, n, decades):
    g = np.random.default_rng(7)
    Q1, _ = np.linalg.qr(g.standard_normal((n, n)))
    Q2, _ = np.linalg.qr(g.standard_normal((n, n)))
    A = (Q1 * 10.0 ** -np.linspace(0, decades, n)) @ Q2
    _check(A, *ttgpu.dense_svd(A, ctx=ctx))


@pytest.mark.parametrize("n", [30, 56, 140])
def test_columns_of_very_different_size(ctx, n):
    """Norms over 60 decades and two columns almost parallel: angles far below
    what single precision holds by itself."""
    g = np.random.default_rng(n)
    A = g.standard_normal((n, n)) * 10.0 ** -np.linspace(0, 60, n)
    A[:, 3] = A[:, 2] * (1.0 + 1e-9) + 1e-12 * A[:, 5]
    _check(A, *ttgpu.dense_svd(A, ctx=ctx))


def test_zero_and_repeated_columns(ctx):
    A = np.random.default_rng(0).standard_normal((80, 80))
    A[:, 10] = 0.0
    A[:, 70] = A[:, 9]
    U, s, VT = ttgpu.dense_svd(A, ctx=ctx)
    assert np.linalg.norm(U * s @ VT - A) <= 1e-13 * np.linalg.norm(A)
    assert s[-1] < 1e-13 * s[0]


def test_diagonal_needs_no_rotation(ctx):
    d = np.linspace(3.0, 1.0, 72)
    U, s, VT = ttgpu.dense_svd(np.diag(d), ctx=ctx)
    assert np.array_equal(s, d)
    assert np.array_equal(U, np.eye(72)) and np.array_equal(VT, np.eye(72))
