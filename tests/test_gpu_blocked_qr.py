"""Blocked one-CTA Householder QR (csrc/small_dense.cu) at the edges of its
panels of 8: row and column remainders, last panels that end inside a tile of
a wide matrix, one row or column, and the largest that shared memory holds."""
import numpy as np
import pytest

import ttgpu

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 9), (9, 1), (2, 2), (7, 8), (8, 7), (8, 8), (8, 9), (9, 8), (15, 16), (16, 15),
          (17, 17), (10, 20), (20, 10), (3, 100), (100, 3), (31, 33), (64, 40), (65, 41), (130, 130),
          (140, 137), (700, 33), (1599, 15), (2500, 9), (12, 300), (36, 250)]


@pytest.mark.parametrize("m,n", SHAPES)
def test_matches_lapack(ctx, m, n):
    A = np.random.default_rng(m + 1000 * n).standard_normal((m, n))
    Q, R = ttgpu.dense_qr(A, ctx=ctx)
    Qr, Rr = np.linalg.qr(A)
    k = min(m, n)
    # backward error and orthogonality of Householder QR: a few eps per column
    assert np.linalg.norm(Q @ R - A) <= 1e-14 * np.linalg.norm(A)
    assert np.linalg.norm(Q.T @ Q - np.eye(k)) <= 1e-15 * (k + 10)
    assert np.array_equal(np.tril(R, -1), np.zeros_like(R))
    # LAPACK's signs; a square Gaussian matrix has a condition of some 1e3
    assert np.linalg.norm(R - Rr) <= 1e-11 * np.linalg.norm(Rr)


def test_zero_and_dependent_columns(ctx):
    g = np.random.default_rng(4)
    A = g.standard_normal((60, 21))
    A[:, 0] = 0.0
    A[:, 9] = 2.0 * A[:, 8]
    A[5:, 20] = 0.0
    Q, R = ttgpu.dense_qr(A, ctx=ctx)
    assert np.linalg.norm(Q @ R - A) <= 1e-14 * np.linalg.norm(A)
    assert np.linalg.norm(Q.T @ Q - np.eye(21)) <= 4e-14
    Z, T = ttgpu.dense_qr(np.zeros((12, 5)), ctx=ctx)
    assert np.array_equal(Z, np.eye(12, 5)) and np.array_equal(T, np.zeros((5, 5)))


def test_triangular_input_keeps_its_columns(ctx):
    """Nothing below the diagonal: no reflector, as LAPACK's dlarfg."""
    A = np.triu(np.random.default_rng(6).standard_normal((30, 30)))
    Q, R = ttgpu.dense_qr(A, ctx=ctx)
    assert np.array_equal(Q, np.eye(30)) and np.array_equal(R, A)
