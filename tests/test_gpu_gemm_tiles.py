"""The FP64 GEMM's tiles (csrc/kernels_f64.cu) at their edges, through the
contractions that are made of it: one row past a tile, remainders of the k
step, odd leading dimensions (8-byte copies) and even ones (16-byte), products
that one CTA holds, that many fill, and long ones cut into slices."""
import numpy as np
import pytest

import ttgpu

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (2, 3, 1, 2), (17, 5, 16, 1), (31, 7, 33, 2), (32, 16, 32, 2),
          (33, 9, 31, 3), (64, 4, 65, 2), (65, 15, 63, 1), (66, 31, 34, 3), (128, 2, 96, 2),
          (129, 17, 40, 3)]


def _operands(r1, n, r2, ra):
    g = np.random.default_rng(r1 + 100 * n + 10000 * r2)
    return (g.standard_normal((r1, r1, ra)), g.standard_normal((ra, n, n, ra)),
            g.standard_normal((r2, ra, r2)), g.standard_normal((r1, n, r2)))


# three chained products of at most K = 1200 terms: each element rounds at
# about sqrt(K) u of its terms' size, some 1e-14 relative in the norm
TOL = 1e-12


@pytest.mark.parametrize("r1,n,r2,ra", SHAPES)
def test_local_matvec_tiles(ctx, r1, n, r2, ra):
    P1, A, P2, x = _operands(r1, n, r2, ra)
    t = np.einsum("amb,bqk->amqk", x, P2)
    t = np.einsum("pjmq,amqk->apjk", A, t)
    ref = np.einsum("iap,apjk->ijk", P1, t).ravel(order="F")
    got = ttgpu.bfun3(P1, A, P2, x, ctx=ctx)
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("direction", ["lr", "rl"])
@pytest.mark.parametrize("r1,n,r2,ra", SHAPES + [(3, 64, 200, 2), (200, 64, 3, 2)])
def test_next_phi_tiles(ctx, direction, r1, n, r2, ra):
    P1, A, P2, x = _operands(r1, n, r2, ra)
    y = np.random.default_rng(5).standard_normal(x.shape)
    if direction == "lr":
        t = np.einsum("abp,ajc->bpjc", P1, x)
        t = np.einsum("bpjc,pjmq->bmqc", t, A)
        ref = np.einsum("bmqc,bme->ceq", t, y)
    else:
        t = np.einsum("bme,eqc->bmqc", y, P2)
        t = np.einsum("bmqc,pjmq->bpjc", t, A)
        ref = np.einsum("bpjc,ajc->bpa", t, x)
    got = ttgpu.compute_next_Phi(P1 if direction == "lr" else P2, x, A, y, direction, ctx=ctx)
    assert np.linalg.norm(got - ref) <= TOL * np.linalg.norm(ref)
