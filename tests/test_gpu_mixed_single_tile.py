"""Mixed local matvec whose vectors are one 32 x 32 tile of the layout changes
(csrc/mixed_ops.cu): nothing is launched for the empty half of its tiles."""
import numpy as np
import pytest

import ttgpu
from oracle import amen as oamen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rx1,n,rx2,launches", [
    (1, 1, 1, 9), (7, 1, 32, 9), (32, 1, 32, 9), (33, 1, 5, 10), (3, 2, 4, 10)])
def test_launches_and_result(ctx, rx1, n, rx2, launches):
    rng = np.random.default_rng(rx1 + n + rx2)
    Phi1, A = rng.standard_normal((rx1, rx1, 2)), rng.standard_normal((2, n, n, 2))
    Phi2, x = rng.standard_normal((rx2, 2, rx2)), rng.standard_normal(rx1 * n * rx2)
    ttgpu.bfun3(Phi1, A, Phi2, x, ctx=ctx, precision="mixed")
    before = ctx.launch_count()
    y = ttgpu.bfun3(Phi1, A, Phi2, x, ctx=ctx, precision="mixed")
    assert ctx.launch_count() - before == launches
    ref = oamen.bfun3(Phi1, A, Phi2, x)
    # BF16 operands: 2^-9 each of four factors, relative to the sum of magnitudes
    mag = oamen.bfun3(np.abs(Phi1), np.abs(A), np.abs(Phi2), np.abs(x))
    assert np.all(np.abs(y.ravel() - ref.ravel()) <= 5 * 2.0 ** -9 * mag.ravel())
