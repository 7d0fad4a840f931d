"""Network rows below and above the size from which they are copied to the device
instead of read in place (320 KB of inputs and targets): the same weights and
outputs as in passes that are small enough to be read in place."""
import numpy as np
import pytest

from phylommand_gb300 import plk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [372, 374, 375, 1024])  # 219 floats a row: 374 rows are the last below
def test_outputs_do_not_depend_on_the_route(rows):
    rng = np.random.default_rng(rows)
    x = rng.normal(size=(rows, 205)).astype(np.float32)
    t = rng.normal(size=(rows, 14)).astype(np.float32)
    with plk.MLP(205, 14, 45, 3, seed=3) as m:
        y = m.forward(x)
        # a row's outputs do not depend on the rows beside it
        parts = [m.forward(x[i:i + 128]) for i in range(0, rows, 128)]
        np.testing.assert_array_equal(y, np.concatenate(parts))
        g, loss = m.gradients(x, t)
        want = np.mean((y.astype(np.float64) - t) ** 2)
        # FP32 sums of 14 * rows positive terms, 2^-24 each: at most 14 * 1024 * 6e-8 of it
        assert loss == pytest.approx(want, rel=9e-4)
        assert np.isfinite(g).all()
