"""The row kernel's cluster where some of its four CTAs own no columns of a layer
(widths up to 48) or of none but the first: those CTAs have no slice to send and
still have to be waited for, or a fast one's slices would run ahead of them."""
import numpy as np
import pytest

from phylommand_gb300 import plk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in, n_hidden, layers, n_out", [(16, 16, 7, 1), (3, 32, 7, 16), (256, 48, 3, 3), (43, 256, 3, 7)])
def test_repeated_passes_give_the_same_bits(n_in, n_hidden, layers, n_out):
    rng = np.random.default_rng(n_hidden)
    rows = 128 * 60 + 1  # 61 clusters
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    t = rng.normal(size=(rows, n_out)).astype(np.float32)
    with plk.MLP(n_in, n_out, n_hidden, layers, seed=2) as net:
        y, (g, loss) = net.forward(x), net.gradients(x, t)
        assert np.isfinite(loss)
        for _ in range(100):
            np.testing.assert_array_equal(net.forward(x), y)
            got, again = net.gradients(x, t)
            np.testing.assert_array_equal(got, g)
            assert again == loss
