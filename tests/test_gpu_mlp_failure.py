"""Failure paths of the networks up to 256 wide: a bounded wait that runs out is
reported by the pass it happened in, whichever CTA's it was, and the network
goes on as if that pass had not been."""
import numpy as np
import pytest

from phylommand_gb300 import plk

pytestmark = pytest.mark.gpu


def _case(n_in=43, n_out=64, rows=300):
    # 64 outputs: every CTA of a row block's cluster has columns of the last layer
    rng = np.random.default_rng(rows)
    return rng.normal(size=(rows, n_in)).astype(np.float32), rng.normal(size=(rows, n_out)).astype(np.float32)


def _times_out(call, *args):
    with pytest.raises(plk.PlkError) as err:
        call(*args)
    assert err.value.status == plk.PLK_ERR_TIMEOUT


def test_a_row_kernel_that_gives_up():
    x, t = _case()
    with plk.MLP(43, 64, 256, 2, seed=1) as net, plk.MLP(43, 64, 256, 2, seed=1) as ref:
        y, p = ref.forward(x), ref.get_params()
        net.test_withhold(1)
        _times_out(net.forward, x)
        np.testing.assert_array_equal(net.forward(x), y)
        net.test_withhold(1)
        _times_out(net.gradients, x, t)
        net.test_withhold(1)
        _times_out(net.train_step, x, t, 1e-3)
        np.testing.assert_array_equal(net.get_params(), p)  # no update
        assert net.train_step(x, t, 1e-3) == ref.train_step(x, t, 1e-3)
        np.testing.assert_array_equal(net.get_params(), ref.get_params())  # Adam's first step, not its second
        np.testing.assert_array_equal(net.forward(x), ref.forward(x))


def test_an_update_kernel_that_gives_up():
    x, t = _case()
    with plk.MLP(43, 64, 256, 2, seed=1) as net, plk.MLP(43, 64, 256, 2, seed=1) as ref:
        net.test_withhold(2)
        _times_out(net.gradients, x, t)
        np.testing.assert_array_equal(net.gradients(x, t)[0], ref.gradients(x, t)[0])
        p = net.get_params()
        net.test_withhold(2)
        _times_out(net.train_step, x, t, 1e-3)
        got = net.get_params()
        ref.train_step(x, t, 1e-3)
        # the tile that gave up, the last layer's last inputs (its bias belongs to the first), kept its weights
        w = slice(p.size - 64 - 64 * 256, p.size - 64)
        np.testing.assert_array_equal(got[w].reshape(64, 256)[:, 224:], p[w].reshape(64, 256)[:, 224:])
        np.testing.assert_array_equal(got[:w.start], ref.get_params()[:w.start])
        assert np.isfinite(net.train_step(x, t, 1e-3))


def test_a_batch_that_does_not_fit_leaves_the_network_usable():
    # 2^26 rows: 34 GB a hidden layer, twice, so an allocation in the middle fails
    rows = 1 << 26
    big = np.zeros((rows, 1), dtype=np.float32)
    x, t = _case(1, 1, 40)
    with plk.MLP(1, 1, 256, 7, seed=1) as net, plk.MLP(1, 1, 256, 7, seed=1) as ref:
        for _ in range(2):
            with pytest.raises(plk.PlkError) as err:
                net.gradients(big, big)
            assert err.value.status == plk.PLK_ERR_ALLOC
        np.testing.assert_array_equal(net.gradients(x, t)[0], ref.gradients(x, t)[0])
