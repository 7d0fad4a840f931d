"""The row and update kernels of networks up to 256 wide at the edges of their
tiles: 1, 127, 128, 129, 257 and 600 rows, widths that are no multiple of 16
or of the 32-input update tile, one to eight weight layers; and the
layer-by-layer kernels of a wider one.

Against the BF16-mirrored oracle, with the tolerances of the network tests:
FP32 accumulation differs from the oracle's FP64 by 2^-24 sqrt(K), and a value
that falls on the other side of a BF16 rounding moves by 2^-9 of itself: 2e-3
of the output norm and 5e-3 of a layer's gradient norm through three layers,
four times that through eight."""
import numpy as np
import pytest

from oracle import mlp as M
from phylommand_gb300 import plk
from test_gpu_mlp import _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,n_hidden,layers,n_out,rows", [
    (43, 256, 3, 7, 256), (43, 256, 3, 7, 1), (43, 64, 2, 7, 127), (17, 129, 1, 3, 128), (5, 33, 2, 1, 129),
    (256, 16, 1, 256, 257), (1, 1, 0, 1, 3), (43, 100, 7, 7, 600), (43, 260, 2, 7, 70)])
def test_forward_gradients_and_step(n_in, n_hidden, layers, n_out, rows):
    rng = np.random.default_rng(rows + n_hidden)
    dims = [n_in] + [n_hidden] * layers + [n_out]
    slack = 4.0 if layers > 3 else 1.0
    x = rng.normal(size=(rows, n_in)).astype(np.float32)
    t = rng.normal(size=(rows, n_out)).astype(np.float32)
    with plk.MLP(n_in, n_out, n_hidden, layers, seed=3) as net:
        p = net.get_params()
        p += 0.1 * rng.normal(size=p.size).astype(np.float32)  # biases too
        net.set_params(p)
        y, _, _ = M.forward(p, dims, x, bf16_mirror=True)
        assert _rel(net.forward(x), y) < 2e-3 * slack
        loss, ref = M.loss_and_grad(p, dims, x, t, bf16_mirror=True)
        g, got = net.gradients(x, t)
        assert abs(got - loss) < 1e-3 * slack * loss
        off = 0
        for a, b in zip(dims, dims[1:]):
            for lo, hi in ((off, off + a * b), (off + a * b, off + a * b + b)):
                assert _rel(g[lo:hi], ref[lo:hi]) < 5e-3 * slack, (lo, hi)
            off += a * b + b
        assert net.train_step(x, t, 1e-3) == pytest.approx(got, rel=1e-6)
        z = np.zeros(p.size)
        want, _, _ = M.adam(p.astype(np.float64), g.astype(np.float64), z, z, 1, 1e-3)
        np.testing.assert_allclose(net.get_params(), want, rtol=1e-5, atol=1e-6)
        # the images the next pass reads hold the new weights
        y, _, _ = M.forward(net.get_params(), dims, x, bf16_mirror=True)
        assert _rel(net.forward(x), y) < 2e-3 * slack
