"""The derivatives' sums over a long alignment are as exact as FP64 ones: a column
pattern repeated k times has k times its derivatives, to the rounding that FP64
sums would have.

160 columns are whole warp tiles at four categories, so every repeat has the same
3,000 partial sums r; 32 FP64 chains of 94 additions and one of 32 round by at most
(94 + 32) 2^-53 of sum |r|, the short alignment's ten by 10 2^-53, and sum |r|
is taken from single tiles: items of 16 columns each."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_a_repeated_alignment_scales_its_derivatives(seed):
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(seed), 40, 160, C=4)
    k = 300
    with plk.Batch(4) as b:
        for m in [np.tile(masks, (1, k)), masks] + [masks[:, 16 * i:16 * i + 16] for i in range(10)]:
            b.set_model(b.add(np.ascontiguousarray(m), left, right, bl), Q, f, cr, cw)
        long, short, *tiles = b.edge_derivatives()
    size = k * np.sum(np.abs(tiles), axis=0)
    assert np.all(np.abs(long - k * short) <= (94 + 32 + 10 + 2) * 2.0 ** -53 * size)
    np.testing.assert_allclose(short, np.sum(tiles, axis=0), rtol=0, atol=1e-15 * size.max())
