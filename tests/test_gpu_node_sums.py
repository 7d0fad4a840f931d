"""FP32 node states are normalised to FP64's bits but three: a probability is rounded
at 2^-50 of its size, so a site's sum to one within 2^-50 and the additions' S 2^-53
(and 2^-50 for the total's own rounding), whatever FP32 did to the vectors."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S, C, n_tips, n_sites, shape, scale", [
    (2, 4, 26, 55, "balanced", 0.1), (4, 1, 39, 218, "yule", 30.0), (4, 4, 100, 1000, "yule", 1.0),
    (4, 8, 31, 195, "caterpillar", 1e-3), (5, 3, 250, 98, "balanced", 0.1), (7, 1, 224, 30, "caterpillar", 30.0),
    (20, 4, 20, 300, "yule", 1.0), (24, 4, 96, 246, "yule", 1.0), (4, 16, 12, 33, "yule", 1.0)])
def test_probabilities_sum_to_one(S, C, n_tips, n_sites, shape, scale):
    rng = np.random.default_rng(S * C + n_tips)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, S=S, C=C, shape=shape, missing=0.1)
    cw = np.maximum(rng.dirichlet(np.full(C, 0.5)), 1e-9)
    with _engine(left, right, bl * scale, masks, S, Q, f, cr, cw / cw.sum()) as h:
        for mode in (plk.PLK_NODES_COND, plk.PLK_NODES_MARGINAL):
            p = h.node_states(mode, plk.PLK_FP32S)
            assert np.abs(p.sum(axis=-1) - 1.0).max() <= 2.0 ** -49 + S * 2.0 ** -53
