"""FP32 node states where a vector holds nothing but the rounding noise of P(0), of
either sign (two tips that differ at zero effective length, the reference's root
rule): the values mean nothing, but they are the FP64 engine's to FP32's rounding,
finite where those are."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [163032499, 120458263, 5, 6])
@pytest.mark.parametrize("C", [1, 2, 4])
def test_noise_stays_finite(seed, C):
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(seed), 2, 400, C=C)
    with plk.Handle() as h:
        h.set_alignment(masks, 4)
        h.set_tree(left, right, bl)  # the root quirk is the default
        h.set_model(Q, f, True, cr, cw, plk.PLK_P_EXACT)
        for mode in (plk.PLK_NODES_COND, plk.PLK_NODES_MARGINAL):
            got, want = h.node_states(mode, plk.PLK_FP32S), h.node_states(mode, plk.PLK_FP64)
            ok = np.isfinite(want)
            assert np.array_equal(np.isfinite(got), ok)
            # noise terms cancel in the total: errors relative to the largest value
            size = np.abs(want[ok].reshape(-1, 4)).max(axis=1, keepdims=True)
            assert np.all(np.abs(got[ok] - want[ok]).reshape(-1, 4) <= 1e-5 * size * np.maximum(size, 1.0))
