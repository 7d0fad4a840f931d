"""The series P(t) of 4 states (plk_pmat_taylor20's operations) where its layout
changes: matrices that do not fill a warp or a CTA, codes of ambiguous cells, a
zero-length and a long branch.

The kernel does the oracle's operations in its order, so P(t) has its bits; the
per-site values are held to 1e-13 relative (logarithms of the two libraries)."""
import numpy as np
import pytest

from oracle import oracle as O
from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 2, 3, 8, 16])
@pytest.mark.parametrize("n_tips", [2, 3, 5, 16, 61])
def test_series_pmat_against_the_oracle(n_tips, C):
    rng = np.random.default_rng(100 * n_tips + C)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, 37, C=C, missing=0.05)
    amb = rng.random(masks.shape) < 0.1
    masks[amb] = rng.integers(1, 16, size=int(amb.sum()))
    bl = bl.copy()
    bl[:2] = 0.0, 30.0
    teff = plk.effective_lengths(left, right, bl, False)
    orc = O.loglik(left, right, masks, teff, Q, f, cr, cw, p_mode=O.P_TAYLOR20)
    with _engine(left, right, bl, masks, 4, Q, f, cr, cw, p_mode=plk.PLK_P_TAYLOR20) as h:
        assert h.loglik(plk.PLK_FP64) == pytest.approx(orc.lnl, rel=1e-13)
        np.testing.assert_allclose(h.site_loglik(), orc.site_lnl, rtol=1e-13, atol=1e-13)
        assert h.loglik(plk.PLK_FP32S) == pytest.approx(orc.lnl, rel=1e-6)
