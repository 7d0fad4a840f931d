"""prune_any_kernel and down_any_kernel (any state count, FP64 and FP32, node
states) at the sizes
where its lane layout changes: one site, a warp's last site, odd state and
category counts, the widest site (16 categories), deep rescaling, one op.

FP64 keeps the oracle's operations and order, so sites agree to the last
place of a log (1e-14 of the value plus 1e-14); FP32 rounds each of the ~2 S
operations of n ops at 2^-24 relative, so a site of 40 taxa is within
40 * 2 * 24 * 6e-8 = 1.2e-4 of its likelihood at the very worst (a marginal,
from two such vectors, twice that; 600 taxa 1e-3)."""
import numpy as np
import pytest

from oracle import oracle as O
from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,C,n_sites,n_tips,shape", [
    (2, 1, 1, 2, "yule"), (2, 4, 33, 9, "balanced"), (3, 3, 101, 12, "yule"), (4, 1, 31, 40, "balanced"),
    (4, 4, 7, 40, "yule"), (4, 5, 129, 16, "yule"), (4, 16, 65, 11, "yule"), (5, 4, 1000, 23, "caterpillar"),
    (7, 5, 13, 20, "yule"), (8, 1, 500, 10, "balanced"), (9, 16, 5, 8, "yule"), (13, 2, 64, 9, "yule"),
    (20, 1, 17, 33, "balanced"), (20, 4, 311, 16, "yule"), (20, 8, 40, 12, "yule"), (23, 3, 9, 15, "yule"),
    (24, 4, 50, 40, "balanced"), (24, 16, 3, 6, "yule")])
def test_any_state_count_matches_oracle(S, C, n_sites, n_tips, shape):
    rng = np.random.default_rng(S * 1000 + C * 10 + n_sites)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, S=S, C=C, shape=shape)
    teff = plk.effective_lengths(left, right, bl, False)
    orc = O.loglik(left, right, masks, teff, Q, f, cr, cw, p_mode=O.P_TAYLOR20, want_cond_norm=True, want_marginal=True)
    with _engine(left, right, bl, masks, S, Q, f, cr, cw, p_mode=plk.PLK_P_TAYLOR20) as h:
        assert h.loglik(plk.PLK_FP64) == pytest.approx(orc.lnl, rel=1e-13)
        np.testing.assert_allclose(h.site_loglik(), orc.site_lnl, rtol=1e-14, atol=1e-14)
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_COND, plk.PLK_FP64), orc.cond_norm, rtol=0, atol=1e-13)
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_MARGINAL, plk.PLK_FP64), orc.marginal, rtol=0, atol=1e-12)
        assert h.loglik(plk.PLK_FP32S) == pytest.approx(orc.lnl, abs=1.2e-4 * n_sites)
        np.testing.assert_allclose(h.site_loglik(), orc.site_lnl, rtol=0, atol=1.2e-4)
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_COND, plk.PLK_FP32S), orc.cond_norm, rtol=0, atol=1.2e-4)
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_MARGINAL, plk.PLK_FP32S), orc.marginal, rtol=0, atol=2.4e-4)


@pytest.mark.parametrize("S,C,n_tips", [(4, 1, 600), (20, 4, 200), (6, 2, 300)])
def test_deep_caterpillar_rescales(S, C, n_tips):
    """FP64 vectors of a 600-tip caterpillar pass 2^-256 several times."""
    rng = np.random.default_rng(n_tips)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, 21, S=S, C=C, shape="caterpillar")
    teff = plk.effective_lengths(left, right, bl, False)
    orc = O.loglik(left, right, masks, teff, Q, f, cr, cw, p_mode=O.P_TAYLOR20, want_marginal=True)
    with _engine(left, right, bl, masks, S, Q, f, cr, cw, p_mode=plk.PLK_P_TAYLOR20) as h:
        assert h.loglik(plk.PLK_FP64) == pytest.approx(orc.lnl, rel=1e-12)
        assert h.loglik(plk.PLK_FP32S) == pytest.approx(orc.lnl, rel=1e-6)
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_MARGINAL, plk.PLK_FP64), orc.marginal, rtol=0, atol=1e-11)
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_MARGINAL, plk.PLK_FP32S), orc.marginal, rtol=0, atol=1e-3)
