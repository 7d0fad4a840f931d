"""FP64 likelihoods and node states of few states over the site counts where the plan
changes: lanes per category, whole CTAs on an SM, and the kernels that store vectors
and normalise them after.  Sites are independent, so a sample of them is compared
with the oracle, by the bounds of the small alignments: sites agree to the last place
of a log (1e-14 of the value plus 1e-14), states to 1e-13 (marginals 1e-12)."""
import numpy as np
import pytest

from oracle import oracle as O
from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S, C, n_tips", [(4, 1, 2), (4, 1, 24), (4, 2, 9), (4, 4, 4), (4, 4, 14), (4, 8, 5),
                                          (2, 4, 6), (5, 4, 4), (5, 1, 9)])
@pytest.mark.parametrize("n_sites", [4863, 9727, 13000, 19457, 38912, 40001, 90001])
def test_few_states_many_sites(S, C, n_tips, n_sites):
    rng = np.random.default_rng(S * 100 + C * 10 + n_tips)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, S=S, C=C)
    some = np.unique(np.r_[0, 31, n_sites // 2, n_sites - 2, n_sites - 1, rng.integers(0, n_sites, 20)])
    teff = plk.effective_lengths(left, right, bl, False)
    orc = O.loglik(left, right, masks[:, some], teff, Q, f, cr, cw, p_mode=O.P_TAYLOR20,
                   want_cond_norm=True, want_marginal=True)
    with _engine(left, right, bl, masks, S, Q, f, cr, cw, p_mode=plk.PLK_P_TAYLOR20) as h:
        lnl, site = h.loglik(plk.PLK_FP64), h.site_loglik()
        np.testing.assert_allclose(site[some], orc.site_lnl, rtol=1e-14, atol=1e-14)
        assert lnl == pytest.approx(np.sum(site.astype(np.longdouble)), rel=1e-13)
        for mode, want, tol in ((plk.PLK_NODES_COND, orc.cond_norm, 1e-13),
                                (plk.PLK_NODES_MARGINAL, orc.marginal, 1e-12)):
            got = h.node_states(mode, plk.PLK_FP64)
            np.testing.assert_allclose(got[:, some], want, rtol=0, atol=tol)
            assert np.abs(got.sum(axis=-1) - 1.0).max() <= 1e-13


@pytest.mark.parametrize("S, C, n_tips", [(2, 11, 3), (2, 5, 9), (3, 7, 3), (5, 6, 2), (9, 9, 4), (12, 2, 3), (20, 12, 3), (24, 1, 5)])
@pytest.mark.parametrize("n_sites", [9727, 9728, 30001])
def test_stored_or_not(S, C, n_tips, n_sites):
    """Where the kernels that store the vectors take over: more categories, few taxa.
    FP32 rounds each of the ~2 S operations of n ops at 2^-24, so a site of these
    trees is within 9 * 2 * 24 * 6e-8 = 2.6e-5 of its likelihood (a marginal twice)."""
    rng = np.random.default_rng(S * 100 + C * 10 + n_tips)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, S=S, C=C)
    some = np.unique(np.r_[0, 31, n_sites - 1, rng.integers(0, n_sites, 12)])
    teff = plk.effective_lengths(left, right, bl, False)
    orc = O.loglik(left, right, masks[:, some], teff, Q, f, cr, cw, p_mode=O.P_TAYLOR20,
                   want_cond_norm=True, want_marginal=True)
    with _engine(left, right, bl, masks, S, Q, f, cr, cw, p_mode=plk.PLK_P_TAYLOR20) as h:
        for precision, rel, tol in ((plk.PLK_FP64, 1e-14, 1e-13), (plk.PLK_FP32S, 0.0, 2.6e-5)):
            lnl, site = h.loglik(precision), h.site_loglik()
            np.testing.assert_allclose(site[some], orc.site_lnl, rtol=rel, atol=max(1e-14, tol if rel == 0.0 else 0.0))
            assert lnl == pytest.approx(np.sum(site.astype(np.longdouble)), rel=1e-7 if rel == 0.0 else 1e-13)
            for mode, want, k in ((plk.PLK_NODES_COND, orc.cond_norm, 1), (plk.PLK_NODES_MARGINAL, orc.marginal, 10 if rel else 2)):
                got = h.node_states(mode, precision)
                np.testing.assert_allclose(got[:, some], want, rtol=0, atol=k * tol)


@pytest.mark.parametrize("n_tips", [301, 302, 700])
@pytest.mark.parametrize("n_sites", [1, 65])
def test_long_chain_of_one_category(n_tips, n_sites):
    """FP32 conditionals either side of the tree size where the stored form takes over:
    700 nodes of 8 operations round at 2^-24 each, 3.4e-4 of a vector."""
    rng = np.random.default_rng(n_tips)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, S=4, C=1)
    teff = plk.effective_lengths(left, right, bl, False)
    orc = O.loglik(left, right, masks, teff, Q, f, cr, cw, p_mode=O.P_TAYLOR20, want_cond_norm=True)
    with _engine(left, right, bl, masks, 4, Q, f, cr, cw, p_mode=plk.PLK_P_TAYLOR20) as h:
        np.testing.assert_allclose(h.node_states(plk.PLK_NODES_COND, plk.PLK_FP32S), orc.cond_norm, rtol=0, atol=3.4e-4)
