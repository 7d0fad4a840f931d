"""Evaluations for which the kernels that store every vector are chosen for speed:
without room for the vectors (PLK_STORED_BYTES bounds them) the any-state kernel runs
them as before, FP64 with the same operations in the same order."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S, C, n_tips", [(2, 11, 3), (4, 8, 5), (9, 9, 4)])
def test_bound_on_stored_vectors(monkeypatch, S, C, n_tips):
    n_sites = 30001
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(S), n_tips, n_sites, S=S, C=C)
    got = []
    for most in ("0", "8e9"):
        monkeypatch.setenv("PLK_STORED_BYTES", most)
        with _engine(left, right, bl, masks, S, Q, f, cr, cw) as h:
            got.append([(h.loglik(p), h.site_loglik(), h.node_states(plk.PLK_NODES_COND, p),
                         h.node_states(plk.PLK_NODES_MARGINAL, p)) for p in (plk.PLK_FP64, plk.PLK_FP32S)])
    # the tolerances of the any-state kernel against the oracle, from either side
    for (lnl, site, cond, marg), want, rel, tol in zip(got[0], got[1], (1e-14, 0.0), (1e-13, 2.6e-5)):
        assert lnl == pytest.approx(want[0], rel=max(rel, 1e-13) if rel else 2e-6)
        np.testing.assert_allclose(site, want[1], rtol=rel, atol=2 * (1e-14 if rel else tol))
        np.testing.assert_allclose(cond, want[2], rtol=0, atol=2 * tol)
        np.testing.assert_allclose(marg, want[3], rtol=0, atol=20 * tol if rel else 4 * tol)
