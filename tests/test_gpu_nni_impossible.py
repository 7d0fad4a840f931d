"""NNI scores of sites whose likelihood is zero: -inf, as the logarithm has it, and
never a finite value that would rank among the others."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 3, 4])
@pytest.mark.parametrize("n_sites", [1, 70])
def test_an_impossible_site_scores_minus_infinity(C, n_sites):
    left, right, bl, masks, _, _, cr, cw = _random_case(np.random.default_rng(C), 12, n_sites, C=C, missing=0.0)
    masks[:] = np.where(masks < 4, 1, 4)  # A or G in every cell
    f = np.full(4, 0.25)
    Q = np.zeros((4, 4))  # transitions only: no path between A, G and C, T
    Q[0, 2] = Q[2, 0] = Q[1, 3] = Q[3, 1] = 1.0
    Q -= np.diag(Q.sum(axis=1))
    bad = masks.copy()
    bad[5, n_sites // 2] = 2  # a C among them
    with plk.Batch(C) as b:
        for m in (masks, bad, masks):
            b.set_model(b.add(m, left, right, bl), Q, f, cr, cw)
        ok, impossible, again = b.nni_loglik()
    assert np.all(np.isfinite(ok)) and np.array_equal(ok, again)
    assert np.all(np.isneginf(impossible)), impossible
