"""The FP64 log-likelihood is the exact sum of the sites' values with two roundings
at the end (the high part, the rest): within 2^-52 of math.fsum, for sites of any
size down to 2^-26, in each kernel that sums them (small, several CTAs, the
thread-per-site form, more states)."""
import math

import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S, n_tips, n_sites, small", [
    (4, 8, 40, 1e-6), (4, 8, 40, 1e-3), (4, 8, 30011, 1e-6), (4, 30, 100003, 1e-4), (5, 9, 3001, 1e-5), (20, 7, 501, 1e-6),
    (4, 60, 100003, 0.1), (20, 30, 777, 0.02)])
def test_total_is_the_exact_sum(S, n_tips, n_sites, small):
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(n_sites), n_tips, n_sites, S=S, C=1)
    if small < 0.01:  # one state almost certain, and seen or missing in every tip: likelihoods just below one
        f = np.full(S, small)
        f[0] = 1.0 - (S - 1) * small
        masks = np.where(np.random.default_rng(1).random(masks.shape) < 0.5, 1, (1 << S) - 1).astype(np.uint32)
        masks[0] = 1
    Q = np.outer(np.ones(S), f)
    np.fill_diagonal(Q, 0.0)
    Q -= np.diag(Q.sum(axis=1))
    with _engine(left, right, bl, masks, S, Q, f, cr, cw) as h:
        lnl = h.loglik(plk.PLK_FP64)
        want = math.fsum(h.site_loglik())
    assert abs(lnl - want) <= 2.0 ** -52 * abs(want)
    if small < 0.01:
        assert 2.0 ** -26 < abs(want) / n_sites < 2.0 ** -7
