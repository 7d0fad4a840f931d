"""Exact P(t) where a method that is backward stable for the symmetrised Q is not good
enough: states that never mix (exact zeros, or a tip combination that is impossible
turns finite), and frequencies over many decades, by whose square root the entries
are divided.

Tolerance of the skewed case: 16 n eps of an entry, as the method exact to each
entry has it; one exact to the vectors' length loses up to sqrt(pi_max / pi_min)."""
import numpy as np
import pytest

from phylommand_gb300 import plk


def _q(ex, f):
    ex = np.triu(ex, 1)
    Q = (ex + ex.T) * f[None, :]
    np.fill_diagonal(Q, 0.0)
    Q -= np.diag(Q.sum(axis=1))
    return Q / -np.dot(f, np.diag(Q))


@pytest.mark.parametrize("n", [4, 5, 8, 9, 12, 20, 24])
def test_states_that_never_mix_have_probability_zero(n):
    rng = np.random.default_rng(n)
    for _ in range(5):
        cls = rng.permutation(n) % 2
        ex = rng.uniform(0.5, 3, (n, n)) * (cls[:, None] == cls[None, :])
        f = rng.dirichlet(np.full(n, 5.0))
        for t in (0.0, 1e-4, 0.1, 5.0):
            P = plk.pmat_host(_q(ex, f), t, plk.PLK_P_EXACT, f, True)
            assert np.all(P[cls[:, None] != cls[None, :]] == 0.0)


@pytest.mark.parametrize("n", [5, 9, 20])
@pytest.mark.parametrize("decades", [1, 2, 3, 6])
def test_skewed_frequencies(n, decades):
    mp = pytest.importorskip("mpmath")
    mp.mp.dps = 40
    rng = np.random.default_rng(100 * n + decades)
    f = 10.0 ** rng.uniform(-decades, 0, n)
    f[0], f[1] = 1.0, 10.0 ** -decades
    f /= f.sum()
    Q = _q(rng.uniform(0.5, 3, (n, n)), f)
    for t in (1e-3, 0.3):
        E = mp.expm(mp.matrix(Q.tolist()) * mp.mpf(t), method="taylor")
        want = np.array([[float(E[i, j]) for j in range(n)] for i in range(n)])
        got = plk.pmat_host(Q, t, plk.PLK_P_EXACT, f, True)
        assert np.abs(got - want).max() <= 16 * n * 2.0 ** -53
