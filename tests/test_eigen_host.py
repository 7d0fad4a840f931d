"""P(t) of reversible models through their eigen system, where its method
changes with the number of states (4 | 5) and where eigenvalues coincide:
equal rates, a chain that falls apart, rates over many orders of magnitude.

Tolerance: |error| <= 2e-13, as the other exact P(t) tests; the methods are
backward stable, so eigenvalues move by at most about n eps |Q| = 24 x 1.1e-16 x
4, and |Q| t <= 50 here."""
import numpy as np
import pytest
from scipy.linalg import expm

from phylommand_gb300 import plk


def _model(rng, n, kind):
    f = rng.dirichlet(np.full(n, 3.0)) if kind != "equal" else np.full(n, 1.0 / n)
    ex = np.ones((n, n))
    if kind == "random":
        ex = np.exp(rng.normal(size=(n, n)))
    elif kind == "wide":
        ex = 10.0 ** rng.uniform(-9, 0, size=(n, n))
    elif kind == "apart":  # two classes that never mix
        ex = np.fromfunction(lambda i, j: 1.0 * ((i % 2) == (j % 2)), (n, n))
    elif kind == "chain":
        ex = np.fromfunction(lambda i, j: 1.0 * (abs(i - j) == 1), (n, n))
    ex = np.triu(ex, 1)
    ex = ex + ex.T
    Q = ex * f[None, :]
    np.fill_diagonal(Q, 0.0)
    np.fill_diagonal(Q, -Q.sum(1))
    mu = -(f * np.diag(Q)).sum()
    return (Q / mu if mu > 0 else Q), f


@pytest.mark.parametrize("kind", ["random", "equal", "wide", "apart", "chain"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 20, 24])
def test_exact_pmat_every_method(n, kind):
    Q, f = _model(np.random.default_rng(n), n, kind)
    for t in (0.0, 1e-6, 0.1, 3.0):
        np.testing.assert_allclose(plk.pmat_host(Q, t, plk.PLK_P_EXACT, f, True), expm(Q * t), atol=2e-13, rtol=0)


@pytest.mark.parametrize("scale", [1e-90, 1e90])
def test_scaled_rates_give_the_same_matrix(scale):
    Q, f = _model(np.random.default_rng(8), 20, "random")
    want = plk.pmat_host(Q, 0.3, plk.PLK_P_EXACT, f, True)
    np.testing.assert_allclose(plk.pmat_host(Q * scale, 0.3 / scale, plk.PLK_P_EXACT, f, True), want, atol=2e-13, rtol=0)
