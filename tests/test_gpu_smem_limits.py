"""Trees whose tables, op lists and stacks come close to a CTA's shared memory:
a kernel's plan has to leave room for its static shared memory too, and a size
that does not fit must not show up as an error of a later launch.

Every 4-state FP32 form gives the same per-site bits, so the tuned form's are
those of the staged form with one site a thread (variant 1)."""
import numpy as np
import pytest

from oracle import oracle as O
from phylommand_gb300 import plk
from phylommand_gb300.nni import neighbour_tree
from test_gpu_batch import _single
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C, tips", [(4, range(243, 257)), (4, (515, 521, 527)), (4, (787, 793, 799)),
                                     (2, (115, 121, 127)), (8, (35, 41, 47)), (5, (115, 121, 127))])
def test_streamed_tables_beside_a_full_shared_memory(monkeypatch, C, tips):
    monkeypatch.delenv("PLK_PRUNE_VARIANT", raising=False)
    for n_tips in tips:
        left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(n_tips), n_tips, 20000, C=C)
        with _engine(left, right, bl, masks, 4, Q, f, cr, cw) as h:
            lnl = h.loglik(plk.PLK_FP32S)  # untuned: every form is tried
            site = h.site_loglik()
            assert h.loglik(plk.PLK_FP32S) == lnl
        with monkeypatch.context() as m:
            m.setenv("PLK_PRUNE_VARIANT", "1")
            with _engine(left, right, bl, masks, 4, Q, f, cr, cw) as h:
                assert h.loglik(plk.PLK_FP32S) == pytest.approx(lnl, rel=1e-12)
                np.testing.assert_array_equal(h.site_loglik(), site, err_msg=f"{n_tips} tips")


# The first two shapes need just less than the 48 KB that a kernel has without
# asking for more, static bytes left out; the others just less than 227 KB.
# FP64 1e-11 (P(t) of the eigen form); FP32 2 S roundings an op, two vectors a
# marginal.
@pytest.mark.parametrize("S, C, n_tips, n_sites, shape, precision", [
    (4, 1, 561, 5000, "caterpillar", plk.PLK_FP64), (5, 4, 327, 5000, "balanced", plk.PLK_FP32S),
    (4, 1, 284, 200, "balanced", plk.PLK_FP64), (4, 1, 286, 200, "caterpillar", plk.PLK_FP64),
    (5, 4, 158, 5000, "balanced", plk.PLK_FP32S), (5, 4, 174, 500, "balanced", plk.PLK_FP32S),
    (20, 8, 207, 5000, "balanced", plk.PLK_FP64), (24, 4, 393, 5000, "balanced", plk.PLK_FP64)])
def test_any_state_lnl_beside_a_full_shared_memory(S, C, n_tips, n_sites, shape, precision):
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(S + n_tips), n_tips, n_sites, S=S, C=C,
                                                        shape=shape)
    some = np.linspace(0, n_sites - 1, 16).astype(int)  # the oracle's sites
    orc = O.loglik(left, right, masks[:, some], plk.effective_lengths(left, right, bl, False), Q, f, cr, cw,
                   p_mode=O.P_EXACT)
    with _engine(left, right, bl, masks, S, Q, f, cr, cw) as h:
        h.loglik(precision)
        tol = 1e-11 if precision == plk.PLK_FP64 else 6e-8 * 2 * S * n_tips
        np.testing.assert_allclose(h.site_loglik()[some], orc.site_lnl, rtol=1e-11, atol=tol)


@pytest.mark.parametrize("S, C, n_tips, n_sites, shape, precision, mode", [
    (4, 4, 31, 200, "caterpillar", plk.PLK_FP32S, plk.PLK_NODES_COND),
    (4, 4, 31, 500, "caterpillar", plk.PLK_FP32S, plk.PLK_NODES_MARGINAL),
    (4, 4, 147, 500, "caterpillar", plk.PLK_FP32S, plk.PLK_NODES_COND),
    (4, 4, 147, 500, "yule", plk.PLK_FP32S, plk.PLK_NODES_MARGINAL),
    (4, 2, 294, 500, "balanced", plk.PLK_FP32S, plk.PLK_NODES_MARGINAL),
    (7, 2, 92, 1000, "caterpillar", plk.PLK_FP64, plk.PLK_NODES_MARGINAL),
    (3, 1, 588, 1000, "balanced", plk.PLK_FP64, plk.PLK_NODES_COND)])
def test_node_states_beside_a_full_shared_memory(S, C, n_tips, n_sites, shape, precision, mode):
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(S + n_tips), n_tips, n_sites, S=S, C=C,
                                                        shape=shape)
    some = np.linspace(0, n_sites - 1, 16).astype(int)
    orc = O.loglik(left, right, masks[:, some], plk.effective_lengths(left, right, bl, False), Q, f, cr, cw,
                   p_mode=O.P_EXACT, want_cond_norm=True, want_marginal=True)
    want = orc.cond_norm if mode == plk.PLK_NODES_COND else orc.marginal
    with _engine(left, right, bl, masks, S, Q, f, cr, cw) as h:
        got = h.node_states(mode, precision)[:, some]
        np.testing.assert_allclose(got, want, rtol=0, atol=1e-11 if precision == plk.PLK_FP64 else 6e-8 * 4 * S * n_tips)


# One item whose tables take the last 64 of 227 KB: they go through L1 instead.
# Tolerances as in test_gpu_down.
@pytest.mark.parametrize("C, n_tips, n_sites", [(5, 253, 700), (1, 464, 38000)])
def test_nni_beside_a_full_shared_memory(C, n_tips, n_sites):
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(C), n_tips, n_sites, C=C)
    with plk.Batch(C) as b:
        b.set_model(b.add(masks, left, right, bl), Q, f, cr, cw)
        got, moves = b.nni_loglik()[0], b.nni_moves(0)
    for m in (0, 1, len(moves) // 2, len(moves) - 1):
        L, R = neighbour_tree(left, right, int(moves[m][0]), int(moves[m][1]))
        assert got[m] == pytest.approx(_single(masks, L, R, bl, Q, f, cr, cw, plk.PLK_FP64), rel=1e-6)


def test_edge_derivatives_beside_a_full_shared_memory():
    C, n_tips, n_sites = 6, 226, 20000
    left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(C), n_tips, n_sites, C=C)
    with plk.Batch(C) as b:
        b.set_model(b.add(masks, left, right, bl), Q, f, cr, cw)
        d = b.edge_derivatives()[0]
    for v in (0, n_tips // 2, n_tips + 7):
        eps = 1e-4 * max(bl[v], 1e-2)
        lp, lm = (_single(masks, left, right, np.where(np.arange(len(bl)) == v, x, bl), Q, f, cr, cw, plk.PLK_FP64)
                  for x in (bl[v] + eps, bl[v] - eps))
        d1 = (lp - lm) / (2 * eps)
        assert abs(d[v, 0] - d1) <= 2e-4 * (abs(d1) + n_sites), (v, d[v], d1)
