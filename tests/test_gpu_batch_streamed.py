"""The batch's streamed-table form (PLK_BATCH_PAIRED=2): every count of
categories, one and two sites a thread, trees of one stage and of many, units
whose last warps have no sites, more units than CTAs, ambiguity codes.

Its per-site values are the bits of the staged forms and a unit's sites are
summed in FP32 TwoSum either way, so an item's lnL differs from theirs by less
than 1e-12 relative (the sums' low parts, 2^-46 of a site each)."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _random_case

pytestmark = pytest.mark.gpu


def _lnl(monkeypatch, C, items, paired, spt):
    monkeypatch.setenv("PLK_BATCH_PAIRED", paired)
    monkeypatch.setenv("PLK_BATCH_SPT", spt)
    with plk.Batch(C) as b:
        for masks, left, right, bl, Q, f, cr, cw in items:
            b.set_model(b.add(masks, left, right, bl), Q, f, cr, cw)
        first = np.array(b.loglik())
        assert np.array_equal(np.array(b.loglik()), first)
        return first


def _items(C, shapes, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n_tips, n_sites, shape in shapes:
        left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, C=C, shape=shape, missing=0.05)
        amb = rng.random(masks.shape) < 0.03
        masks[amb] = rng.integers(1, 16, size=int(amb.sum()))
        out.append((masks, left, right, bl, Q, f, cr, rng.dirichlet(np.full(C, 5.0))))
    return out


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8])
def test_streamed_form_matches_the_staged_form(monkeypatch, C):
    items = _items(C, [(2, 1, "yule"), (3, 32, "yule"), (9, 257, "balanced"), (128, 900, "balanced"),
                       (300, 133, "caterpillar"), (61, 5000, "yule")], C)
    want = _lnl(monkeypatch, C, items, "0", "1")
    for spt in ("1", "2"):
        np.testing.assert_allclose(_lnl(monkeypatch, C, items, "2", spt), want, rtol=1e-12)


def test_more_units_than_ctas_and_op_lists_above_shared_memory(monkeypatch):
    items = _items(4, [(6, 200000, "yule"), (700, 700, "yule"), (33, 40001, "balanced")], 5)
    want = _lnl(monkeypatch, 4, items, "0", "1")
    for spt in ("1", "2"):
        np.testing.assert_allclose(_lnl(monkeypatch, 4, items, "2", spt), want, rtol=1e-12)
