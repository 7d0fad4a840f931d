"""NNI scoring and branch-length derivatives where their layout changes: every
count of categories (lanes per site, an odd last one), trees whose tables fit
in shared memory beside trees whose tables do not, one site, a warp's last
site, ambiguity codes, vectors that rescale on the way up and down.

Tolerances: a neighbour's lnL 1e-6 relative of the FP64 engine's, as every FP32
form's; a derivative against central differences of the FP64 lnL with the
step's own error (1e-4 relative of the length) plus FP32 rounding per site."""
import numpy as np
import pytest

from phylommand_gb300 import plk, synth
from phylommand_gb300.nni import neighbour_tree
from test_gpu_batch import _single
from test_gpu_parity import _random_case

pytestmark = pytest.mark.gpu


def _items(C, shapes, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n_tips, n_sites, shape in shapes:
        left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, C=C, shape=shape, missing=0.05)
        amb = rng.random(masks.shape) < 0.03
        masks[amb] = rng.integers(1, 16, size=int(amb.sum()))
        cw = rng.dirichlet(np.full(C, 5.0))
        out.append((masks, left, right, bl, Q, f, cr, cw))
    return out


def _batch(items, C):
    b = plk.Batch(C)
    for masks, left, right, bl, Q, f, cr, cw in items:
        b.set_model(b.add(masks, left, right, bl), Q, f, cr, cw)
    return b


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8])
def test_nni_every_category_count(C):
    items = _items(C, [(5, 1, "yule"), (6, 33, "balanced"), (150, 70, "caterpillar"), (420, 19, "yule")], C)
    rng = np.random.default_rng(C)
    with _batch(items, C) as b:
        nni = b.nni_loglik()
        moves = [b.nni_moves(i) for i in range(len(items))]
    for (masks, left, right, bl, Q, f, cr, cw), got, mv in zip(items, nni, moves):
        assert len(got) == 2 * (masks.shape[0] - 3)
        pick = rng.choice(len(mv), size=min(len(mv), 9), replace=False)
        for m in set(pick) | {len(mv) - 1, len(mv) - 2}:  # the root edge's moves come last
            L, R = neighbour_tree(left, right, int(mv[m][0]), int(mv[m][1]))
            assert got[m] == pytest.approx(_single(masks, L, R, bl, Q, f, cr, cw, plk.PLK_FP64), rel=1e-6)


@pytest.mark.parametrize("C", [1, 2, 3, 4, 6, 8])
def test_edge_derivatives_every_category_count(C):
    items = _items(C, [(4, 1, "yule"), (9, 45, "balanced"), (60, 130, "caterpillar"), (420, 17, "yule")], 50 + C)
    rng = np.random.default_rng(C)
    with _batch(items, C) as b:
        der = b.edge_derivatives()
    for (masks, left, right, bl, Q, f, cr, cw), d in zip(items, der):
        root, scale = len(bl) - 1, masks.shape[1]
        assert np.all(d[root] == 0.0) and np.all(np.isfinite(d))
        for v in rng.choice(root, size=min(4, root), replace=False):
            eps = 1e-4 * max(bl[v], 1e-2)
            def at(x):
                return _single(masks, left, right, np.where(np.arange(len(bl)) == v, x, bl), Q, f, cr, cw, plk.PLK_FP64)
            lp, l0, lm = at(bl[v] + eps), at(bl[v]), at(bl[v] - eps)
            d1, d2 = (lp - lm) / (2 * eps), (lp - 2 * l0 + lm) / eps ** 2
            assert abs(d[v, 0] - d1) <= 2e-4 * (abs(d1) + scale), (v, d[v], d1)
            # a second difference of lnL values of size |l0| carries |l0| 2^-52 * 4 / eps^2
            assert abs(d[v, 1] - d2) <= 2e-2 * abs(d2) + 1e-3 * scale / max(bl[v], 1e-2) + 4 * abs(l0) * 2.3e-16 / eps ** 2
