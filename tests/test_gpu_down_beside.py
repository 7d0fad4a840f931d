"""NNI scores and derivatives of a batch in which some items read their tables through
L1 and the others from shared memory: the two launches run side by side over their
own parts of the scratch, with the bits that every item has in a batch of its own
(the sites' order of summation is an item's own)."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_down import _batch, _items

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [
    [(900, 40, "yule"), (3, 1, "yule")],
    [(900, 3000, "yule"), (300, 4000, "balanced"), (5, 1, "yule"), (61, 15000, "yule"), (30, 130, "caterpillar")],
    [(1000, 12, "caterpillar"), (950, 700, "yule"), (120, 20000, "yule"), (2, 33, "yule"), (400, 65, "yule")]])
@pytest.mark.parametrize("C", [1, 4, 6])
def test_side_by_side_gives_the_bits_of_each_alone(C, shapes):
    items = _items(C, shapes, C)
    want = []
    for item in items:
        with _batch([item], C) as b:
            want.append((b.nni_loglik()[0], b.edge_derivatives()[0], b.loglik()[0]))
    with _batch(items, C) as b:
        for _ in range(3):
            lnl, nni, der = b.loglik(), b.nni_loglik(), b.edge_derivatives()
            for i, (n, d, l) in enumerate(want):
                np.testing.assert_array_equal(nni[i], n)
                np.testing.assert_array_equal(der[i], d)
                assert lnl[i] == pytest.approx(l, rel=1e-6)
