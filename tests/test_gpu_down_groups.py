"""NNI scores and derivatives of a batch whose records do not fit at once: its items
go in groups over the same records, with the same bits (PLK_BATCH_RECORD_BYTES
lowers the bound; 0 is a group per item)."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_down import _batch, _items

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", ["0", "40000", "300000"])
@pytest.mark.parametrize("C", [1, 4, 5])
def test_groups_give_the_same_bits(monkeypatch, C, most):
    # the 900 taxa read their tables through L1, the others from shared memory
    items = _items(C, [(900, 40, "yule"), (5, 1, "yule"), (60, 700, "balanced"), (3, 9, "yule"), (30, 130, "caterpillar"),
                       (61, 33, "yule")], C)
    with _batch(items, C) as b:
        nni, der = b.nni_loglik(), b.edge_derivatives()
    monkeypatch.setenv("PLK_BATCH_RECORD_BYTES", most)
    with _batch(items, C) as b:
        for _ in range(2):
            for got, want in zip(b.nni_loglik() + b.edge_derivatives(), nni + der):
                np.testing.assert_array_equal(got, want)
