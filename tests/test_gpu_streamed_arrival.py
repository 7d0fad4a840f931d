"""The wait for a streamed alignment's codes by itself: only the arrivals are
withheld, the tables and the ring's stages come, so a pass that did not wait
would give a finite value."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["12", "13", "14", "15", "16", "17", "18"])
def test_a_withheld_arrival_is_reported_and_the_handle_recovers(monkeypatch, variant):
    rng = np.random.default_rng(33)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, 24, 17000, C=4)
    monkeypatch.setenv("PLK_PRUNE_VARIANT", variant)
    m8 = masks.astype(np.uint8)
    with _engine(left, right, bl, m8, 4, Q, f, cr, cw) as h:
        good = h.loglik(plk.PLK_FP32S)
        assert h.prune_variant() == int(variant)
        h.set_alignment(m8, 4)
        h.test_withhold_arrival()
        with pytest.raises(plk.PlkError) as err:
            h.loglik(plk.PLK_FP32S)
        assert err.value.status == plk.PLK_ERR_NUMERIC
        assert h.loglik(plk.PLK_FP32S) == good
        # an alignment that is not streamed has no arrivals to withhold
        h.set_alignment(masks, 4)
        h.test_withhold_arrival()
        assert h.loglik(plk.PLK_FP32S) == good
