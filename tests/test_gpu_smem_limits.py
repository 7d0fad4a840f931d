"""Trees whose tables, op lists and stacks come close to a CTA's shared memory:
a kernel's plan has to leave room for its static shared memory too, and a size
that does not fit must not show up as an error of a later launch.

Every 4-state FP32 form gives the same per-site bits, so the tuned form's are
those of the staged form with one site a thread (variant 1)."""
import numpy as np
import pytest

from phylommand_gb300 import plk
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
