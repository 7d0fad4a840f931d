"""The streamed-table post-order forms (PLK_PRUNE_VARIANT 12, 13, 14) where their
layout changes: every count of categories (an odd last one is paired with
itself), fewer stages than ring slots, many more, a warp's last site, several
tiles a warp, spill stacks deeper than the tensor memory of many warps holds.

Every form does the same operations in the same order, so the per-site values
are the bits of the staged form (variant 1)."""
import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


def _sites(monkeypatch, case, variant):
    left, right, bl, masks, Q, f, cr, cw = case
    monkeypatch.setenv("PLK_PRUNE_VARIANT", variant)
    with _engine(left, right, bl, masks, 4, Q, f, cr, cw) as h:
        lnl = h.loglik(plk.PLK_FP32S)
        assert h.prune_kernel() == plk.Handle.PRUNE_KERNELS[4][int(variant)]
        site = h.site_loglik()
        assert h.loglik(plk.PLK_FP32S) == lnl
        return site


@pytest.mark.parametrize("C", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("n_tips, n_sites, shape", [(3, 1, "yule"), (2, 129, "balanced"), (150, 1027, "yule"),
                                                    (700, 333, "caterpillar")])
def test_same_bits_every_category_count(monkeypatch, C, n_tips, n_sites, shape):
    rng = np.random.default_rng(1000 * C + n_tips)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, n_tips, n_sites, C=C, shape=shape, missing=0.05)
    amb = rng.random(masks.shape) < 0.03
    masks[amb] = rng.integers(1, 16, size=int(amb.sum()))
    case = (left, right, bl, masks, Q, f, cr, rng.dirichlet(np.full(C, 5.0)))
    want = _sites(monkeypatch, case, "1")
    for v in ("12", "13") + (("14",) if C <= 4 else ()):
        np.testing.assert_array_equal(_sites(monkeypatch, case, v), want, err_msg=v)


@pytest.mark.parametrize("n_tips, n_sites, variant", [(512, 170001, "13"), (512, 330001, "14"), (256, 90011, "12")])
def test_same_bits_several_tiles_and_deep_stacks(monkeypatch, n_tips, n_sites, variant):
    rng = np.random.default_rng(n_sites)
    case = _random_case(rng, n_tips, n_sites, C=4, shape="balanced", missing=0.02)
    want = _sites(monkeypatch, case, "1")
    np.testing.assert_array_equal(_sites(monkeypatch, case, variant), want)


def test_an_op_list_above_shared_memory(monkeypatch):
    # more than 96 KB of ops: read from global memory
    case = _random_case(np.random.default_rng(3), 3300, 70, C=4, shape="yule", missing=0.02)
    want = _sites(monkeypatch, case, "1")
    for v in ("12", "13", "14"):
        np.testing.assert_array_equal(_sites(monkeypatch, case, v), want, err_msg=v)


def test_a_withheld_stage_times_out_and_the_handle_recovers(monkeypatch):
    rng = np.random.default_rng(79)
    left, right, bl, masks, Q, f, cr, cw = _random_case(rng, 40, 700, C=4)
    monkeypatch.setenv("PLK_PRUNE_VARIANT", "13")
    with _engine(left, right, bl, masks, 4, Q, f, cr, cw) as h:
        good = h.loglik(plk.PLK_FP32S)
        h.test_withhold_stage()
        with pytest.raises(plk.PlkError) as err:
            h.loglik(plk.PLK_FP32S)
        assert err.value.status == plk.PLK_ERR_NUMERIC
        assert h.loglik(plk.PLK_FP32S) == good
