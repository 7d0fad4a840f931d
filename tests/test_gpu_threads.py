"""Handles and batches of different sizes in different host threads: the largest
dynamic shared memory a kernel may be launched with is one attribute per kernel,
so no launch may lower it under another thread's."""
import threading

import numpy as np
import pytest

from phylommand_gb300 import plk
from test_gpu_parity import _engine, _random_case

pytestmark = pytest.mark.gpu


def _together(make, call, sizes, reps):
    """call() of one object per size, reps times each at the same time; the
    values are those of the first call."""
    errors, start = [], threading.Barrier(len(sizes))

    def work(size):
        try:
            with make(size) as obj:
                want = call(obj)
                start.wait(60)
                for _ in range(reps):
                    np.testing.assert_array_equal(call(obj), want)
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append((size, repr(e)[:300]))
            start.abort()

    threads = [threading.Thread(target=work, args=(s,)) for s in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("S, sizes", [(20, (1, 4, 8)), (5, (2, 4, 8)), (4, (3, 4))])
@pytest.mark.parametrize("what", ["lnl", "cond", "marginal"])
def test_handles_in_threads(S, sizes, what):
    def make(C):  # the category count sets the size
        left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(C), 12 + 6 * C, 30, S=S, C=C)
        return _engine(left, right, bl, masks, S, Q, f, cr, cw)

    call = {"lnl": lambda h: h.loglik(plk.PLK_FP64),
            "cond": lambda h: h.node_states(plk.PLK_NODES_COND, plk.PLK_FP64),
            "marginal": lambda h: h.node_states(plk.PLK_NODES_MARGINAL, plk.PLK_FP64)}[what]
    _together(make, call, sizes, 1500)


@pytest.mark.parametrize("what", ["nni_loglik", "edge_derivatives"])
def test_batches_in_threads(what):
    def make(n_tips):
        left, right, bl, masks, Q, f, cr, cw = _random_case(np.random.default_rng(n_tips), n_tips, 50, C=4)
        b = plk.Batch(4)
        b.set_model(b.add(masks, left, right, bl), Q, f, cr, cw)
        return b

    _together(make, lambda b: getattr(b, what)()[0], (9, 150), 1500)
