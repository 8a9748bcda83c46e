"""Served results when the buffers of released requests are used again: a
second batch of other inputs and sizes on the same ensemble, results read in
another order and after cancelled and unread requests, equal to the plain
Solver's bit for bit."""
import numpy as np
import pytest

from test_gpu_ensemble import _case, _params, _same, _solo

pytestmark = pytest.mark.gpu


def test_second_batch_on_the_same_ensemble():
    from mhit36_b200.ensemble import Ensemble
    reqs = [(64, True, 3), (32, False, 4), (64, False, 2), (64, True, 5)]
    with Ensemble(slots_per_class=2) as ens:
        for batch in range(3):
            cases = [_case(n, pf, 10 * batch + i) for i, (n, pf, _) in enumerate(reqs)]
            ids = [ens.submit(n, _params(), *cases[i], nsteps=st) for i, (n, pf, st) in enumerate(reqs)]
            ens.run()
            for i in (2, 0, 3):  # request 1 is released unread
                n, pf, st = reqs[i]
                _same(ens.result(ids[i]), _solo(n, _params(), cases[i], st))
            for i in ids:
                ens.release(i)


def test_batch_after_cancelled_requests():
    """Cancelled while queued, while loading or running, and when done (which
    leaves a request as it is): the next batch's results are its own."""
    from mhit36_b200.ensemble import Ensemble
    with Ensemble(slots_per_class=2) as ens:
        for batch in range(3):
            cases = [_case(64, True, 20 * batch + i) for i in range(4)]
            ids = [ens.submit(64, _params(), *c, nsteps=4 if i else 5000) for i, c in enumerate(cases)]
            for _ in range(30 * batch):  # admitted and loading, or some steps in
                ens.progress()
            ens.cancel(ids[0])
            ens.cancel(ids[3])
            gone = [i for i in (0, 3) if ens.query(ids[i])["state"] == "cancelled"]
            assert 0 in gone
            ens.run()
            for i in range(4):
                if i not in gone:
                    _same(ens.result(ids[i]), _solo(64, _params(), cases[i], 4))
            for i in ids:
                ens.release(i)


def test_large_result_is_copied_whole():
    """A field of 7 MB is copied by several threads."""
    from mhit36_b200.ensemble import Ensemble
    case = _case(96, True, 5)
    with Ensemble(slots_per_class=1) as ens:
        i = ens.submit(96, _params(), *case, nsteps=2)
        ens.run()
        got = ens.result(i)
    _same(got, _solo(96, _params(), case, 2))
    assert all(np.isfinite(a).all() for a in got)
