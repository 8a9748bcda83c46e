"""A stopped simulation: every kernel of a further step leaves as a whole CTA
before it arms a barrier or loads a plane, so the call returns at once, the
fields stay the same bits and a new state steps as in a fresh handle.  Sizes
with edge tiles only (32), with interior tiles (96) and with the fused
projection (256), both forms, solver and ensemble.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(precision, **kw):
    from mhit36_b200.config import InputParams
    return InputParams(dt=2e-4, sigma=0.5, lin_force=0.1, k2_mode=1 if precision == "fp32" else 0, **kw)


@pytest.mark.parametrize("n,precision,phase", [(32, "fp64", True), (96, "fp64", True), (96, "fp64", False),
                                               (96, "fp32", True), (256, "fp64", True), (256, "fp32", True)])
def test_stopped_simulation_stays_as_it_is(n, precision, phase):
    from mhit36_b200 import Solver, capi, fields
    case = fields.seeded_case(n, phase_field=phase, ndrops=2, rmin=0.5, rmax=0.7)
    with Solver(n, _params(precision, cfl_limit=1e-9), precision=precision, phase_field=phase) as s:
        s.set_fields(*case)
        assert s.step(1, raise_on_error=False)["rc"] == capi.MHIT_ERR_CFL
        before = s.get_fields()
        d = s.step(5, raise_on_error=False)
        assert d["rc"] == capi.MHIT_ERR_CFL and d["step"] == 1
        after = s.get_fields()
        s.set_fields(*case)  # a new state starts again
        s.step(1, raise_on_error=False)
        again = s.get_fields()
    with Solver(n, _params(precision), precision=precision, phase_field=phase) as s:
        s.set_fields(*case)
        s.step(1)
        fresh = s.get_fields()
    for a, b, c, f in zip(before, after, again, fresh):
        assert a is None or (np.array_equal(a, b) and np.array_equal(a, c) and np.array_equal(a, f))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_stopped_request_beside_a_running_one(precision):
    from mhit36_b200 import Solver, capi, fields
    from mhit36_b200.ensemble import Ensemble
    n = 96
    case = fields.seeded_case(n, ndrops=2, rmin=0.5, rmax=0.7)
    with Ensemble(slots_per_class=2) as e:
        bad = e.submit(n, _params(precision, cfl_limit=1e-9), *case, nsteps=6, precision=precision)
        good = e.submit(n, _params(precision), *case, nsteps=6, precision=precision)
        e.run()
        q = e.query(bad)
        assert q["state"] == "failed" and q["status"] == capi.MHIT_ERR_CFL and q["diag"]["step"] == 1
        assert e.query(good)["state"] == "done"
        stopped, whole = e.result(bad), e.result(good)
    for steps, got in ((1, stopped), (6, whole)):
        with Solver(n, _params(precision), precision=precision) as s:
            s.set_fields(*case)
            s.step(steps)
            want = s.get_fields()
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
