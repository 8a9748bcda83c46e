"""The FP32 refinement form at the sizes 3*2^k, whose column passes start with
a radix-12 stage, against the FP64 form of the same discrete problem.

Tolerances: the FP32 form stores u, v, w, phi and the transforms in FP32
(half an ulp is 6e-8) and rounds each some tens of times a step, so that five
steps stay within 2e-5 of a field's largest value; the first solve's error is
removed by the FP64 residual's, which leaves max |div u| at 1e-10 and p = p0 +
dp within the same 2e-5 (both bars are those of the power-of-two sizes or
below them).
"""
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,phase", [(96, True), (192, True), (384, False)])
def test_fp32_matches_fp64(n, phase):
    from mhit36_b200 import Solver, fields
    from mhit36_b200.config import InputParams
    p = InputParams(dt=2e-4, mu=6e-3, sigma=0.5, lin_force=0.1, k2_mode=1)
    case = fields.seeded_case(n, phase_field=phase, ndrops=4, rmin=0.4, rmax=0.6)
    with Solver(n, p, phase_field=phase) as a, Solver(n, p, precision="fp32", phase_field=phase) as b:
        a.set_fields(*case)
        b.set_fields(*case)
        a.step(5)
        div = b.step(5)["max_div"]
        fa, fb = a.get_fields(), b.get_fields()
        pa, pb = a.get_pressure(), b.get_pressure()
    assert 0 < div <= 1e-10
    errs = [rel_err(y, x) for x, y in zip(fa, fb) if x is not None] + [rel_err(pb, pa)]
    assert max(errs) <= 2e-5, errs
