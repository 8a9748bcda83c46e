"""phi_floor = 0: psi is the logarithm of min(phi, 1) as it is, so a cell with
phi below -1e-16 makes psi NaN, and one at exactly that value -inf; phi of the
next step is then NaN where the oracle's is (both lose the same neighbourhood)
and agrees with it everywhere else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("n,identity", [(64, 1), (96, 1), (96, 0)])  # edge tiles only, and interior ones
def test_negative_phi_without_floor(n, identity, precision, tol):
    from mhit36_b200 import Solver, fields
    from mhit36_b200.config import InputParams
    from oracle import Oracle
    u, v, w, phi = fields.seeded_case(n, ndrops=2, rmin=0.6, rmax=0.8)
    low = -float(np.float32(1e-16))
    for value, cell in ((-1e-3, (n // 2, n // 2 + 1, n // 3)), (-0.25, (0, n - 1, 5)), (low, (7, 3, n - 2)),
                        (0.5 * low, (n // 2, 3, n // 2))):  # the last is above -1e-16: finite
        phi[cell] = value
    p = InputParams(dt=2e-4, sigma=0.5, lin_force=0.1, tanh_identity=identity, phi_floor=0, k2_mode=1)
    with Solver(n, p, precision=precision) as s:
        s.set_fields(u, v, w, phi)
        s.step(1, raise_on_error=False)
        got = s.get_fields()[3]
    o = Oracle(n, dt=p.dt, mu=p.mu, rho=p.rho, sigma=p.sigma, epsr=p.epsr, lin_force=p.lin_force, phase_field=1,
               tanh_identity=identity, phi_floor=0, k2_mode=1)
    o.set_fields(u, v, w, phi)
    o.step(1)
    want = o.get_fields()[3]
    o.close()
    bad = np.isnan(want)
    assert 3 <= bad.sum() < 200 and np.array_equal(np.isnan(got), bad)
    assert np.max(np.abs(got - want)[~bad]) <= tol
