"""The on-GPU diagnostics against numpy in 64 bits, at sizes on both sides of
the kernel's plane counts.  Sums of n^3 terms of one sign: 1e-13 relative is
far above their rounding (n^3 = 4e6 terms in blocks, about 1e-15)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,phase", [(32, True), (96, False), (128, True), (256, True)])
def test_stats_match_numpy(n, phase):
    from mhit36_b200 import Solver
    from mhit36_b200.config import InputParams
    rng = np.random.default_rng(n)
    u, v, w = (rng.standard_normal((n, n, n)) for _ in range(3))
    phi = rng.random((n, n, n)) if phase else None
    p = InputParams()
    with Solver(n, p, phase_field=phase) as s:
        s.set_fields(u, v, w, phi)
        st = s.stats(pi_f32=False)
    dxi = (n - 1) / (2 * np.pi)
    up, dn = (lambda a, ax: np.roll(a, -1, ax)), (lambda a, ax: np.roll(a, 1, ax))
    d = [[(up(a, ax) - dn(a, ax)) * (0.5 * dxi) for ax in range(3)] for a in (u, v, w)]
    ss = sum(d[a][a] ** 2 for a in range(3))
    for a, b in ((0, 1), (0, 2), (1, 2)):
        ss = ss + 2.0 * (0.5 * (d[a][b] + d[b][a])) ** 2
    div = (up(u, 0) - u + up(v, 1) - v + up(w, 2) - w) * dxi
    want = {"ke": 0.5 * np.mean(u * u + v * v + w * w), "dissipation": 2 * p.mu / p.rho * np.mean(ss),
            "max_div": np.max(np.abs(div)), "phi_sum": phi.sum() if phase else 0.0,
            "phi_min": phi.min() if phase else 0.0, "phi_max": phi.max() if phase else 0.0}
    for k, x in want.items():
        assert abs(st[k] - x) <= 1e-13 * abs(x), (k, st[k], x)
    assert abs(st["umean"] - u.mean()) <= 1e-13
