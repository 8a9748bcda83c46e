"""max |div u| of a field with NaN is NaN, wherever the NaN sits: one cell in
the middle of a thread's column, so that later planes, other lanes, warps and
CTAs all bring finite values after it."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(32, "fp64"), (128, "fp32"), (256, "fp64")])
def test_stats_keep_one_nan(n, precision):
    from mhit36_b200 import Solver
    from mhit36_b200.config import InputParams
    rng = np.random.default_rng(n)
    f = [rng.standard_normal((n, n, n)) for _ in range(4)]
    with Solver(n, InputParams(k2_mode=1), precision=precision) as s:
        s.set_fields(*f)
        assert math.isfinite(s.stats()["max_div"])
        for c, at in ((0, (5, 3, 1)), (1, (n - 1, 0, n // 2 + 1)), (2, (n // 2, n - 1, n - 2))):
            g = [a.copy() for a in f]
            g[c][at] = np.nan
            s.set_fields(*g)
            st = s.stats()
            assert math.isnan(st["max_div"]) and math.isnan(st["ke"]), (c, at, st)


@pytest.mark.parametrize("n", [64, 256])  # inside the step, and measured when the call returns
def test_fp32_step_reports_nan_divergence(n):
    from mhit36_b200 import Solver, capi
    from mhit36_b200.config import InputParams
    u, v, w = (np.zeros((n, n, n)) for _ in range(3))
    u[3, n // 2, n // 2 + 1] = np.nan
    with Solver(n, InputParams(k2_mode=1), precision="fp32", phase_field=False) as s:
        s.set_fields(u, v, w)
        d = s.step(1, raise_on_error=False)
        assert d["rc"] == capi.MHIT_ERR_NONFINITE and math.isnan(d["max_div"])
