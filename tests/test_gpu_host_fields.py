"""Fields across the host boundary: one chunk and several, whole and ragged
last chunks, both layouts and both forms.  FP64 comes back bit for bit, FP32
as the value rounded to the nearest float, infinities and zeros included."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision,layout", [(32, "fp32", 0), (96, "fp32", 1), (192, "fp32", 0), (192, "fp32", 1),
                                                (32, "fp64", 1), (192, "fp64", 0), (192, "fp64", 1)])
def test_round_trip(n, precision, layout):
    from mhit36_b200 import Solver, capi
    from mhit36_b200.config import InputParams
    rng = np.random.default_rng(n + layout)
    shape = (n, n, n) if layout == capi.MHIT_LAYOUT_RAW else (n + 2, n + 2, n)  # (z, y, x)
    a = [rng.standard_normal(shape) for _ in range(4)]
    a[0].flat[:6] = [1e300, -1e300, 1e-300, 0.0, -0.0, 3.4028235677973366e38]
    got = [np.zeros(shape) for _ in range(4)]
    with Solver(n, InputParams(k2_mode=1), precision=precision) as s:
        s.set_fields_ptr(*[x.ctypes.data for x in a], layout=layout)
        s.get_fields_ptr(*[x.ctypes.data for x in got], layout=layout)
        p = np.zeros(shape)
        s._check(s.lib.mhit_get_pressure(s.h, ctypes.c_void_p(p.ctypes.data), layout), "mhit_get_pressure")
    assert not p.any()
    core = (slice(None),) * 3 if layout == capi.MHIT_LAYOUT_RAW else (slice(1, n + 1), slice(1, n + 1), slice(None))
    for x, y in zip(a, got):
        with np.errstate(over="ignore"):
            want = x[core].astype(np.float32).astype(np.float64) if precision == "fp32" else x[core]
        assert np.array_equal(y[core], want)
        if layout == capi.MHIT_LAYOUT_PIX_HALO:  # periodic halo
            assert np.array_equal(y[0], y[n]) and np.array_equal(y[:, n + 1], y[:, 1])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_pinned_arrays(precision):
    """Pinned arrays are copied without the staging chunks."""
    import torch
    from mhit36_b200 import Solver
    from mhit36_b200.config import InputParams
    n = 128
    a = [torch.randn(n ** 3, dtype=torch.float64).pin_memory() for _ in range(4)]
    got = [torch.zeros(n ** 3, dtype=torch.float64).pin_memory() for _ in range(4)]
    with Solver(n, InputParams(k2_mode=1), precision=precision) as s:
        s.set_fields_ptr(*[x.data_ptr() for x in a])
        s.get_fields_ptr(*[x.data_ptr() for x in got])
    for x, y in zip(a, got):
        assert torch.equal(y, x.float().double() if precision == "fp32" else x)


@pytest.mark.parametrize("n,precision,layout", [(256, "fp32", 1), (384, "fp64", 0)])
def test_round_trip_in_larger_pieces(n, precision, layout):
    test_round_trip(n, precision, layout)
