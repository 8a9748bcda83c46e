"""The stencil kernels' default z chunks: uneven chunks (n not a multiple of
their number; the FP32 phase kernel takes them up to 256^3) and chunks of a few
planes give the same bits as the even 32-plane chunks, in both forms and with
and without the phase field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision,phase", [(32, "fp64", True), (64, "fp64", False), (96, "fp64", True),
                                               (128, "fp64", True), (192, "fp64", True), (96, "fp32", True),
                                               (192, "fp32", True), (256, "fp32", True)])
def test_default_chunks_match_even_chunks(n, precision, phase):
    from mhit36_b200 import Solver, fields
    from mhit36_b200.config import InputParams
    p = InputParams(dt=2e-4, sigma=0.5, lin_force=0.1, k2_mode=1 if precision == "fp32" else 0)
    case = fields.seeded_case(n, phase_field=phase, ndrops=2, rmin=0.5, rmax=0.7)
    got = []
    for kz in (0, 32):
        with Solver(n, p, precision=precision, phase_field=phase) as s:
            s.set_fields(*case)
            s.set_tiles(kz, 0)
            s.step(3)
            got.append(s.get_fields())
    for a, b in zip(*got):
        assert (a is None and b is None) or np.array_equal(a, b)
