"""Drop counting on packed words: random cells at densities from isolated
single cells to a percolating tangle, where runs cross word boundaries and
the periodic faces in every direction, and more drops than the first call's
room, against the oracle's flood fill."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,density,precision", [(32, 0.01, "fp64"), (32, 0.1, "fp64"), (32, 0.5, "fp64"),
                                                 (64, 0.05, "fp64"), (64, 0.08, "fp32"), (96, 0.02, "fp64"),
                                                 (32, 0.0, "fp64"), (32, 1.0, "fp64")])
def test_random_cells(n, density, precision):
    from oracle import drop_count
    from mhit36_b200 import Solver
    from mhit36_b200.config import InputParams
    rng = np.random.default_rng(n)
    phi = (rng.random((n, n, n)) < density) * np.where(rng.random((n, n, n)) < 0.5, 0.5, 1.0)
    z = np.zeros((n, n, n))
    with Solver(n, InputParams(k2_mode=1), precision=precision) as s:
        s.set_fields(z, z, z, phi)
        first = s.drops()
        again = s.drops()
    ref_cells, ref_deq = drop_count(phi, 2 * np.pi / (n - 1))
    assert np.array_equal(first[0], ref_cells) and np.array_equal(again[0], ref_cells)
    assert np.allclose(first[1], ref_deq, rtol=1e-15, atol=0)
