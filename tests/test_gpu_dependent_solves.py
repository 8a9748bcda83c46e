"""The stand-alone Poisson solves up to 128^3, whose kernels are launched to
start while the one before them drains: solves queued back to back share the
spectrum, and each reads its right-hand side where the solve before it wrote
its result, so a kernel that ran ahead of the one before it would show.  Both
as plain launches and as a captured graph.
"""
import pytest

pytestmark = pytest.mark.gpu

SOLVES = 8
# each solve's error is that of an FP64 FFT pair, ~log2(n^3) ulp of its largest
# value (3e-15); solving again damps every mode but k^2 = 1, so the errors of
# the chain add up to at most SOLVES of them: 3e-14, held to 1e-13
TOL = 1e-13


def _chain(rhs, n):
    """SOLVES solves in a row by torch's FFT: p -> -p_hat / k^2, mean 0."""
    import torch
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=rhs.device)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    f = torch.fft.fftn(rhs.reshape(n, n, n))
    f[0, 0, 0] = 0.0
    return torch.fft.ifftn(f / (-k2) ** SOLVES).real.reshape(-1)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n", [32, 64, 96, 128])
def test_chained_solves(n, graph):
    import torch
    from mhit36_b200 import capi
    lib = capi.load_library()
    gen = torch.Generator(device="cuda").manual_seed(n)
    rhs = torch.randn(n ** 3, dtype=torch.float64, device="cuda", generator=gen)
    want = _chain(rhs, n)
    buf = [rhs.clone(), torch.empty_like(rhs)]
    stream = torch.cuda.Stream()

    def solves():
        for s in range(SOLVES):
            rc = lib.mhit_poisson_noalloc(buf[s & 1].data_ptr(), buf[(s & 1) ^ 1].data_ptr(), n, 0, 1,
                                          stream.cuda_stream)
            assert rc == capi.MHIT_OK, lib.mhit_strerror(rc)

    torch.cuda.synchronize()
    solves()
    stream.synchronize()
    if graph:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            solves()
        buf[0].copy_(rhs)
        buf[1].fill_(float("nan"))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
    got = buf[SOLVES & 1]
    assert float((got - want).abs().max() / want.abs().max()) <= TOL


@pytest.mark.parametrize("n", [32, 64, 96, 128, 192])  # 192: plain launches
def test_chained_solves_through_a_handle(n):
    import torch
    from mhit36_b200 import Solver
    from mhit36_b200.config import InputParams
    gen = torch.Generator(device="cuda").manual_seed(n)
    rhs = torch.randn(n ** 3, dtype=torch.float64, device="cuda", generator=gen)
    want = _chain(rhs, n)
    buf = [rhs.clone(), torch.empty_like(rhs)]
    torch.cuda.synchronize()
    with Solver(n, InputParams(grid_mode=1), phase_field=False) as s:
        for q in range(SOLVES):
            s.poisson_device(buf[q & 1].data_ptr(), buf[(q & 1) ^ 1].data_ptr())
        torch.cuda.synchronize()
    got = buf[SOLVES & 1]
    assert float((got - want).abs().max() / want.abs().max()) <= TOL
