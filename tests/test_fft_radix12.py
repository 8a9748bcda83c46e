"""CPU model of the column passes' radix-12 first stage (sizes 3*2^k up to
384, mhit36_b200/csrc/fft.cuh; 768 starts with radix 4, as test_fft_layout.py
models it): the Good-Thomas index maps of the butterfly, and the
register-resident transform's exchange slots with it."""
import numpy as np
import pytest

import test_fft_layout as layout


def test_dft12_index_maps():
    """n = 4 n1 + 3 n2, k = 4 k1 + 9 k2 (mod 12): DFTs of 3, then of 4, no twiddles between."""
    rng = np.random.default_rng(12)
    x = rng.standard_normal(12) + 1j * rng.standard_normal(12)
    v = x.copy()
    for n2 in range(4):
        i = [(4 * k + 3 * n2) % 12 for k in range(3)]
        v[i] = np.fft.fft(v[i])
    out = np.empty_like(v)
    for k1 in range(3):
        a = np.fft.fft(v[[(4 * k1 + 3 * n2) % 12 for n2 in range(4)]])
        out[[(4 * k1 + 9 * k2) % 12 for k2 in range(4)]] = a
    assert np.max(np.abs(out - np.fft.fft(x))) < 1e-14 * np.max(np.abs(x)) * 12


@pytest.mark.parametrize("n", (96, 192, 384))
@pytest.mark.parametrize("elem", [16, 8])
def test_column_slab_with_radix12(n, elem, monkeypatch):
    plain = layout.pick_radix
    monkeypatch.setattr(layout, "pick_radix", lambda rem, e: 12 if rem % 12 == 0 and e % 12 == 0 else plain(rem, e))
    cc = layout.lines_per_cta(n) * (1 if elem == 16 else 2)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((cc, n)) + 1j * rng.standard_normal((cc, n))
    at = lambda c, k: layout.pad(k) * cc + c  # noqa: E731
    y = layout.model_fft(x, -1, at, layout.reg_rows(n) * cc)
    assert np.max(np.abs(y - np.fft.fft(x, axis=1))) < 1e-9 * np.max(np.abs(y))
    z = layout.model_fft(y, +1, at, layout.reg_rows(n) * cc)
    assert np.max(np.abs(z / n - x)) < 1e-12 * n
