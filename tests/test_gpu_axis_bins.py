"""Narrow bins far from their line, integrated over the whole axis in float.

Without a far field every line reaches every bin. One line much wider than a bin
is compared with the FP64 scorer where sinc^2 is away from its zeros, 2.25 to 2.75
first-zero widths from the centre: a float line energy is off by 1e-6 of itself,
which moves the phase by 3e-6 and the value by at most 2 pi cot(pi / 4) times that,
2e-5; the float weight carries 1e-5, the midpoint series 1e-6. 1e-4 bounds them. (A
bin width taken as a difference of phases is off by 2e-7 / width, 5e-4 here.)
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", ["uniform", "geometric"])
def test_narrow_bins_of_one_wide_line(axis, cuda_device):
    from pyrite_b200 import mc_cxr_spectrum
    from test_gpu_short_segments import _scene

    n_E = 9000
    E_grid = np.linspace(1000.0, 60000.0, n_E) if axis == "uniform" else np.geomspace(1000.0, 60000.0, n_E)
    L = np.array([1.0])
    for _ in range(2):  # the second time with the length that puts the axis' end 3 widths off
        seg, kw = _scene(L, 7, E_grid, 11)
        kw.update(exact_widths=None, device=cuda_device)
        one, pairs = mc_cxr_spectrum(seg, E_grid, "silicon", None, precision="fp64", return_pairs=True, **kw)
        E, a, w, good = (x[pairs[0][3].astype(bool)] for x in pairs[0])
        assert E.size == 1
        L = L * 3.0 * np.pi / (a * (E_grid[-1] - E))
    x = a[0] / np.pi * (E_grid - E[0])
    assert abs(x[-1] - 3.0) < 0.01
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, precision="mixed", **kw)
    far = (x > 2.25) & (x < 2.75)
    assert far.sum() > 200 and np.all(one[far] > 0.0)
    assert np.max(np.abs(got[far] - one[far]) / one[far]) <= 1e-4
