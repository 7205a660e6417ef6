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


@pytest.mark.parametrize("n_E", [3991, 3997, 4001, 4003])
def test_wide_bins_of_a_resolved_line(n_E, cuda_device):
    """Bins of 0.11 first-zero widths, 0.8 eV, about the centre of a line above 4.1
    keV, where a float edge is off by up to 2.4e-4 eV. Against the oracle's bin means
    of the line that the mixed scorer found: moving a bin by that much changes its
    mean by at most 1.7 x 0.14 x 2.4e-4 = 6e-5 within a quarter width of the centre;
    with the antiderivative's 5e-7 of 0.11, 7e-5. (A mass between float edges divided
    by the width of the FP64 edges is off by up to 6e-4.)"""
    import oracle
    from pyrite_b200 import mc_cxr_spectrum
    from test_gpu_short_segments import _scene

    wide = np.linspace(1000.0, 60000.0, 2048)
    seg, kw = _scene(np.full(3, 1.0e5), 7, wide, 11)
    kw.update(exact_widths=None, device=cuda_device, precision="mixed", return_pairs=True)
    _, pairs = mc_cxr_spectrum(seg, wide, "silicon", None, **kw)
    E, a, w, good = pairs[0]
    k = int(np.argmax(np.where(good, E, 0.0)))
    assert E[k] > 4200.0
    n_g = kw["rows"].G.shape[0]
    one = {x: (v[k // n_g:k // n_g + 1] if isinstance(v, np.ndarray) else v) for x, v in seg.items()}
    one["L_ang"] = one["L_ang"] * (0.11 * np.pi / (a[k] * 0.8))
    E_grid = np.linspace(E[k] - 0.4 * n_E, E[k] + 0.4 * n_E, n_E)
    got, pairs = mc_cxr_spectrum(one, E_grid, "silicon", None, **kw)
    E, a, w, good = (x[pairs[0][3].astype(bool)] for x in pairs[0])
    assert E.size == 1
    edges = oracle.energy_bin_edges(E_grid)
    ref = oracle.reduce_binmean(E, a, w, edges) / seg["Ne"]
    near = np.abs(a[0] / np.pi * (E_grid - E[0])) < 0.25
    assert 4 <= near.sum() <= 5 and 0.1 < a[0] / np.pi * (edges[1] - edges[0]) < 0.14
    assert np.max(np.abs(got[near] - ref[near]) / ref[near]) <= 7e-5
