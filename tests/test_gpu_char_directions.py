"""Characteristic-line yields by direction group, against the oracle.

Directions on one exit face within 2 % (FP64) or 1 % (mixed) of one another share
exponentials through moments; wider groups and both faces are scored one by one;
more than 16 directions take several groups. FP64: sums of n terms of 1e-16 and a
moment truncation of 2e-17 of the unattenuated term, 1e-12 of the yield. Mixed: a
float exponential of an optical depth up to 20 carries 1e-6 of itself and the
moments' 1 - e^-x 4e-7: 1e-5.
"""

import numpy as np
import pytest

from oracle import characteristic as OC
from test_gpu_brem_moments import DIRS, SLAB, _directions, _segments

pytestmark = pytest.mark.gpu

LAYERS = [(0.0, 5.0e5), (5.0e5, 1.2e6), (1.2e6, 2.0e6)]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("layered", [False, True])
@pytest.mark.parametrize("n_seg", [1, 33, 3000])
@pytest.mark.parametrize("n_dir,rho,face", DIRS)
def test_yields_by_direction_group(n_dir, rho, face, n_seg, layered, precision, tol, cuda_device):
    from pyrite_b200 import mc_characteristic_spectrum
    from pyrite_b200 import placeholder_data as P

    seg = _segments(n_seg, 6)
    lines = P.characteristic_lines("W")
    comps = [[("C", 0.113)], [("Si", 0.05)], [("W", 0.063)]] if layered else [[("Si", 0.05)]]
    mu = np.stack([P.mu_total(c, lines.line_E) for c in comps])
    E = np.linspace(5000.0, 70000.0, 50)
    n_hat = _directions(n_dir, rho, face)
    _spec, y, kept = mc_characteristic_spectrum(seg, E, lines=lines, n_atoms_per_ang3=0.063, n_hat=n_hat,
                                                mu_by_line=mu, layers=LAYERS if layered else None,
                                                precision=precision, device=cuda_device, return_yields=True)
    off = np.cumsum([0] + [e.size for e in lines.shell_E])
    oseg = dict(r_mid=seg["r_mid"], v_hat=seg["v_hat"], L=seg["L_ang"], E_keV=seg["E_repr_keV"], elec_id=seg["elec_id"])
    for got, nh in zip(np.atleast_2d(y), n_hat):
        ref = OC.line_yields(oseg, nh, SLAB, 0.063, np.concatenate(lines.shell_E), np.concatenate(lines.shell_sigma), off,
                             lines.response[:, kept], mu[:, kept], layers=LAYERS if layered else None, Ne=seg["Ne"])
        np.testing.assert_allclose(got, ref, rtol=tol, atol=tol * np.max(np.abs(ref)))
