"""Energy windows of the mixed bremsstrahlung scorer's depth-node form.

A list whose electrons slow down is scored window by window (a quarter octave
of the electron energy each, from 2.5 times the highest photon energy up), the
rest by the per-(segment, energy) kernels. Bounds: where every segment lies in
a window, 1e-6 of each direction's peak against the FP64 scorer (the fit's 1e-7
and float sums of ~1e-7, as for the single window); with segments left to the
per-(segment, energy) kernels, theirs, 1e-4.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _segments(E, seed, thickness=1.0e7):
    rng = np.random.default_rng(seed)
    n = E.size
    v = rng.normal(size=(n, 3))
    v[:, 2] += 1.0
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    z = thickness * (0.001 + 0.998 * rng.random(n))
    L = 200.0 * (np.maximum(E, 1.0) / 8.0) ** 0.8 * rng.exponential(size=n)
    L = np.maximum(np.minimum(L, 2.0 * np.minimum(z, thickness - z) / np.maximum(np.abs(v[:, 2]), 1e-3)), 1.0)
    r = np.stack([np.zeros(n), np.zeros(n), z], 1)
    return dict(v_hat=v, E_repr_keV=E, L_ang=L, r_mid=r, elec_id=np.arange(n) // 100, Ne=(n + 99) // 100,
                thickness_ang=thickness)


def _directions(both):
    th = np.linspace(0.30, 0.33, 6)
    n = np.stack([np.sin(th), np.zeros_like(th), -np.cos(th)], axis=1)
    if both:
        n[::2, 2] *= -1.0
    return n


def _compare(E, E_grid, comp, both, tol, cuda_device):
    from pyrite_b200 import mc_brem_spectrum

    seg = _segments(E, E.size)
    mu = 2.0e-4 * (1000.0 / E_grid) ** 2.8 + 1.0e-8
    kw = dict(composition=comp, n_hat=_directions(both), mu=mu, device=cuda_device)
    ref = mc_brem_spectrum(seg, E_grid, precision="fp64", **kw)
    got = mc_brem_spectrum(seg, E_grid, precision="mixed", **kw)
    for g, r in zip(got, ref):
        assert np.max(np.abs(g - r)) <= tol * np.max(np.abs(r))


@pytest.mark.parametrize("both", [False, True])
@pytest.mark.parametrize("comp", [[("Si", 0.05)], [("Si", 0.0266), ("O", 0.0532)]])
def test_every_segment_in_a_window(comp, both, cuda_device):
    E = np.exp(np.random.default_rng(3).uniform(np.log(165.0), np.log(1.0e4), 20001))
    E[:6] = [256.0, 320.0, 384.0, np.nextafter(512.0, 0.0), 512.0, 8192.0]  # on the windows' edges
    _compare(E, np.linspace(1000.0, 60000.0, 2047), comp, both, 1e-6, cuda_device)


@pytest.mark.parametrize("n", [511, 512, 513, 1025])
def test_tiles_of_a_window(n, cuda_device):
    """Windows of n segments, one more and one less than a tile among them,
    and empty ones between."""
    E = np.concatenate([np.full(n, T) for T in (170.0, 300.0, 1000.0, 1100.0, 1500.0, 6000.0, 9000.0)] * (9000 // n // 6 + 1))
    _compare(E, np.linspace(1000.0, 60000.0, 2048), [("Si", 0.05)], False, 1e-6, cuda_device)


@pytest.mark.parametrize("n_E", [2045, 75])
def test_segments_outside_every_window(n_E, cuda_device):
    """Energies below the lowest window, beyond the counted range, at the tip of
    the spectrum and without radiation; 75 energies stay with one window."""
    rng = np.random.default_rng(n_E)
    E = np.exp(rng.uniform(np.log(2.0), np.log(2.0e4), 15000))
    E[::97] = 0.0
    E[5], E[6] = 2.0e6, 1.04e6
    _compare(E, np.linspace(500.0, 102300.0, n_E), [("Si", 0.05)], False, 1e-4, cuda_device)
