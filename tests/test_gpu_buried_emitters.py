"""Emitters below an absorber: spectra and yields relative to what is left of them.

Narrow groups of directions share exponentials through moments, whose truncation
is relative to the term without attenuation. Here all light (at a photon energy,
or at all of them) comes from many attenuation lengths below the exit face, the
segments in any order of depth, with slow electrons near the face that do not
reach the higher photon energies. Every value is compared with the oracle's to a
bound relative to itself.

FP64: 1e-12 for the sums and the Born logarithm (as above the surface), rounding of
an optical depth of up to 200, 4 x 2.2e-16 x 200: 2e-12. Mixed: 2e-6 (bremsstrahlung) or
1e-5 (lines) as above the surface, and four roundings of the optical depth, 2.4e-7
of it.
"""

import numpy as np
import pytest

import oracle
from oracle import characteristic as OC
from test_gpu_brem_moments import LAYERS, SLAB, Z, _directions

pytestmark = pytest.mark.gpu

DIRS = [(1, 0.0, "down"), (16, 0.0013, "up"), (9, 0.0019, "down"), (16, 0.0095, "up"), (5, 0.018, "down"), (16, 0.019, "up")]


def _segments(n, lo, hi, order, up, veil, seed):
    """Depths from lo to hi (fractions of the slab), sorted towards or away from
    the exit face or not; ``veil``: every fifth is an electron of 5 to 15 keV near
    the exit face."""
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, 3)) + np.array([0.0, 0.0, 1.5])
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    z = lo + (hi - lo) * (0.02 + 0.96 * rng.random(n))
    if order != "random":
        z = np.sort(z) if (order == "towards") != up else np.sort(z)[::-1].copy()
    L = np.minimum(0.1 * (hi - lo) * rng.exponential(size=n), 1.9 * np.minimum(z - lo, hi - z) / np.abs(v[:, 2]))
    E = 100.0 + 20000.0 * rng.random(n) ** 3
    if veil:
        E[::5] = 5.0 + 10.0 * rng.random(E[::5].size)
        z[::5] = (0.001 + 0.01 * rng.random(E[::5].size)) if up else (0.989 + 0.01 * rng.random(E[::5].size))
        L[::5] = 1e-4
    return dict(v_hat=v, E_repr_keV=E, L_ang=SLAB * L, r_mid=np.stack([rng.normal(size=n), rng.normal(size=n), SLAB * z], 1),
                elec_id=np.arange(n) // 5, Ne=(n + 4) // 5, thickness_ang=SLAB)


def _oseg(seg, on=slice(None)):
    return dict(E_keV=seg["E_repr_keV"][on], L_ang=seg["L_ang"][on], r_mid=seg["r_mid"][on], v_hat=seg["v_hat"][on])


@pytest.mark.parametrize("veil", [False, True])
@pytest.mark.parametrize("order", ["random", "towards", "away"])
@pytest.mark.parametrize("n_dir,rho,face", DIRS)
def test_fp64_slab(n_dir, rho, face, order, veil, cuda_device):
    from pyrite_b200 import mc_brem_spectrum

    up = face == "up"
    seg = _segments(700, *((0.8, 1.0) if up else (0.0, 0.2)), order, up, veil, 3)
    E = np.linspace(1000.0, 60000.0, 301)
    mu = np.geomspace(150.0, 0.5, E.size) / SLAB
    n_hat, comp = _directions(n_dir, rho, face), LAYERS[1][2]
    got = mc_brem_spectrum(seg, E, composition=comp, n_hat=n_hat, mu=mu, precision="fp64", device=cuda_device)
    for g, nh in zip(np.atleast_2d(got), n_hat):
        ref = oracle.brem_spectrum(_oseg(seg), [Z[e] for e, _ in comp], [n for _, n in comp], SLAB, nh, E, mu, seg["Ne"])
        assert ref.min() > 0.0
        assert np.all(np.abs(g - ref) <= 2e-12 * ref)


def _stack(seg, E, n_hat, up, precision, emit, cuda_device):
    """(got, oracle, bound) of the bottom (up) or top layer's segments."""
    from pyrite_b200 import mc_brem_spectrum

    mu = np.stack([np.geomspace(40.0, 0.5, E.size), np.geomspace(30.0, 0.2, E.size), np.geomspace(50.0, 1.0, E.size)]) / SLAB
    top, bot = np.array([l[0] for l in LAYERS]), np.array([l[1] for l in LAYERS])
    k, comp = (2, LAYERS[2][2]) if up else (0, LAYERS[0][2])
    if emit:
        seg["layer"] = np.searchsorted(top[1:], seg["r_mid"][:, 2], side="right").astype(np.int32)
    got = mc_brem_spectrum(seg, E, composition=comp, n_hat=n_hat, layers=LAYERS, mu_layer=mu, emit_layer=k if emit else None,
                           precision=precision, device=cuda_device)
    on = seg["layer"] == k if emit else slice(None)
    ref = np.stack([oracle.brem_spectrum_layered(_oseg(seg, on), [Z[e] for e, _ in comp], [n for _, n in comp],
                                                 oracle.LayerEscape(top, bot), nh, E, mu, seg["Ne"]) for nh in n_hat])
    tau = (mu * (bot - top)[:, None]).sum(0)[None, :] / np.abs(n_hat[:, 2:])
    return np.atleast_2d(got), ref, 2e-12 if precision == "fp64" else 2e-6 + 2.4e-7 * tau


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("emit", [False, True])
@pytest.mark.parametrize("order", ["random", "towards", "away"])
@pytest.mark.parametrize("n_dir,rho,face", DIRS)
def test_stack(n_dir, rho, face, order, emit, precision, cuda_device):
    """The bottom layer's light through the top face, or the top layer's through
    the bottom one."""
    up = face == "up"
    seg = _segments(900, *((0.6, 1.0) if up else (0.0, 0.25)), order, up, False, 4)
    got, ref, tol = _stack(seg, np.linspace(1000.0, 60000.0, 257), _directions(n_dir, rho, face), up, precision, emit,
                           cuda_device)
    assert ref.min() > 0.0
    assert np.all(np.abs(got - ref) <= tol * ref)


@pytest.mark.parametrize("order", ["random", "towards", "away"])
@pytest.mark.parametrize("f", [[1.0, 1.2, 1.5], [1.0, -1.0, 1.3, -1.4]])
def test_mixed_stack_direction_groups(f, order, cuda_device):
    fs = np.concatenate([np.asarray(f) * (1.0 + s) for s in (0.0, 0.004, -0.004, 0.002)])
    nz = np.sign(fs) * 0.9 / np.abs(fs)
    n_hat = np.stack([np.sqrt(1.0 - nz**2), np.zeros(fs.size), nz], 1)
    seg = _segments(900, 0.6, 1.0, order, True, False, 5)
    got, ref, tol = _stack(seg, np.linspace(1000.0, 60000.0, 257), n_hat, True, "mixed", True, cuda_device)
    assert ref.min() > 0.0
    assert np.all(np.abs(got - ref) <= tol * ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("layered", [False, True])
@pytest.mark.parametrize("order", ["random", "towards", "away"])
@pytest.mark.parametrize("n_dir,rho,face", DIRS)
def test_characteristic_yields(n_dir, rho, face, order, layered, precision, cuda_device):
    from pyrite_b200 import mc_characteristic_spectrum
    from pyrite_b200 import placeholder_data as P

    up = face == "up"
    # electrons of 5 to 15 keV near the face: too slow for the K lines
    seg = _segments(900, *((0.6, 1.0) if up else (0.0, 0.25)), order, up, layered, 6)
    lines = P.characteristic_lines("W")
    n_line = lines.line_E.size
    layers = [(a, b) for a, b, _ in LAYERS] if layered else None
    mu = np.stack([np.geomspace(50.0, 0.5, n_line)] * (3 if layered else 1)) * ([[1.0], [0.7], [1.3]] if layered else 1.0) / SLAB
    n_hat = _directions(n_dir, rho, face)
    _spec, y, kept = mc_characteristic_spectrum(seg, np.linspace(5000.0, 70000.0, 50), lines=lines, n_atoms_per_ang3=0.063,
                                                n_hat=n_hat, mu_by_line=mu, layers=layers, precision=precision,
                                                device=cuda_device, return_yields=True)
    off = np.cumsum([0] + [e.size for e in lines.shell_E])
    oseg = dict(r_mid=seg["r_mid"], v_hat=seg["v_hat"], L=seg["L_ang"], E_keV=seg["E_repr_keV"], elec_id=seg["elec_id"])
    for got, nh in zip(np.atleast_2d(y), n_hat):
        ref = OC.line_yields(oseg, nh, SLAB, 0.063, np.concatenate(lines.shell_E), np.concatenate(lines.shell_sigma), off,
                             lines.response[:, kept], mu[:, kept], layers=layers, Ne=seg["Ne"])
        assert ref.min() > 0.0
        tau = mu[:, kept].max(0) * SLAB / abs(nh[2])
        assert np.all(np.abs(got - ref) <= (2e-12 if precision == "fp64" else 1e-5 + 2.4e-7 * tau) * ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("f", [[1.0], [1.0, 1.005], [1.0, -1.0, 1.3, -1.4]])
@pytest.mark.parametrize("scale", [1e3, 1e6, 1e9, 1e12])
def test_no_light_left(scale, f, precision, cuda_device):
    """Optical depths far beyond what an exponential of it can hold: zero, as the
    oracle has it, and not a number that float noise of the depth makes."""
    fs = np.asarray(f)
    nz = np.sign(fs) * 0.9 / np.abs(fs)
    n_hat = np.stack([np.sqrt(1.0 - nz**2), np.zeros(fs.size), nz], 1)
    seg = _segments(300, 0.3, 0.6, "random", True, False, 8)
    from pyrite_b200 import mc_brem_spectrum

    E = np.linspace(100.0, 2000.0, 40)
    mu = np.full((3, E.size), scale * 1e3 / SLAB)
    got = mc_brem_spectrum(seg, E, composition=LAYERS[1][2], n_hat=n_hat, layers=LAYERS, mu_layer=mu, precision=precision,
                           device=cuda_device)
    assert np.all(got == 0.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("f", [[450.0], [450.0, 1300.0], [3.0, -3.0, 450.0, -1300.0]])
@pytest.mark.parametrize("tau", [1.0, 1e3, 1e5, 1e7])
def test_segments_through_both_faces_of_an_opaque_stack(tau, f, precision, cuda_device):
    """Each segment runs from face to face, so a direction sees its end on the
    exit face whatever the optical depth below: FP64 2e-12 of a value, mixed 4e-6
    (the float cross section, depth ratio and exponential, a few 1e-7 each)."""
    from pyrite_b200 import mc_brem_spectrum

    rng = np.random.default_rng(1)
    fs = np.asarray(f)
    nz = np.sign(fs) / np.abs(fs)
    n_hat = np.stack([np.sqrt(1.0 - nz**2), np.zeros(fs.size), nz], 1)
    n = 40
    v = np.tile([np.sqrt(0.75), 0.0, 0.5], (n, 1))
    L = np.full(n, 2.0 * SLAB)
    r = np.stack([np.zeros(n), np.zeros(n), np.full(n, 0.5 * SLAB)], 1)
    seg = dict(v_hat=v, E_repr_keV=50.0 + 1000.0 * rng.random(n), L_ang=L, r_mid=r, elec_id=np.arange(n), Ne=n, thickness_ang=SLAB)
    E = np.linspace(1000.0, 40000.0, 60)
    comp = LAYERS[2][2]
    top, bot = np.array([l[0] for l in LAYERS]), np.array([l[1] for l in LAYERS])
    mu = np.stack([np.geomspace(tau, 0.1 * tau, E.size) / SLAB * k for k in (1.0, 0.7, 1.4)])
    got = np.atleast_2d(mc_brem_spectrum(seg, E, composition=comp, n_hat=n_hat, layers=LAYERS, mu_layer=mu,
                                         precision=precision, device=cuda_device))
    for g, nh in zip(got, n_hat):
        ref = oracle.brem_spectrum_layered(_oseg(seg), [Z[e] for e, _ in comp], [x for _, x in comp],
                                           oracle.LayerEscape(top, bot), nh, E, mu, seg["Ne"])
        assert ref.min() > 0.0
        assert np.all(np.abs(g - ref) <= (2e-12 if precision == "fp64" else 4e-6) * ref)
