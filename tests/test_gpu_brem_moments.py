"""The direction-moment forms of the bremsstrahlung scorers against the oracle.

One exit face and a narrow band of path factors share two exponentials a
(segment, energy) through moments about the band centre: FP64 slab and stack to
order 0, 5 or 9 by the spread (truncation below 2e-17 of the unattenuated term),
the mixed stack to order 3 (2e-9). Wider bands and directions through both faces
stay per direction. Spreads on both sides of each limit, a single direction, a
group of 17 (two launches), segments across layer boundaries, an energy above
some segments' tip.

FP64 sums n terms of rounding 1e-16 each, the Born logarithm of the difference
p_i - p_f carries 5e-12 / 11 of a term at k = 1 keV and 50 MeV, of either sign:
1e-12 of the peak. Mixed: the float cross section and transmissions carry a few
1e-7 each, the layered moments' 1 - e^-x up to 4e-7: 2e-6 of the peak.
"""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SLAB = 2.0e6
LAYERS = [(0.0, 5.0e5, [("C", 0.113)]), (5.0e5, 1.2e6, [("Si", 0.05), ("O", 0.1)]), (1.2e6, 2.0e6, [("W", 0.063)])]
Z = {"C": 6.0, "Si": 14.0, "O": 8.0, "W": 74.0}


def _segments(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, 3)) + np.array([0.0, 0.0, 1.5])
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    z = SLAB * (0.02 + 0.96 * rng.random(n))
    L = np.minimum(1.0e5 * rng.exponential(size=n), 1.9 * np.minimum(z, SLAB - z) / np.abs(v[:, 2]))
    return dict(v_hat=v, E_repr_keV=30.0 + 20000.0 * rng.random(n) ** 3, L_ang=L,
                r_mid=np.stack([rng.normal(size=n), rng.normal(size=n), z], 1), elec_id=np.arange(n) // 5,
                Ne=(n + 4) // 5, thickness_ang=SLAB)


def _directions(n_dir, rho, face):
    c = np.ones(1) if n_dir == 1 else np.linspace(1.0 - rho, 1.0 + rho, n_dir) / (1.0 - rho)
    nz = 0.9 / c
    n = np.stack([np.sqrt(1.0 - nz**2), np.zeros(n_dir), nz], 1)
    if face == "up":
        n[:, 2] *= -1.0
    elif face == "both":
        n[::2, 2] *= -1.0
    return n


def _oseg(seg, on=slice(None)):
    return dict(E_keV=seg["E_repr_keV"][on], L_ang=seg["L_ang"][on], r_mid=seg["r_mid"][on], v_hat=seg["v_hat"][on])


DIRS = [(1, 0.0, "down"), (16, 0.0013, "up"), (9, 0.0025, "down"), (16, 0.0095, "up"), (5, 0.018, "down"),
        (17, 0.03, "up"), (4, 0.001, "both")]


@pytest.mark.parametrize("n_dir,rho,face", DIRS)
def test_fp64_slab(n_dir, rho, face, cuda_device):
    from pyrite_b200 import mc_brem_spectrum
    from pyrite_b200 import placeholder_data as P

    seg, comp = _segments(300, 3), LAYERS[1][2]
    E = np.linspace(1000.0, 60000.0, 301)
    n_hat, mu = _directions(n_dir, rho, face), P.mu_total(LAYERS[1][2], E)
    got = mc_brem_spectrum(seg, E, composition=comp, n_hat=n_hat, mu=mu, precision="fp64", device=cuda_device)
    for g, nh in zip(np.atleast_2d(got), n_hat):
        ref = oracle.brem_spectrum(_oseg(seg), [Z[e] for e, _ in comp], [n for _, n in comp], SLAB, nh, E, mu, seg["Ne"])
        assert np.max(np.abs(g - ref)) <= 1e-12 * np.max(ref)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 2e-6)])
@pytest.mark.parametrize("n_dir,rho,face", DIRS)
def test_stack(n_dir, rho, face, precision, tol, cuda_device):
    from pyrite_b200 import mc_brem_spectrum
    from pyrite_b200 import placeholder_data as P

    seg = _segments(700, 4)
    E = np.linspace(1000.0, 60000.0, 257)
    n_hat = _directions(n_dir, rho, face)
    mu = np.stack([P.mu_total(c, E) for _, _, c in LAYERS])
    top, bot = np.array([l[0] for l in LAYERS]), np.array([l[1] for l in LAYERS])
    seg["layer"] = np.searchsorted(top[1:], seg["r_mid"][:, 2], side="right").astype(np.int32)
    for k, (_a, _b, comp) in enumerate(LAYERS):
        got = mc_brem_spectrum(seg, E, composition=comp, n_hat=n_hat, layers=LAYERS, mu_layer=mu, emit_layer=k,
                               precision=precision, device=cuda_device)
        on = seg["layer"] == k
        for g, nh in zip(np.atleast_2d(got), n_hat):
            ref = oracle.brem_spectrum_layered(_oseg(seg, on), [Z[e] for e, _ in comp], [n for _, n in comp],
                                               oracle.LayerEscape(top, bot), nh, E, mu, seg["Ne"])
            assert np.max(np.abs(g - ref)) <= tol * np.max(ref)


@pytest.mark.parametrize("f", [[1.0, 1.3], [1.0, 1.0097, 1.0099, 1.02], [-1.0, 1.0, -1.3, 1.3], [133.0, -133.0, 400.0, -400.0],
                               [1.0, 1.1, 1.2, 1.3, 1.4], [1.0, -1.0, 1.2, -1.2, 1.5]])
def test_mixed_stack_direction_groups(f, cuda_device):
    """Directions in two to four narrow groups (path factors over that of the
    first, the sign the face) share the exponentials of each group; five groups,
    or more than 16 directions in a launch, are the per-direction form's. Four
    directions a group within 0.4 % of it."""
    from pyrite_b200 import mc_brem_spectrum
    from pyrite_b200 import placeholder_data as P

    seg = _segments(600, 9)
    E = np.linspace(1000.0, 60000.0, 129)
    fs = np.concatenate([np.asarray(f) * (1.0 + s) for s in (0.0, 0.001, -0.002, 0.002)][: 16 // len(f)])
    nz = np.sign(fs) * 0.9 / np.maximum(np.abs(fs), 1.0)
    n_hat = np.stack([np.sqrt(1.0 - nz**2), np.zeros(fs.size), nz], 1)
    mu = np.stack([P.mu_total(c, E) for _, _, c in LAYERS])
    top, bot = np.array([l[0] for l in LAYERS]), np.array([l[1] for l in LAYERS])
    seg["layer"] = np.searchsorted(top[1:], seg["r_mid"][:, 2], side="right").astype(np.int32)
    for k, (_a, _b, comp) in enumerate(LAYERS):
        got = mc_brem_spectrum(seg, E, composition=comp, n_hat=n_hat, layers=LAYERS, mu_layer=mu, emit_layer=k,
                               precision="mixed", device=cuda_device)
        on = seg["layer"] == k
        for g, nh in zip(got, n_hat):
            ref = oracle.brem_spectrum_layered(_oseg(seg, on), [Z[e] for e, _ in comp], [n for _, n in comp],
                                               oracle.LayerEscape(top, bot), nh, E, mu, seg["Ne"])
            # along the surface all light is attenuated, and a float e^-x carries x ulps
            tol = 2e-6 * max(1.0, abs(1.0 / nh[2]) / 10.0)
            assert np.max(np.abs(g - ref)) <= tol * np.max(ref)
