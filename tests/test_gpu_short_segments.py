"""Segments of next to no length in the bin-mean deposit of PXR + CBS.

A transport in float positions a history a fraction of a milliangstrom short of
a layer face now and then, and takes one more step of that length. Its line has
next to no mass (length squared), but an envelope w / (2 a^2) as large as any
other line's, which the far field spreads over the axis and the exact window,
as wide as the axis, takes out again.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

T = 5.0e6


def _scene(L, n_g, E_grid, seed):
    from pyrite_b200 import placeholder_data as P
    from pyrite_b200.tables import SILICON, diamond_hkls, reflection_rows, tilted_geometry

    rng = np.random.default_rng(seed)
    n = L.size
    beam, n_hat = tilted_geometry(np.deg2rad(20.0), np.deg2rad(10.0))
    v = beam + 0.01 * rng.normal(size=(n, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    r = np.stack([rng.normal(size=n), rng.normal(size=n), T * (0.1 + 0.8 * rng.random(n))], 1)
    seg = dict(v_hat=v, E_repr_keV=50000.0 - 100.0 * rng.random(n), L_ang=L, r_mid=r, elec_id=np.arange(n) % 4, Ne=4,
               thickness_ang=T)
    hkl = [h for h in diamond_hkls(9.0) if np.dot(h, (1, 1, 0)) > 0]  # the half space that radiates
    hkl = hkl[:: max(1, len(hkl) // n_g)][:n_g]
    rows = reflection_rows(SILICON, hkl, n_hat[None], surface_hkl=(2, 2, 0))
    kw = dict(tables=P.line_tables(SILICON, hkl, E_grid), n_hat=n_hat, rows=rows, line_quadrature="bin-mean",
              exact_widths=64.0)
    return seg, kw


def _layers(on):
    from pyrite_b200 import placeholder_data as P
    from pyrite_b200.tables import SILICON

    if not on:
        return {}
    comp = [("Si", SILICON.n_atoms_per_ang3)]
    mu = P.exact_mu_table(comp)
    return dict(layers=[(0.0, 0.4 * T, comp), (0.4 * T, T, comp)], mu_tables=[mu, mu])


@pytest.mark.parametrize("layered", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_E", [300, 2048])
def test_short_segments_among_ordinary_ones(n_E, precision, layered, cuda_device):
    """70 segments of 1e-14 to 1e-2 Angstrom among 40 ordinary ones leave the
    spectrum as it is: finite, and off by the rounding of their envelopes, at most
    twice the ordinary lines': FP64 1e-12 of the peak, mixed 2e-6 (float partial
    sums 1e-6, the envelopes' products 5e-7)."""
    from pyrite_b200 import mc_cxr_spectrum

    rng = np.random.default_rng(n_E)
    E_grid = np.linspace(1000.0, 60000.0, n_E)
    L = 1.5e5 * (0.2 + rng.exponential(size=110))
    short = np.zeros(110, dtype=bool)
    short[rng.permutation(110)[:70]] = True
    L[short] = np.logspace(-14, -2, 70)
    seg, kw = _scene(L, 40, E_grid, n_E)
    kw.update(_layers(layered), precision=precision, device=cuda_device)
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, **kw)
    alone = {k: (v[~short] if isinstance(v, np.ndarray) else v) for k, v in seg.items()}
    ref = mc_cxr_spectrum(alone, E_grid, "silicon", None, **kw)
    assert np.all(np.isfinite(got)) and np.max(ref) > 0.0
    assert np.max(np.abs(got - ref)) <= (1e-12 if precision == "fp64" else 2e-6) * np.max(ref)


@pytest.mark.parametrize("layered", [False, True])
@pytest.mark.parametrize("L", [1e-12, 1e-8, 1e-6, 1e-4])
def test_short_segments_alone_leave_rounding_of_their_envelope(L, layered, cuda_device):
    """Mixed precision, a few lines that are all envelope: what the far field
    spreads at D bins and the window takes out again differ by the rounding of
    two products and of a sum of at most 32 float terms, 4e-6 of the envelope
    wherever the bin lies (a difference of two edge values would leave 6e-8 D of
    it: 1e-4 at the axis' ends). Within two bins of a line there is no envelope;
    a float antiderivative leaves 1e-6 of w / a a bin."""
    from pyrite_b200 import mc_cxr_spectrum

    n_E = 2048
    E_grid = np.linspace(1000.0, 60000.0, n_E)
    seg, kw = _scene(np.full(3, L), 7, E_grid, 11)
    kw.update(_layers(layered), device=cuda_device)
    ref, pairs = mc_cxr_spectrum(seg, E_grid, "silicon", None, precision="fp64", return_pairs=True, **kw)
    E, a, w, good = (x[pairs[0][3].astype(bool)] for x in pairs[0])
    assert E.size >= 3
    W = E_grid[1] - E_grid[0]
    c = np.floor((E - (E_grid[0] - 0.5 * W)) / W)
    D = np.abs(np.arange(n_E)[None, :] - c[:, None])
    env = np.where(D > 1, (w / (2.0 * a * a))[:, None] / (W * W * (np.maximum(D, 2) ** 2 - 0.25)), 0.0).sum(0)
    bound = (4e-6 * env + 1e-6 * np.sum(w / a) / W) / seg["Ne"]
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, precision="mixed", **kw)
    assert np.all(np.isfinite(got))
    # line weights below the smallest normal float vanish on the mixed path
    assert np.all(np.abs(got - ref) <= bound + float(np.finfo(np.float32).tiny))
