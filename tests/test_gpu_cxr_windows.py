"""The bin-mean deposit of the PXR + CBS scorer at the edges of its work split.

The oracle's FP64 lines are deposited here as the scorer defines it: exact bin
means (the oracle's sinc^2 antiderivative) within ``exact_widths`` first-zero
widths of each line, at least two bins a side, and beyond them the far envelope
expanded to second order about the line's centre bin. The cases put the line
count, rows, segments and window widths on both sides of the kernel's limits:
one pair, a last partial round, one row more than a chunk, windows of 3 to
several hundred bins a side (each lane grouping, the strips), bins below 0.1
first-zero widths (the midpoint series), a non-uniform axis, tiles without a
radiating segment.

FP64 bound: the midpoint series omits up to 2.5e-9 of a line's envelope and a
phase of 1e3 rad carries 1e-12, so 5e-9 of the peak. Mixed bound: a float line
energy is off by up to 1e-6 of it (test_gpu_cxr), 0.03 eV at 30 keV against
first-zero widths of 1 eV and more, so up to 3 % of a line's mass can cross a bin
edge, of either sign; summed over the bins 3e-2 of the spectrum bounds the worst
case of a single line and 2e-3 the average over many. Line weights below the
smallest normal float vanish on the mixed path.
"""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _scene(n_seg, n_g, E_grid, L_mean, seed):
    from pyrite_b200 import placeholder_data as P
    from pyrite_b200.tables import SILICON, diamond_hkls, reflection_rows, tilted_geometry

    rng = np.random.default_rng(seed)
    beam, n_hat = tilted_geometry(np.deg2rad(20.0), np.deg2rad(10.0))
    T = 5.0e6
    v = beam + 0.01 * rng.normal(size=(n_seg, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    r = np.stack([rng.normal(size=n_seg), rng.normal(size=n_seg), T * (0.1 + 0.8 * rng.random(n_seg))], 1)
    seg = dict(v_hat=v, E_repr_keV=50000.0 - 100.0 * rng.random(n_seg), L_ang=L_mean * (0.2 + rng.exponential(size=n_seg)),
               r_mid=r, elec_id=np.arange(n_seg) // 4, Ne=(n_seg + 3) // 4, thickness_ang=T)
    hkl = [h for h in diamond_hkls(9.0) if np.dot(h, (1, 1, 0)) > 0]  # the half space that radiates
    hkl = hkl[:: max(1, len(hkl) // n_g)][:n_g]
    assert len(hkl) == n_g
    rows = reflection_rows(SILICON, hkl, n_hat[None], surface_hkl=(2, 2, 0))
    return seg, rows, P.line_tables(SILICON, hkl, E_grid), n_hat


def _lines(seg, rows, tables, n_hat, E_grid):
    pad = 0.2 * (E_grid[-1] - E_grid[0])
    t = dict(G=rows.G, ES=rows.ES[0], EP=rows.EP[0], WM=rows.WM, row_table=rows.row_table, E_tab=tables.E_tab,
             chi_re=tables.chi_re, chi_im=tables.chi_im, u_re=tables.u_re, u_im=tables.u_im, log_mu=tables.log_mu,
             delta=tables.delta, lo_keep=E_grid[0] - pad, hi_keep=E_grid[-1] + pad)
    oseg = dict(v_hat=seg["v_hat"], E_keV=seg["E_repr_keV"], L_ang=seg["L_ang"], r_mid=seg["r_mid"],
                elec_id=seg["elec_id"])
    E, a, w, good = oracle.cxr_lines(t, n_hat, seg["thickness_ang"], oseg, seg["Ne"])
    return E[good], a[good], w[good]


def _deposit(E, a, w, edges, widths):
    n = edges.size - 1
    if not widths:
        return oracle.reduce_binmean(E, a, w, edges)
    W = (edges[-1] - edges[0]) / n
    spec = np.zeros(n)
    b = np.arange(n)
    for Er, aj, wj in zip(E, a, w):
        c = int(np.floor((Er - edges[0]) / W))
        K = max(2, int(np.ceil(widths * np.pi / (aj * W))))
        b0, b1 = max(0, c - K), min(n - 1, c + K)
        if b1 >= b0:
            spec[b0:b1 + 1] += oracle.reduce_binmean(np.array([Er]), np.array([aj]), np.array([wj]), edges[b0:b1 + 2])
        far = np.abs(b - c) > K
        Ec = edges[0] + (c + 0.5) * W
        A, B, d = edges[:-1][far] - Ec, edges[1:][far] - Ec, Er - Ec
        AB = A * B
        spec[far] += wj / (2 * aj * aj) * (1 / AB + d * (A + B) / AB**2 + d * d * (A * A + AB + B * B) / AB**3)
    return spec


CASES = [  # segments, rows, bins, first and last bin [eV], mean length [Angstrom], widths
    (1, 1, 40, 5000.0, 30000.0, 1.5e5, 64.0),
    (3, 7, 33, 2000.0, 50000.0, 1.5e5, 64.0),
    (17, 49, 31, 2000.0, 50000.0, 1.5e5, 64.0),
    (5, 121, 2048, 1000.0, 60000.0, 1.5e5, 64.0),
    (33, 48, 1500, 1000.0, 60000.0, 2.0e4, 64.0),
    (8, 60, 700, 1000.0, 60000.0, 1.0e3, 64.0),
    (8, 60, 900, 8000.0, 9000.0, 1.0e4, 64.0),
    (20, 120, 512, 1000.0, 60000.0, 1.5e5, 2.0),
    (9, 50, 257, 1000.0, 60000.0, 1.5e5, 0.0),
    (6, 20, 300, 8000.0, 8030.0, 2.0e4, 0.0),
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_seg,n_g,n_E,lo,hi,L,widths", CASES)
def test_deposit_matches_oracle_lines(n_seg, n_g, n_E, lo, hi, L, widths, precision, cuda_device):
    from pyrite_b200 import mc_cxr_spectrum

    E_grid = np.linspace(lo, hi, n_E)
    seg, rows, tables, n_hat = _scene(n_seg, n_g, E_grid, L, n_seg * 1000 + n_g)
    E, a, w = _lines(seg, rows, tables, n_hat, E_grid)
    ref = _deposit(E, a, w, oracle.energy_bin_edges(E_grid), widths) / seg["Ne"]
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, tables=tables, n_hat=n_hat, rows=rows,
                          line_quadrature="bin-mean", precision=precision, exact_widths=widths or None,
                          device=cuda_device)
    if E.size == 0:
        assert not got.any()
        return
    if precision == "fp64":
        assert np.max(np.abs(got - ref)) <= 5e-9 * np.max(np.abs(ref))
    else:
        floor = E.size * float(np.finfo(np.float32).tiny)
        assert np.sum(np.abs(got - ref)) <= (2e-3 if E.size > 100 else 3e-2) * np.sum(np.abs(ref)) + floor


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_deposit_on_a_non_uniform_axis(precision, cuda_device):
    from pyrite_b200 import mc_cxr_spectrum

    E_grid = np.geomspace(1000.0, 60000.0, 400)
    seg, rows, tables, n_hat = _scene(10, 30, E_grid, 1.0e5, 5)
    E, a, w = _lines(seg, rows, tables, n_hat, E_grid)
    ref = oracle.reduce_binmean(E, a, w, oracle.energy_bin_edges(E_grid)) / seg["Ne"]
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, tables=tables, n_hat=n_hat, rows=rows,
                          line_quadrature="bin-mean", precision=precision, exact_widths=64.0, device=cuda_device)
    if precision == "fp64":
        assert np.max(np.abs(got - ref)) <= 5e-9 * np.max(np.abs(ref))
    else:
        assert np.sum(np.abs(got - ref)) <= 2e-3 * np.sum(np.abs(ref))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_seg", [40, 700])
def test_tiles_without_radiating_segments(n_seg, precision, cuda_device):
    """Segments of another layer leave whole tiles without work: the spectrum
    is that of the emitting layer's segments alone (FP64 sums in another
    order; float partial sums within 1e-6 of the peak)."""
    from pyrite_b200 import mc_cxr_spectrum

    E_grid = np.linspace(1000.0, 60000.0, 300)
    seg, rows, tables, n_hat = _scene(n_seg, 25, E_grid, 1.5e5, 77)
    seg["layer"] = np.zeros(n_seg, dtype=np.int32)
    seg["layer"][n_seg // 2: n_seg // 2 + 19] = 1
    kw = dict(tables=tables, n_hat=n_hat, rows=rows, line_quadrature="bin-mean", precision=precision,
              exact_widths=64.0, device=cuda_device)
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, emit_layer=1, **kw)
    on = seg["layer"] == 1
    alone = {k: (v[on] if isinstance(v, np.ndarray) else v) for k, v in seg.items()}
    ref = mc_cxr_spectrum(alone, E_grid, "silicon", None, **kw)
    assert np.max(ref) > 0.0
    assert np.max(np.abs(got - ref)) <= (1e-12 if precision == "fp64" else 1e-6) * np.max(ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_E", [2, 45, 63, 64, 65, 364, 366, 1463, 9301])
def test_far_field_at_the_edges_of_its_chunks(n_E, precision, cuda_device):
    """Two-width windows leave nearly every bin to the far field, whose blocks
    take 64 bins and stage the n_E + 2 pad centres in chunks of at most 512
    (pad = 0.2 n_E + 2: 364 bins fill one chunk, 366 take two)."""
    from pyrite_b200 import mc_cxr_spectrum

    E_grid = np.linspace(1000.0, 60000.0, n_E)
    seg, rows, tables, n_hat = _scene(8, 40, E_grid, 1.5e5, 40 + n_E)
    E, a, w = _lines(seg, rows, tables, n_hat, E_grid)
    assert E.size > 40
    ref = _deposit(E, a, w, oracle.energy_bin_edges(E_grid), 2.0) / seg["Ne"]
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, tables=tables, n_hat=n_hat, rows=rows,
                          line_quadrature="bin-mean", precision=precision, exact_widths=2.0, device=cuda_device)
    if precision == "fp64":
        assert np.max(np.abs(got - ref)) <= 5e-9 * np.max(np.abs(ref))
    else:
        # 320 lines at most: between the single line's 3e-2 and the 2e-3 of many
        assert np.sum(np.abs(got - ref)) <= 3e-2 * np.sum(np.abs(ref))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_seg,n_g", [(16, 119), (17, 48), (100, 121), (33, 145), (900, 60)])
def test_waiting_survivors_over_tiles_rows_and_directions(n_seg, n_g, precision, cuda_device):
    """Pairs that pass the prefilter wait for a whole round over tiles, but not
    over a change of rows or direction: three directions in one call are the
    three single calls, and those the sums over single segments (FP64 sums in
    another order; float partial sums within 1e-6 of the peak)."""
    from pyrite_b200 import mc_cxr_spectrum
    from pyrite_b200.tables import SILICON, diamond_hkls, reflection_rows

    E_grid = np.linspace(1000.0, 60000.0, 200)
    seg, _, tables, n_hat = _scene(n_seg, n_g, E_grid, 1.5e5, n_seg + n_g)
    n_hats = np.stack([n_hat, n_hat + [0.02, 0.0, 0.0], n_hat + [0.0, 0.03, 0.0]])
    n_hats /= np.linalg.norm(n_hats, axis=1, keepdims=True)
    hkl = [h for h in diamond_hkls(9.0) if np.dot(h, (1, 1, 0)) > 0]
    hkl = hkl[:: max(1, len(hkl) // n_g)][:n_g]  # those of the scene
    rows = reflection_rows(SILICON, hkl, n_hats, surface_hkl=(2, 2, 0))
    kw = dict(tables=tables, line_quadrature="bin-mean", precision=precision, exact_widths=8.0, device=cuda_device)
    tol = 1e-12 if precision == "fp64" else 1e-6
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, n_hat=n_hats, rows=rows, **kw)
    for d in range(3):
        one_rows = reflection_rows(SILICON, hkl, n_hats[d:d + 1], surface_hkl=(2, 2, 0))
        one = mc_cxr_spectrum(seg, E_grid, "silicon", None, n_hat=n_hats[d], rows=one_rows, **kw)
        assert np.max(one) > 0.0
        assert np.max(np.abs(got[d] - one)) <= tol * np.max(one)
    if n_seg <= 17:
        parts = 0.0
        for i in range(n_seg):
            s = {k: (v[i:i + 1] if isinstance(v, np.ndarray) else v) for k, v in seg.items()}
            s["elec_id"] = np.zeros(1, dtype=np.int64)
            s["Ne"] = 1
            parts = parts + mc_cxr_spectrum(s, E_grid, "silicon", None, n_hat=n_hats, rows=rows, **kw)
        parts = parts / seg["Ne"]
        assert np.max(np.abs(got - parts)) <= tol * np.max(got)


@pytest.mark.parametrize("quadrature", ["node", "bin-mean"])
@pytest.mark.parametrize("n_mu", [1, 2, 4])
def test_largest_tables_with_several_absorbers(n_mu, quadrature, cuda_device):
    """The FP64 tables of 4,096 energies fit shared memory for one absorber;
    with more they are read from global memory. The attenuation split evenly
    over the absorbers is the same attenuation (1e-12 of the peak)."""
    import dataclasses

    from pyrite_b200 import mc_cxr_spectrum
    from pyrite_b200 import placeholder_data as P
    from pyrite_b200.tables import SILICON, diamond_hkls

    E_grid = np.linspace(1000.0, 60000.0, 150)
    seg, rows, _, n_hat = _scene(40, 30, E_grid, 1.5e5, 8)
    hkl = [h for h in diamond_hkls(9.0) if np.dot(h, (1, 1, 0)) > 0]
    hkl = hkl[:: max(1, len(hkl) // 30)][:30]
    tables = P.line_tables(SILICON, hkl, E_grid, n_tab=4096)
    assert np.asarray(tables.E_tab).size == 4096
    lm = np.atleast_2d(np.asarray(tables.log_mu))
    split = dataclasses.replace(tables, log_mu=np.repeat(lm - np.log(n_mu), n_mu, axis=0))
    kw = dict(n_hat=n_hat, rows=rows, line_quadrature=quadrature, precision="fp64", device=cuda_device)
    ref = mc_cxr_spectrum(seg, E_grid, "silicon", None, tables=tables, **kw)
    got = mc_cxr_spectrum(seg, E_grid, "silicon", None, tables=split, **kw)
    assert np.max(ref) > 0.0
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(ref)
