"""Energy windows of the mixed bremsstrahlung scorer that take every segment.

Where each electron lies in a window whose fit holds, the list left to the
per-(segment, energy) kernels is empty. What the windows and the list came to
is read back from the workspace, so that the cases are what they say. Bound:
1e-6 of each direction's peak against the FP64 scorer (the fit's 1e-7 and float
sums of about 1e-7).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SI, SIO2 = [("Si", 0.05)], [("Si", 0.0266), ("O", 0.0532)]

HEADER = np.dtype([  # BremNodeHdr
    ("t_max", "u8"), ("t_minc", "u8"), ("n_out", "u8"), ("ok", "u4"), ("faces", "u4"), ("n_cells", "i4"), ("n_win", "i4"),
    ("T", "f8", 4), ("h_min", "f8"), ("z_g", "f8"), ("zb", "f8", 65), ("node", "f8", 512), ("Lm", "f8", 64), ("n_rad", "u8"),
    ("hist", "u4", 256), ("fill", "u4", 257), ("win_of", "i4", 64), ("win_Tc", "f8", 32), ("win_Th", "f8", 32),
    ("win_n", "u4", 32), ("win_fill", "u4", 32), ("win_bad", "u4", 32)], align=True)


def _segments(E, seed, thickness=1.0e7):
    rng = np.random.default_rng(seed)
    n = E.size
    v = rng.normal(size=(n, 3))
    v[:, 2] += 1.0
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    z = thickness * (0.001 + 0.998 * rng.random(n))
    L = 200.0 * (E / 8.0) ** 0.8 * rng.exponential(size=n)
    L = np.maximum(np.minimum(L, 2.0 * np.minimum(z, thickness - z) / np.maximum(np.abs(v[:, 2]), 1e-3)), 1.0)
    return dict(v_hat=v, E_repr_keV=E, L_ang=L, r_mid=np.stack([np.zeros(n), np.zeros(n), z], 1),
                elec_id=np.arange(n) // 100, Ne=(n + 99) // 100, thickness_ang=thickness)


def _directions(kind):
    th = {"one": np.array([0.3]), "detector": np.linspace(0.30, 0.31, 16), "faces": np.linspace(0.30, 0.33, 6)}[kind]
    n = np.stack([np.sin(th), np.zeros_like(th), -np.cos(th)], axis=1)
    if kind == "faces":
        n[::2, 2] *= -1.0
    return n


def _score(seg, E_grid, comp, n_hat, monkeypatch, device):
    """(mixed, FP64, header of the mixed call's workspace)."""
    import torch

    from pyrite_b200 import api

    mu = 2.0e-4 * (1000.0 / E_grid) ** 2.8 + 1.0e-8
    kw = dict(composition=comp, n_hat=n_hat, mu=mu, device=device)
    ref = api.mc_brem_spectrum(seg, E_grid, precision="fp64", **kw)
    work = []
    empty = api._Holder.empty

    def kept(self, shape, dtype):
        t = empty(self, shape, dtype)
        if dtype == torch.uint8:
            work.append(t)
        return t

    monkeypatch.setattr(api._Holder, "empty", kept)
    got = api.mc_brem_spectrum(seg, E_grid, precision="mixed", **kw)
    monkeypatch.undo()
    assert len(work) == 1
    return got, ref, work[0][:HEADER.itemsize].cpu().numpy().view(HEADER)[0]


@pytest.mark.parametrize("kind", ["one", "detector", "faces"])
@pytest.mark.parametrize("comp", [SI, SIO2])
@pytest.mark.parametrize("n,lo,hi,k_hi,n_E", [(20000, 5.0, 30.0, 1990.0, 1024), (20000, 165.0, 2000.0, 60000.0, 2047),
                                              (9001, 5.0, 30.0, 1990.0, 2048)])
def test_no_segment_left_out(n, lo, hi, k_hi, n_E, comp, kind, monkeypatch, cuda_device):
    E = np.exp(np.random.default_rng(n_E).uniform(np.log(lo), np.log(hi), n))
    got, ref, h = _score(_segments(E, n), np.linspace(0.1 * k_hi if k_hi < 1e4 else 1000.0, k_hi, n_E), comp,
                         _directions(kind), monkeypatch, cuda_device)
    n_win = int(h["n_win"])
    assert h["ok"] == 1 and n_win > 4 and not h["win_bad"][:n_win].any() and h["n_out"] == 0
    assert int(h["win_n"][:n_win].sum()) == n == int(h["n_rad"])
    for g, r in zip(np.atleast_2d(got), np.atleast_2d(ref)):
        assert np.max(np.abs(g - r)) <= 1e-6 * np.max(np.abs(r))


@pytest.mark.parametrize("n", [511, 512, 513, 1025])
def test_tiles_of_windows_that_hold(n, monkeypatch, cuda_device):
    """Windows of n segments, one more and one less than a tile among them, and
    empty ones between; none is given up."""
    E = np.concatenate([np.full(n, T) for T in (170.0, 300.0, 700.0, 1000.0, 1100.0, 1500.0, 1900.0)] * (9000 // n // 6 + 1))
    got, ref, h = _score(_segments(E, n), np.linspace(1000.0, 60000.0, 2048), SI, _directions("detector"), monkeypatch,
                         cuda_device)
    n_win = int(h["n_win"])
    assert h["ok"] == 1 and n_win == 7 and not h["win_bad"][:n_win].any() and h["n_out"] == 0
    for g, r in zip(got, ref):
        assert np.max(np.abs(g - r)) <= 1e-6 * np.max(np.abs(r))


def test_windows_given_up(monkeypatch, cuda_device):
    """From 2 MeV up the first quarter of an octave (upper end 1.25 times the
    lower) misses the fit's bound at the lowest photon energies: its segments are
    the list's, in full, and no others'."""
    E = np.exp(np.random.default_rng(5).uniform(np.log(165.0), np.log(1.0e4), 20001))
    got, ref, h = _score(_segments(E, 5), np.linspace(1000.0, 60000.0, 2047), SI, _directions("detector"), monkeypatch,
                         cuda_device)
    n_win = int(h["n_win"])
    bad = h["win_bad"][:n_win] != 0
    lo = h["win_Tc"][:n_win] - h["win_Th"][:n_win]
    assert h["ok"] == 1 and sorted(lo[bad]) == [2048.0, 4096.0, 8192.0]
    assert int(h["n_out"]) == int(h["win_n"][:n_win][bad].sum()) == sum(
        int(((E >= a) & (E < 1.25 * a)).sum()) for a in (2048.0, 4096.0, 8192.0))
    for g, r in zip(got, ref):
        assert np.max(np.abs(g - r)) <= 1e-6 * np.max(np.abs(r))
