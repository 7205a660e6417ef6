"""A line outside the window |v| <= sinc_cutoff adds nothing, whatever its record holds.

Lines with amplitudes that are not finite stand next to ordinary ones; where
none of them has the energy inside its window, the spectrum is, to the bit, the
one with their amplitudes at zero (the same lines in the same order, whose
terms of zero leave every sum as it is). Inside their windows it is not finite.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CUTOFF = 30.0


def _records(n, E, phase, seed):
    rng = np.random.default_rng(seed)
    ts = rng.uniform(0.0, 4.0, n)
    te = ts + rng.uniform(0.0, 1.0, n)
    a, b = np.exp(-0.5 * ts), np.exp(-0.5 * te)
    return dict(E_vac=rng.uniform(E[0], E[-1], n), a_vac=rng.uniform(0.05, 2.0, n), phase_slope=rng.uniform(-50, 50, n),
                g_phase=rng.uniform(-phase, phase, n), cs_re=rng.normal(0, 1, n), cs_im=rng.normal(0, 1, n),
                cp_re=rng.normal(0, 1, n), cp_im=rng.normal(0, 1, n), L_esc=rng.uniform(0, 10, n),
                half_dL=rng.uniform(-5, 5, n), apb=a + b, bma=b - a, q=0.25 * (te - ts))


# phases to 1e5 rad take the offset form of the phases, to 1e10 rad the general one
@pytest.mark.parametrize("phase", [1e5, 1e10])
@pytest.mark.parametrize("blend", [False, True])
@pytest.mark.parametrize("n_E", [700, 1024, 1025])
def test_amplitudes_outside_the_window_do_not_count(n_E, blend, phase, cuda_device):
    from pyrite_b200.coherent import coherent_reduce

    E = np.linspace(5000.0, 15000.0, n_E)
    n = 900
    rec = _records(n, E, phase, n_E)
    bad = np.arange(5, n, 90)
    rec["E_vac"][bad] = np.linspace(E[0] - 900.0, E[-1] + 900.0, bad.size)  # the outer ones off the axis
    rec["a_vac"][bad] = 0.2  # windows of 150 eV a side
    zero, poor = (dict(rec, **{k: rec[k].copy() for k in ("cs_re", "cs_im", "cp_re", "cp_im")}) for _ in range(2))
    for k, v in zip(("cs_re", "cs_im", "cp_re", "cp_im"), (np.inf, np.nan, -np.inf, 1e300)):
        zero[k][bad] = 0.0
        poor[k][bad] = v
    kw = dict(sinc_cutoff=CUTOFF, device=cuda_device)
    if blend:
        kw.update(elec_id=np.repeat(np.arange(n // 9), 9), F_row=np.stack([np.linspace(0.1, 0.9, n_E)] * 3))
    rows, w, dom = [300, 300, 300], [1.0, 0.5, 2.0], np.zeros(n_E)
    ref = coherent_reduce(zero, rows, w, E, dom, **kw).cpu().numpy()
    got = coherent_reduce(poor, rows, w, E, dom, **kw).cpu().numpy()
    v = np.abs(0.2 * (E[None, :] - rec["E_vac"][bad][:, None]))
    inside = (v < CUTOFF * (1 - 1e-5)).any(0)
    outside = (v > CUTOFF * (1 + 1e-5)).all(0)
    assert inside.sum() > 50 and outside.sum() > 200 and np.isfinite(ref).all()
    assert np.array_equal(got[outside], ref[outside])
    assert not np.isfinite(got[inside]).any()


def test_amplitudes_below_the_smallest_normal_float(cuda_device):
    """Records whose amplitudes are subnormal floats keep their fields: the
    spectrum is that of amplitudes 2^133 as large times 2^-266. 300 lines round
    some ten times each to multiples of 1.4e-45, which for amplitudes of about
    1e-40 and fields of 1e-39 comes to 2e-5 of the field if every rounding is its
    own; 2e-4 of the spectrum."""
    from pyrite_b200.coherent import coherent_reduce

    E = np.linspace(5000.0, 15000.0, 500)
    rec = _records(300, E, 1e5, 3)
    tiny = dict(rec, **{k: rec[k] * 2.0**-133 for k in ("cs_re", "cs_im", "cp_re", "cp_im")})
    dom = np.zeros(E.size)
    ref = coherent_reduce(rec, [300], [1.0], E, dom, device=cuda_device).cpu().numpy() * 2.0**-266
    got = coherent_reduce(tiny, [300], [1.0], E, dom, device=cuda_device).cpu().numpy()
    assert np.linalg.norm(ref) > 0.0
    assert np.linalg.norm(got / 2.0**-266 - ref / 2.0**-266) <= 2e-4 * np.linalg.norm(ref / 2.0**-266)
