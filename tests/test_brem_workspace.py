"""The workspace of the mixed bremsstrahlung scorer holds every shorter list.

A program that sizes it once, for its longest list, uses it for all: the size
``pb_brem_work_size`` gives never falls as the list grows, also where the form
changes from energy windows to one window (at 2^22 segments)."""

import ctypes as C

import pytest

from pyrite_b200 import _lib as L


def _size(n_seg, n_E, n_el):
    b = L.PbBremArgs()
    b.precision = L.PB_MIXED
    b.n_dir, b.n_seg, b.n_el, b.n_E = 16, n_seg, n_el, n_E
    nb = C.c_int64(-1)
    assert L.load().pb_brem_work_size(C.byref(b), C.byref(nb)) == 0
    return nb.value


@pytest.mark.parametrize("n_el", [1, 2])
@pytest.mark.parametrize("n_E", [1, 300, 2048, 20000])
def test_size_never_falls_as_the_list_grows(n_E, n_el):
    edge = 1 << 22
    n = [0, 1, 4095, 4096, 4097, 100_000, edge - 1, edge, edge + 1, 5_000_000, 8 * edge - 40000, 8 * edge, 9 * edge,
         100_000_000]
    sizes = [_size(x, n_E, n_el) for x in n]
    assert sizes == sorted(sizes)
    assert sizes[-1] > sizes[n.index(edge)] > sizes[0] > 0
