"""The table of the halo's edge lines, built from runs of stores, against the one recorded item by
item: every combination of face flags (x-slab exchange faces too), lattices shorter and longer than
the ends that are recorded one by one."""
import ctypes
import itertools

import numpy as np
import pytest

FLAGS = list(itertools.product((0, 1, 5, 6), (0, 1, 4, 6), (0, 1, 3), (0, 1, 3), (0, 1, 2, 3), (0, 1, 3)))
SIZES = [(1, 1, 1), (4, 3, 5), (10, 9, 11), (23, 2, 1), (2, 31, 13), (13, 12, 40), (1, 26, 14), (14, 33, 25)]


def _edges(eup, size, bc, one_by_one):
    f = eup.lib.eup_internal_halo_edges
    f.restype = ctypes.c_int64
    f.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int64]
    flags = (ctypes.c_int * 6)(*bc)
    n = f(*size, flags, one_by_one, None, 0)
    out = np.zeros((n, 5), np.int64)
    assert f(*size, flags, one_by_one, out.ctypes.data, n) == n
    return out


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_runs_equal_the_items(eup, size):
    longer = 0
    for bc in FLAGS:
        want, got = _edges(eup, size, bc, 1), _edges(eup, size, bc, 0)
        assert np.array_equal(want, got), bc
        assert len(np.unique(want[:, 0])) == len(want), bc  # one store to a slot
        longer += len(want)
    assert longer > 0


def test_a_long_lattice_is_cheap(eup):
    """Recorded item by item this table takes minutes; as runs it has a few hundred entries."""
    f = eup.lib.eup_internal_halo_edges
    f.restype = ctypes.c_int64
    f.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_int64]
    flags = (ctypes.c_int * 6)(5, 4, 3, 3, 3, 3)
    assert f(500_000_000, 2, 2, flags, 0, None, 0) > 10**9
