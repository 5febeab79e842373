"""The halo work items of csrc/halo.h, which one kernel runs in any order, against the oracle's
restatement of the reference's block sequence: every combination of face flags, sizes down to
one node, random item orders, several passes (halo values of one step read by the next)."""
import ctypes
import itertools
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "euplectella_hpc_b200", "csrc")
FLAGS = list(itertools.product((0, 1, 5), (0, 1, 4), (0, 1, 3), (0, 1, 3), (0, 1, 2, 3), (0, 1, 3)))


@pytest.fixture(scope="module")
def items(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("halo") / "halo_items.so")
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "halo_items.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.halo_items_run.argtypes = [ctypes.POINTER(ctypes.c_int)] + [ctypes.c_int] * 3 + [ctypes.c_double] * 2 + [
        ctypes.c_uint, ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("size", [(4, 3, 5), (1, 4, 3), (3, 1, 2), (2, 3, 1), (1, 1, 1), (2, 2, 2)],
                         ids=lambda s: "x".join(map(str, s)))
def test_items_in_any_order_equal_the_block_sequence(items, orc, size):
    l, m, n = size
    rng = np.random.default_rng(7)
    start = rng.random((19, n + 2, m + 2, l + 2))
    for t, bc in enumerate(FLAGS):
        p = orc.params(l, m, n, bc, svisc=0.02, u_inflow=0.05, u00=0.12)
        ref, got = start.copy(), start.copy()
        for step in range(3):
            orc.bcond_bc(p, ref)
            items.halo_items_run((ctypes.c_int * 6)(*bc), l, m, n, 0.05, 0.12 / 6.0, 1000 * t + step, got.ctypes.data)
            assert np.array_equal(ref, got), (bc, step, np.argwhere(ref != got)[:4])
            new = rng.random((19, n, m, l))  # the interior of the next step
            ref[:, 1:-1, 1:-1, 1:-1] = new
            got[:, 1:-1, 1:-1, 1:-1] = new
