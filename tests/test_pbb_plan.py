"""The one-pass partial-bounce-back step stores a partial force per thread block: wherever it is
chosen, its blocks fit the partial sums and cover every node, from one node to rows longer than
the partial sums could ever serve."""
import ctypes
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "euplectella_hpc_b200", "csrc")
MOST = int(re.search(r"kReduceMaxBlocks = (\d+)", open(os.path.join(CSRC, "internal.h")).read()).group(1))


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("pbb") / "pbb_plan.so")
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "pbb_plan.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.pbb_plan_run.argtypes = [ctypes.c_int] * 5 + [ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]

    def run(l, m, n, sbytes=4, variant=4096, sectors=0, force=1):
        out = (ctypes.c_int64 * 6)()
        lib.pbb_plan_run(l, m, n, sbytes, variant, sectors, force, MOST, out)
        return list(out)
    return run


@pytest.mark.parametrize("l", [1, 2, 31, 32, 33, 127, 128, 129, 192, 384, 1024, 4097, 128 * MOST - 1, 128 * MOST,
                               128 * MOST + 1, 1398016, 1398017, 100_000_000, 2**31 - 1])
@pytest.mark.parametrize("rows", [(1, 1), (2, 1), (3, 5), (13, 17), (96, 96), (512, 512)])
def test_one_pass_grid_fits_the_partial_sums(plan, l, rows):
    m, n = rows
    if l * m * n > 2**31 - 1:
        pytest.skip("more nodes than a lattice holds")
    for sbytes in (2, 4, 8):
        for variant in (4096, 4096 | 8192, 4096 | 16384):
            for sectors in (0, (l * m * n + 7) // 8):
                one, blocks, threads, nbx, each, slots = plan(l, m, n, sbytes, variant, sectors)
                if not one:
                    continue
                assert 1 <= blocks <= MOST and blocks == nbx * slots
                assert threads % 32 == 0 and threads <= 128
                assert (nbx - 1) * threads < l <= nbx * threads
                assert (slots - 1) * each < m * n <= slots * each


def test_rows_too_long_take_two_passes(plan):
    for sbytes in (2, 4, 8):
        for variant in (4096, 4096 | 16384):
            for force in (0, 1):
                assert plan(128 * MOST, 1, 1, sbytes, variant, 16 * MOST, force)[0] == 1
                assert plan(128 * MOST + 1, 1, 1, sbytes, variant, 16 * MOST + 1, force)[0] == 0
