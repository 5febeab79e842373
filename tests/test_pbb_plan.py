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
    lib.pbb_plan_run.argtypes = [ctypes.c_int] * 5 + [ctypes.c_int64] * 2 + [ctypes.c_int] * 2 + [ctypes.c_void_p]

    def run(l, m, n, sbytes=4, variant=4096, sectors=0, force=1, voxels=0):
        out = (ctypes.c_int64 * 6)()
        lib.pbb_plan_run(l, m, n, sbytes, variant, sectors, voxels, force, MOST, out)
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


# Measured on a B200, us per step: lattice, storage bytes, share of sectors and of voxels, two passes, one.
MEASURED = [
    ((96, 64, 64), 4, .077, .01, 27.2, 29.8), ((96, 64, 64), 4, .279, .04, 28.2, 30.5), ((96, 64, 64), 4, .485, .08, 29.0, 30.9),
    ((96, 64, 64), 4, .215, .197, 28.0, 29.6), ((96, 64, 64), 4, .370, .344, 30.2, 29.8),
    ((96, 64, 64), 8, .215, .03, 42.4, 45.5), ((96, 64, 64), 8, .279, .04, 43.4, 45.6), ((96, 64, 64), 8, .485, .08, 47.9, 45.8),
    ((96, 64, 64), 8, .215, .197, 41.0, 45.0), ((96, 64, 64), 8, .301, .248, 42.5, 45.2), ((96, 64, 64), 8, .370, .344, 47.0, 45.3),
    ((96, 64, 64), 2, .149, .02, 42.7, 39.3), ((96, 64, 64), 2, .485, .08, 40.9, 40.3), ((96, 64, 64), 2, .215, .197, 33.0, 38.7),
    ((192, 96, 96), 4, .078, .01, 73.9, 83.5), ((192, 96, 96), 4, .150, .02, 86.3, 84.5), ((192, 96, 96), 4, .280, .04, 103.1, 86.0),
    ((192, 96, 96), 4, .126, .118, 70.7, 82.7), ((192, 96, 96), 4, .167, .148, 77.0, 82.8), ((192, 96, 96), 4, .222, .199, 84.6, 82.9),
    ((192, 96, 96), 8, .078, .01, 119.9, 131.4), ((192, 96, 96), 8, .217, .03, 154.8, 132.2), ((192, 96, 96), 8, .222, .199, 138.2, 131.0),
    ((192, 96, 96), 2, .280, .04, 82.0, 105.5), ((192, 96, 96), 2, .392, .06, 91.7, 106.6), ((192, 96, 96), 2, .488, .08, 97.0, 107.3),
    ((192, 96, 96), 2, .571, .10, 100.7, 108.0), ((192, 96, 96), 2, .729, .15, 116.9, 108.3), ((192, 96, 96), 2, .222, .199, 95.9, 100.8),
    ((192, 96, 96), 2, .261, .248, 108.9, 101.4), ((192, 96, 96), 2, .392, .347, 129.6, 102.1),
    ((384, 192, 192), 4, .078, .01, 521.0, 518.2), ((384, 192, 192), 4, .279, .04, 729.1, 529.0),
    ((384, 192, 192), 4, .157, .149, 474.1, 516.5), ((384, 192, 192), 4, .261, .250, 540.4, 518.3),
    ((384, 192, 192), 2, .391, .06, 513.8, 576.5), ((384, 192, 192), 2, .487, .08, 561.4, 580.7), ((384, 192, 192), 2, .570, .10, 595.2, 582.7),
    ((384, 192, 192), 2, .157, .149, 520.7, 534.6), ((384, 192, 192), 2, .261, .250, 705.4, 538.0),
]


@pytest.mark.parametrize("size,sbytes,sectors,voxels,two,one", MEASURED)
def test_one_pass_only_where_it_is_not_the_slower(plan, size, sbytes, sectors, voxels, two, one):
    l, m, n = size
    groups = (l * m * n + 7) // 8
    chosen = plan(l, m, n, sbytes, 4096, int(sectors * groups), 1, int(voxels * l * m * n))[0]
    assert not chosen or one <= 1.025 * two
    # and two passes only where one is no more than a sixth faster
    assert chosen or two <= 7 / 6 * one
