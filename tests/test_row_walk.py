"""The walks of the diagnostics over all nodes: every node once, whatever the shape, and no shape
leaves the device to a few warps or a warp to a few lanes (a warp per row did, on lattices of a few
long rows or of many short ones)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "euplectella_hpc_b200", "csrc")
LENGTHS = [1, 2, 3, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33, 64, 65, 127, 128, 129, 200, 1000, 4096, 4097, 70001]
ROWS = [(1, 1), (1, 7), (3, 5), (40, 33), (97, 111)]


@pytest.fixture(scope="module")
def walks(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("walk") / "row_walk.so")
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "row_walk.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.row_walk_run.argtypes = [ctypes.c_int, ctypes.c_int64, ctypes.c_void_p]
    lib.plane_split_run.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p]
    return lib


def _row_walk(lib, l, rows):
    out = (ctypes.c_int64 * 6)()
    lib.row_walk_run(l, rows, out)
    return list(out)[1:]


@pytest.mark.parametrize("l", LENGTHS)
@pytest.mark.parametrize("rows", ROWS)
def test_every_node_once(walks, l, rows):
    rows = rows[0] * rows[1]
    lg, span, pieces, r_, units = _row_walk(walks, l, rows)
    seen = np.zeros((rows, l), np.int32)
    side = 32 >> lg
    for u in range(units):
        group, piece = divmod(u, pieces)
        first = piece * span
        end = min(l - first, span)
        assert end > 0
        for sub in range(min(side, rows - group * side)):
            x = np.arange(end) if lg == 5 else np.arange(min(end, 1 << lg))
            assert x.size == end  # a row side by side with others is one pass
            seen[group * side + sub, first + x] += 1
    assert np.all(seen == 1)


@pytest.mark.parametrize("shape", [(65536, 2, 2), (4096, 8, 8), (16384, 4, 64), (1024, 16, 16), (2, 512, 512), (1, 512, 512),
                                   (4, 256, 256), (8, 256, 256), (16, 128, 128), (64, 32, 8), (256, 128, 64),
                                   (768, 384, 384), (2**31 - 1, 1, 1), (1, 46340, 46340)])
def test_warps_and_lanes_in_use(walks, shape):
    l, m, n = shape
    lg, span, pieces, rows, units = _row_walk(walks, l, m * n)
    assert (pieces - 1) * span < l <= pieces * span
    tiles = -(-l // 32) if lg == 5 else 1
    groups = -(-(m * n) // (32 >> lg))
    # a full wave of warps where there are that many passes of a warp to deal, and half of the
    # lanes in use but for the last pass of a row
    assert units >= min(148 * 32, groups * tiles) // 2
    assert lg == 5 or l > (1 << lg) // 2


@pytest.mark.parametrize("l", LENGTHS)
@pytest.mark.parametrize("mn", [(1, 1), (1, 7), (3, 5), (512, 1), (40, 33)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_planes_every_node_once_and_scratch_bounded(walks, l, mn, axis):
    m, n = mn
    out = (ctypes.c_int64 * 10)()
    walks.plane_split_run(l, m, n, axis, out)
    tx, ty, planes, rows, shares, xblocks, plane, row, blocks, scratch = list(out)
    assert tx * ty == 128 and shares >= 1 and xblocks >= 1 and blocks == planes * shares * xblocks
    x = [i for xb in range(xblocks) for th in range(tx)
         for i in range(xb * tx + th, l, l if axis == 0 else xblocks * tx)]
    assert sorted(x) == list(range(l))
    t = [i for s in range(shares) for th in range(ty) for i in range(s * ty + th, rows, shares * ty)]
    assert sorted(t) == list(range(rows))
    seen = sorted(p * plane + i * row for p in range(planes) for i in range(rows))
    assert seen == list(range(m * n))
    # the partial sums fit beside the result in the staging buffer a state transfer needs
    assert scratch <= 4 * l * max(ty, rows / 8) if axis == 0 else scratch <= 4 * max(blocks, 1)
