"""The page that the latest force lands in is a shortcut: where it cannot be registered or mapped,
nothing is held, no error is left behind, and the handle goes on without it."""
import ctypes
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "euplectella_hpc_b200", "csrc")


@pytest.fixture(scope="module")
def page(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("page") / "host_page.so")
    subprocess.run([shutil.which("g++") or "g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "host_page.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def run(fail):
        out = (ctypes.c_int * 7)()
        lib.host_page_run(fail, out)
        return list(out)
    return run


@pytest.mark.parametrize("fail", range(8))
def test_open_and_close(page, fail):
    opened, again, registered, released, cleared, host, dev = page(fail)
    assert opened == again == (fail == 0)
    assert registered == released  # whatever was registered is released once
    assert registered == (1 if fail == 0 else 0 if fail & 1 else 2)
    assert cleared == (0 if fail == 0 else 2)
    assert host == dev == 0


def test_create_does_not_need_the_page():
    src = open(os.path.join(CSRC, "abi.cu")).read()
    create = src[src.index("int eup_create("):src.index("int eup_destroy(")]
    assert not re.search(r"force_page|cudaHostRegister|cudaMallocHost|cudaHostAlloc", create)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp32", "fp16"])
def test_forces_before_and_with_the_page(eup, require_gpu, prec):
    """The force after every step, over the read at which the page is made, with reads left out, a
    new state and new obstacles in between, against the history."""
    l, m, n = 24, 12, 8
    obs = np.zeros((n, m, l), np.int32)
    obs[2:5, 4:7, 8:11] = 1
    a = eup.init_equilibrium(l, m, n, 0.05, 1e-3, 3, np.float32)
    with eup.Solver(eup.Config(l, m, n, svisc=0.05, u_inflow=0.05,
                               precision=eup.FP32 if prec == "fp32" else eup.FP16_DEV)) as s:
        s.set_obstacles(obs)
        s.upload(a)
        f = {0: s.forces()}
        for t in range(1, 81):
            s.step(1)
            if t % 7:
                f[t] = s.forces()
                assert np.array_equal(f[t], s.forces())
        series = s.force_series(0, 81)
        for t, v in f.items():
            assert np.array_equal(v, series[t]), t
        s.upload(a, 7)
        assert np.array_equal(s.forces(), f[0])
        s.step(1)
        assert np.array_equal(s.forces(), f[1]) and np.array_equal(s.forces(), s.force_series(7, 2)[1])
        s.set_obstacles(np.zeros_like(obs))
        assert np.all(s.forces() == 0.0)
