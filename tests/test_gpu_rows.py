"""The stream-collide over row lengths at the edges of its warps and blocks, with rows on the
y/z boundary planes and both directions of the walk over the planes (successive steps turn):
FP32/FP64 bit for bit against the oracle; 16-bit storage, one and two nodes per thread, alike."""
import numpy as np
import pytest

from conftest import fluid_mask_haloed

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 31, 32, 33, 63, 64, 65, 127, 128, 129, 130, 191, 255, 256, 257, 258, 385]


@pytest.mark.parametrize("l", LENGTHS)
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("yz", [(5, 4), (1, 3), (3, 1)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_row_lengths(eup, orc, require_gpu, l, prec, yz):
    m, n = yz
    dt = np.float32 if prec == "fp32" else np.float64
    bc = (0, 0, 3, 3, 0, 0) if l < 4 else (5, 4, 3, 3, 3, 3)
    obs = np.zeros((n, m, l), np.int32)
    if l > 8:
        obs[n // 2, m // 2, l // 3:l // 3 + 2] = 1
    a = eup.init_equilibrium(l, m, n, 0.03, 1e-2, l, dt)
    p = orc.params(l, m, n, bc, svisc=0.05, u0=0.02, u_inflow=0.03)
    with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.05, u0=0.02, u_inflow=0.03,
                               precision=eup.FP32 if prec == "fp32" else eup.FP64)) as s:
        s.set_obstacles(obs)
        s.upload(a)
        s.step(5)
        got = s.download(dt)
    orc.run(p, a, obs, 5)
    keep = fluid_mask_haloed(obs)
    for q in range(19):
        assert np.array_equal(got[q][keep], a[q][keep]), q + 1


@pytest.mark.parametrize("l", [2, 30, 64, 128, 130, 256, 258])
@pytest.mark.parametrize("prec", ["fp16", "bf16"])
def test_one_and_two_nodes_per_thread(eup, require_gpu, monkeypatch, l, prec):
    m, n = 5, 4
    code = eup.FP16_DEV if prec == "fp16" else eup.BF16_DEV
    a = eup.init_equilibrium(l, m, n, 0.03, 1e-2, l, np.float32)
    res = []
    for var in ("4096", "4104", "4098"):  # two nodes, one node, two without graphs
        monkeypatch.setenv("EUP_STEP_VARIANT", var)
        with eup.Solver(eup.Config(l, m, n, bc=(5, 4, 3, 3, 1, 3), svisc=0.05, u_inflow=0.03, precision=code)) as s:
            s.upload(a)
            s.step(40)  # a run long enough for the 16-step graphs, and a remainder
            res.append(s.download(np.float64))
    assert np.array_equal(res[0], res[1]) and np.array_equal(res[0], res[2])
