"""Bounce-back and momentum-exchange force link by link: random solids of every density, on the
walls, edges and corners too, so that links to fluid, to halo nodes and across periodic faces
all occur, on both x columns; FP32/FP64 fluid and halo values bit for bit against the oracle,
the force of every step to the rounding of its sum."""
import numpy as np
import pytest

from conftest import fluid_mask_haloed

pytestmark = pytest.mark.gpu

BCS = [(0, 0, 0, 0, 0, 0), (1, 1, 1, 1, 1, 1), (5, 4, 3, 3, 0, 0), (0, 0, 3, 3, 2, 1), (5, 4, 0, 0, 3, 3)]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("share", [0.02, 0.3, 0.9])
@pytest.mark.parametrize("bc", BCS, ids=["".join(map(str, b)) for b in BCS])
def test_random_solids(eup, orc, require_gpu, prec, share, bc):
    l, m, n = 37, 11, 9
    dt = np.float32 if prec == "fp32" else np.float64
    obs = (np.random.default_rng(int(100 * share)).random((n, m, l)) < share).astype(np.int32)
    if bc[0] == 5:
        obs[:, :, -1] = 0  # none on the outflow plane
    a = eup.init_equilibrium(l, m, n, 0.02, 1e-3, 3, dt)
    p = orc.params(l, m, n, bc, svisc=0.1, u_inflow=0.02, u00=0.05)
    keep = fluid_mask_haloed(obs)
    with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.1, u_inflow=0.02, u00=0.05,
                               precision=eup.FP32 if prec == "fp32" else eup.FP64)) as s:
        s.set_obstacles(obs)
        s.upload(a)
        for _ in range(3):
            f = s.forces()
            ref = orc.mem_force(p, a, obs)
            # at most 18 links per voxel, each rounding its product and its sum
            np.testing.assert_allclose(f, ref, rtol=0, atol=1e-12 * max(1.0, float(obs.sum())))
            s.step(1)
            orc.run(p, a, obs, 1)
            got = s.download(dt)
            for q in range(19):
                assert np.array_equal(got[q][keep], a[q][keep]), q + 1


def test_force_reads_agree_across_models(eup, require_gpu):
    """The force of the state reached (from host memory) and the same entry of the history, with
    the partial-bounce-back model switched on and off in between."""
    l, m, n = 24, 12, 8
    obs = np.zeros((n, m, l), np.int32)
    obs[2:5, 4:7, 8:11] = 1
    a = eup.init_equilibrium(l, m, n, 0.05, 1e-3, 3, np.float32)
    with eup.Solver(eup.Config(l, m, n, svisc=0.05, u_inflow=0.05)) as s:
        s.set_obstacles(obs)
        s.upload(a, 5)
        for _ in range(3):
            s.step(1)
            assert np.array_equal(s.forces(), s.force_series(s.itime - 1, 2)[1])
        s.set_obstacles(np.zeros_like(obs))
        assert np.all(s.forces() == 0.0)
        s.set_solid_fraction(np.full((n, m, l), 0.3))
        s.upload(a, 8)
        assert np.all(s.forces() == 0.0)  # a fresh state under this model has no recorded force
        s.step(1)
        f = s.forces()
        assert f[0] != 0.0 and np.array_equal(f, s.force_series(8, 2)[1])
        s.set_solid_fraction(None)
        assert np.array_equal(s.forces(), f)
        s.step(1)
        assert np.all(s.forces() == 0.0) and s.itime == 10
