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
