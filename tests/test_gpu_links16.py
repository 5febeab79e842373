"""Bounce-back in 16-bit storage, link by link: a solid voxel takes the word of the fluid node across
as it is, and a halo value (FP32) as storage rounds it, on walls, edges and both x columns; the x
halo of a periodic lattice then carries the same values.  Random solids of every density."""
import numpy as np
import pytest

from test_gpu_force_sum import C, OPP

pytestmark = pytest.mark.gpu

BCS = [(0, 0, 0, 0, 0, 0), (1, 1, 1, 1, 1, 1), (5, 4, 3, 3, 0, 0), (0, 0, 3, 3, 2, 1), (5, 4, 0, 0, 3, 3)]
W = np.array([1 / 18 if np.abs(c).sum() == 1 else 1 / 36 for c in C]).astype(np.float32)
SCALE = np.float32(4096)


def _stored(f, q, prec):
    """The population q that a halo value f comes back as from storage."""
    import torch
    d = torch.from_numpy((f - W[q]) * SCALE)
    d = d.to(torch.float16 if prec == "fp16" else torch.bfloat16).to(torch.float32).numpy()
    return W[q] + d * (np.float32(1) / SCALE)


@pytest.mark.parametrize("prec", ["fp16", "bf16"])
@pytest.mark.parametrize("share", [0.02, 0.3, 0.9])
@pytest.mark.parametrize("bc", BCS, ids=["".join(map(str, b)) for b in BCS])
def test_random_solids(eup, require_gpu, prec, share, bc):
    l, m, n = 37, 11, 9
    obs = (np.random.default_rng(int(100 * share)).random((n, m, l)) < share).astype(np.int32)
    if bc[0] == 5:
        obs[:, :, -1] = 0  # none on the outflow plane
    a = eup.init_equilibrium(l, m, n, 0.02, 1e-3, 3, np.float32)
    inside = np.zeros((n + 2, m + 2, l + 2), bool)
    inside[1:-1, 1:-1, 1:-1] = True
    solid = np.zeros_like(inside)
    solid[1:-1, 1:-1, 1:-1] = obs == 1
    x = np.argwhere(solid)  # k, j, i
    with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.1, u_inflow=0.02, u00=0.05,
                               precision=eup.FP16_DEV if prec == "fp16" else eup.BF16_DEV)) as s:
        s.set_obstacles(obs)
        s.upload(a)
        for _ in range(3):
            before = s.download(np.float32)
            s.step_boundaries()
            after = s.download(np.float32)
            want = before.copy()
            for q in range(18):
                y = x + C[q][::-1]
                at, to = tuple(y.T), tuple(x.T)
                across = before[OPP[q]][at]
                fluid, halo = inside[at] & ~solid[at], ~inside[at]
                v = before[q][to]
                v = np.where(fluid, across, np.where(halo, _stored(across, q, prec), v))
                want[q][to] = v
            assert np.array_equal(after[:, inside], want[:, inside])
            if bc[0] == 0:  # the x halo comes from the x-face copy, which has to follow
                assert np.array_equal(after[9:14, 1:-1, 1:-1, l + 1], after[9:14, 1:-1, 1:-1, 1])
                assert np.array_equal(after[0:5, 1:-1, 1:-1, 0], after[0:5, 1:-1, 1:-1, l])
            s.step_stream()
