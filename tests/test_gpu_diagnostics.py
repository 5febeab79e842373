"""Plane means, monitor and region sums at the edges of their row and column walks: rows of one
node, one short of and one over a warp, over several blocks; one row, one plane.  Against the
oracle's sums over the same per-node values (FP64 sums in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (31, 3, 5), (32, 9, 1), (33, 1, 7), (129, 5, 67), (64, 70, 3), (257, 2, 2)]


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
def test_sums_over_rows_and_columns(eup, orc, require_gpu, prec, size):
    l, m, n = size
    dt = np.float64 if prec == "fp64" else np.float32
    code = {"fp32": eup.FP32, "fp64": eup.FP64, "fp16": eup.FP16_DEV}[prec]
    bc = (0, 0, 0, 0, 0, 0)
    rng = np.random.default_rng(l)
    obs = (rng.random((n, m, l)) < 0.2).astype(np.int32)
    region = rng.random((n, m, l)) < 0.5
    a = eup.init_equilibrium(l, m, n, 0.04, 1e-2, 5, dt)
    p = orc.params(l, m, n, bc, svisc=0.05)
    with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.05, precision=code)) as s:
        s.set_obstacles(obs)
        s.upload(a)
        a = s.download(dt)  # the values the storage holds
        for axis in range(3):
            np.testing.assert_allclose(s.plane_means(axis), orc.plane_means(p, a, axis), rtol=1e-12, atol=1e-14)
        np.testing.assert_allclose(s.monitor(), orc.monitor(p, a, obs), rtol=1e-12, atol=1e-12)
        f = a[:, 1:-1, 1:-1, 1:-1].astype(np.float64)[:, region & (obs == 0)]
        rho = f.sum(0)
        j = [f[:5].sum(0) - f[9:14].sum(0), f[[2, 6, 7, 8, 11]].sum(0) - f[[0, 9, 15, 16, 17]].sum(0),
             f[[3, 5, 6, 12, 17]].sum(0) - f[[1, 8, 10, 14, 15]].sum(0)]
        u = [c / rho for c in j]
        want = [rho.size, rho.sum(), u[0].sum(), u[1].sum(), u[2].sum(), sum((c * c).sum() for c in u)]
        np.testing.assert_allclose(s.region_sums(region), want, rtol=1e-11, atol=1e-12)
