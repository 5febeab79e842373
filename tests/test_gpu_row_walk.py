"""Monitor, region sums and plane means on lattices of a few long rows, in pieces, and of many short
rows, side by side in a warp, at the edges of both: FP64 sums of the same per-node values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 37, 41), (2, 33, 3), (3, 5, 67), (4, 16, 16), (5, 1, 130), (8, 9, 9), (9, 7, 1), (16, 3, 11), (17, 9, 5),
         (4097, 2, 2), (5000, 1, 3), (20011, 1, 1), (1030, 700, 1)]


@pytest.mark.parametrize("size", SIZES, ids=["x".join(map(str, s)) for s in SIZES])
@pytest.mark.parametrize("prec", ["fp32", "fp64", "bf16"])
def test_long_and_short_rows(eup, orc, require_gpu, prec, size):
    l, m, n = size
    dt = np.float64 if prec == "fp64" else np.float32
    code = {"fp32": eup.FP32, "fp64": eup.FP64, "bf16": eup.BF16_DEV}[prec]
    bc = (0, 0, 0, 0, 0, 0)
    rng = np.random.default_rng(l)
    obs = (rng.random((n, m, l)) < 0.2).astype(np.int32)
    region = rng.random((n, m, l)) < 0.5
    a = eup.init_equilibrium(l, m, n, 0.04, 1e-2, 5, dt)
    p = orc.params(l, m, n, bc, svisc=0.05)
    with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.05, precision=code, series_capacity=16)) as s:
        s.set_obstacles(obs)
        s.upload(a)
        a = s.download(dt)  # the values the storage holds
        for axis in range(3):
            # the oracle's plain sums of N terms below 1.1, and of N of them here: N u each, 2 N u / 2 to spare
            np.testing.assert_allclose(s.plane_means(axis), orc.plane_means(p, a, axis), rtol=1e-11, atol=1e-13)
        np.testing.assert_allclose(s.monitor(), orc.monitor(p, a, obs), rtol=1e-11, atol=1e-11 * obs.size / 1000 + 1e-12)
        f = a[:, 1:-1, 1:-1, 1:-1].astype(np.float64)[:, region & (obs == 0)]
        rho = f.sum(0)
        j = [f[:5].sum(0) - f[9:14].sum(0), f[[2, 6, 7, 8, 11]].sum(0) - f[[0, 9, 15, 16, 17]].sum(0),
             f[[3, 5, 6, 12, 17]].sum(0) - f[[1, 8, 10, 14, 15]].sum(0)]
        u = [c / rho for c in j]
        want = [rho.size, rho.sum(), u[0].sum(), u[1].sum(), u[2].sum(), sum((c * c).sum() for c in u)]
        np.testing.assert_allclose(s.region_sums(region), want, rtol=1e-11, atol=1e-11 * obs.size / 1000 + 1e-12)
