"""The halo planes on lattices long enough that the table of the edge lines comes from runs of
stores, against the oracle's block sequence, for every combination of face flags."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLAGS = list(itertools.product((0, 1, 5), (0, 1, 4), (0, 1, 3), (0, 1, 3), (0, 1, 2, 3), (0, 1, 3)))


@pytest.mark.parametrize("prec,size", [("fp32", (14, 12, 11)), ("fp16", (10, 25, 13)), ("fp64", (21, 2, 12))],
                         ids=["fp32", "fp16", "fp64"])
def test_halo_with_runs_of_edge_stores(eup, orc, require_gpu, prec, size):
    l, m, n = size
    code = {"fp32": eup.FP32, "fp64": eup.FP64, "fp16": eup.FP16_DEV}[prec]
    dt = np.float64 if prec == "fp64" else np.float32
    start = eup.init_equilibrium(l, m, n, 0.05, 1e-2, 11, dt)
    start += np.random.default_rng(3).uniform(0, 1e-3, start.shape).astype(dt)  # every value its own
    halo = np.ones(start.shape, bool)
    halo[:, 1:-1, 1:-1, 1:-1] = False
    for bc in FLAGS:
        p = orc.params(l, m, n, bc, svisc=0.05, u_inflow=0.05, u00=0.1)
        with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.05, u_inflow=0.05, u00=0.1, precision=code,
                                   series_capacity=8)) as s:
            s.upload(start)
            for step in range(2):
                ref = s.download(dt)
                orc.bcond_bc(p, ref)
                s.step(1)
                bad = halo & (s.download(dt) != ref)
                assert not bad.any(), (bc, step, np.argwhere(bad)[:4])
