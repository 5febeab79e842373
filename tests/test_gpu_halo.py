"""The halo planes of a step, made by one launch, against the oracle's restatement of the
reference's block sequence: every combination of face flags, in every storage format, down to
one node per side, over steps that read halo values of the step before.  The halo after a step
is the halo of the state it started from, so the expected values follow bit for bit from the
state downloaded before the step."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLAGS = list(itertools.product((0, 1, 5), (0, 1, 4), (0, 1, 3), (0, 1, 3), (0, 1, 2, 3), (0, 1, 3)))


@pytest.mark.parametrize("prec,size", [("fp32", (4, 3, 5)), ("fp64", (3, 4, 2)), ("fp16", (6, 3, 4)), ("bf16", (5, 4, 3)),
                                       ("fp32", (1, 1, 1)), ("fp32", (2, 1, 3))])
def test_halo_of_every_flag_combination(eup, orc, require_gpu, prec, size):
    l, m, n = size
    code = {"fp32": eup.FP32, "fp64": eup.FP64, "fp16": eup.FP16_DEV, "bf16": eup.BF16_DEV}[prec]
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
            for step in range(3):
                ref = s.download(dt)
                orc.bcond_bc(p, ref)
                s.step(1)
                got = s.download(dt)
                bad = halo & (got != ref)
                assert not bad.any(), (bc, step, np.argwhere(bad)[:4])
