"""The force is the exact sum of its links to the rounding of the result, in every step's history
entry and in the force of a state alone: a body's force is a small difference of large sums, and
the order in which the links are listed must not show."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = np.array([(1, -1, 0), (1, 0, -1), (1, 1, 0), (1, 0, 1), (1, 0, 0), (0, 0, 1), (0, 1, 1), (0, 1, 0), (0, 1, -1),
              (-1, -1, 0), (-1, 0, -1), (-1, 1, 0), (-1, 0, 1), (-1, 0, 0), (0, 0, -1), (0, -1, -1), (0, -1, 0),
              (0, -1, 1)])
OPP = [next(p for p in range(18) if (C[p] == -C[q]).all()) for q in range(18)]
U = 2.0**-53


def _terms(a, obs, bc):
    """-2 c_q a_opp(q)(x + c_q) of every link to a fluid node, across periodic faces too: (3, links)."""
    n, m, l = obs.shape
    x = np.argwhere(obs == 1)[:, ::-1]  # i, j, k from 0
    out = []
    for q in range(18):
        y = x + C[q]
        for ax, (size, hi, lo) in enumerate(((l, 0, 1), (m, 2, 3), (n, 4, 5))):
            if bc[hi] == 0 and bc[lo] == 0:
                y[:, ax] %= size
        y = y[((y >= 0) & (y < (l, m, n))).all(1)]
        y = y[obs[y[:, 2], y[:, 1], y[:, 0]] == 0]
        v = a[OPP[q], y[:, 2] + 1, y[:, 1] + 1, y[:, 0] + 1].astype(np.float64)
        out.append(-2.0 * C[q][:, None] * v[None])
    return np.concatenate(out, 1)


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("size", [(64, 32, 8), (200, 90, 60), (37, 11, 9)], ids=["64x32x8", "200x90x60", "37x11x9"])
def test_force_equals_the_exact_sum(eup, require_gpu, prec, size):
    l, m, n = size
    bc = (5, 4, 3, 3, 0, 0) if l != 37 else (0, 0, 0, 0, 0, 0)
    code, dt = {"fp32": (eup.FP32, np.float32), "fp64": (eup.FP64, np.float64), "fp16": (eup.FP16_DEV, np.float32),
                "bf16": (eup.BF16_DEV, np.float32)}[prec]
    if l != 37:
        obs = eup.geometry_cylinder_z(l, m, n, 0.3 * l, 0.5 * m, 0.15 * m)
    else:
        obs = (np.random.default_rng(5).random((n, m, l)) < 0.3).astype(np.int32)
    states = []
    with eup.Solver(eup.Config(l, m, n, bc=bc, svisc=0.05, u_inflow=0.05, precision=code)) as s:
        s.set_obstacles(obs)
        s.upload(eup.init_equilibrium(l, m, n, 0.05, 1e-3, 3, dt))
        for _ in range(4):
            states.append((s.download(dt), s.forces()))
            s.step(1)
        series = s.force_series(0, 5)
    for t, (a, alone) in enumerate(states):
        terms = _terms(a, obs, bc)
        for c in range(3):
            exact = math.fsum(terms[c])
            # FP32 values add up exactly in FP64, and so do the multiples of 2^-24 in FP64 values; the
            # rest, 2^-25 of a value (twice that in a term) at most, in fewer than 64 roundings to a term
            tol = 2 * U * abs(exact) + 64 * U * 2.0**-24 * terms.shape[1]
            assert abs(alone[c] - exact) <= tol, (t, c)
            assert abs(series[t][c] - exact) <= tol, (t, c)
