"""The adjoint of the halo planes (who gets each halo value's adjoint back) for many combinations
of face flags: the gradient of a short partial-bounce-back run against automatic
differentiation of the same steps written in FP64 torch, the halo included."""
import importlib.util
import itertools
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FLAGS = list(itertools.product((0, 1, 5), (0, 1, 4), (0, 1, 3), (0, 1, 3), (0, 1, 2, 3), (0, 1, 3)))
# a periodic y face under a free-slip up face passes on a value of the step before: refused
REFUSED = [bc for bc in FLAGS if bc[4] == 3 and 0 in (bc[2], bc[3])]
TAKEN = [bc for bc in FLAGS if bc not in REFUSED]


@pytest.fixture(scope="module")
def model():
    spec = importlib.util.spec_from_file_location("perf_cases", os.path.join(ROOT, "perf", "cases.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def _config(eup, bc, size):
    return eup.Config(*size, bc=bc, svisc=0.05, u_inflow=0.05, u00=0.1, precision=eup.FP64, cd_uref=0.05,
                      cd_length=2.0, cd_span=float(size[2]))


@pytest.mark.parametrize("size", [(5, 4, 3), (3, 2, 6)], ids=["5x4x3", "3x2x6"])
def test_gradient_for_many_flags(eup, require_gpu, model, size):
    torch = pytest.importorskip("torch")
    l, m, n = size
    steps = 3
    rng = np.random.default_rng(5)
    ns = rng.random((n, m, l)) * 0.8
    start = eup.init_equilibrium(l, m, n, 0.05, 1e-2, 4, np.float64)
    for t in rng.choice(len(TAKEN), 60, replace=False):
        bc = TAKEN[t]
        with eup.Solver(_config(eup, bc, size)) as s:
            s.set_solid_fraction(ns)
            s.upload(start)
            J, grad, _ = s.adjoint(steps, 2, checkpoints=2)
        case = {"lx": l, "ly": m, "lz": n, "bc": "cavity", "svisc": 0.05, "steps": steps}
        x = torch.from_numpy(ns).requires_grad_(True)
        f, total = torch.from_numpy(start), 0.0
        for step in range(steps):
            lat = model._Lattice(case, f.clone(), ns=x)
            lat.bc, lat.u_in, lat.lid = bc, 0.05, 0.1 / 6.0
            lat.halo()
            p = lat.pulled()
            new = lat.collided(p)
            if step >= steps - 2:
                total = total + (2.0 * x * (sum(p[:5]) - sum(p[9:14]))).sum()
            f = lat.f.clone()
            f[:, 1:-1, 1:-1, 1:-1] = torch.stack([(1 - x) * new[q] + x * p[model._OPP[q]] for q in range(19)])
        objective = total / (2 * 0.5 * 0.05 ** 2 * 2.0 * n)
        (want,) = torch.autograd.grad(objective, x)
        assert abs(J - float(objective)) <= 1e-12 * abs(J), bc
        want = want.numpy()
        # FP64 on both sides: rounding of sums of a few hundred terms
        np.testing.assert_allclose(grad, want, rtol=0, atol=1e-11 * np.abs(want).max(), err_msg=str(bc))


def test_older_halo_values_are_refused(eup, require_gpu):
    size = (5, 4, 3)
    for bc in REFUSED[::17]:
        with eup.Solver(_config(eup, bc, size)) as s:
            s.set_solid_fraction(np.full(size[::-1], 0.5))
            s.upload(eup.init_equilibrium(*size, 0.05, 1e-2, 4, np.float64))
            with pytest.raises(eup.EupError) as e:
                s.adjoint(3, 2, checkpoints=2)
            assert e.value.code == 5
