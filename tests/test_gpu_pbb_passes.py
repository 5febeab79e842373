"""The partial-bounce-back step in one pass over every node against the plain stream-collide with
a second pass over the listed voxels: the same populations, the same gradient, and forces that
differ by the order of their sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TWO, ONE = 4096 | 8192, 4096 | 16384
STEPS = 6
SIZES = [
    (3, 3, 3),       # no row away from the boundary planes but one
    (31, 6, 5),      # one block to a row, a lane idle
    (129, 5, 4),     # two blocks to a row, most of the second idle
    (24, 72, 64),    # more rows than partial sums: two rows to a block
    (130, 59, 51),   # two blocks to a row, two rows to a block, the last block with one
]


def _run(eup, monkeypatch, variant, code, size, ns):
    l, m, n = size
    if variant is None:
        monkeypatch.delenv("EUP_STEP_VARIANT", raising=False)
    else:
        monkeypatch.setenv("EUP_STEP_VARIANT", str(variant))
    cfg = eup.Config(lx=l, ly=m, lz=n, precision=code, bc=(5, 4, 3, 3, 0, 0), svisc=0.03, u_inflow=0.05, cd_uref=0.05,
                     cd_length=2.0, cd_span=float(n))
    start = eup.init_equilibrium(l, m, n, 0.05, 1e-2, 3, np.float64)
    with eup.Solver(cfg) as s:
        s.set_solid_fraction(ns)
        s.upload(start)
        s.step(STEPS)
        state, force = s.download(np.float64), s.force_series(1, STEPS)
        J, grad, _ = s.adjoint(5, 3, checkpoints=2)
    return state, np.asarray(force), J, grad


@pytest.mark.parametrize("filled", [0.02, 0.6])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("prec", ["FP32", "FP64", "FP16_DEV", "BF16_DEV"])
def test_one_pass_equals_two(eup, require_gpu, monkeypatch, prec, size, filled):
    code = getattr(eup, prec)
    rng = np.random.default_rng(7)
    shape = size[::-1]
    ns = np.where(rng.random(shape) < filled, rng.random(shape), 0.0)
    ns[shape[0] // 2, shape[1] // 2, shape[2] // 2] = 1.0
    ns[0, 0, 0] = 0.5   # on three boundary planes
    state, force, J, grad = _run(eup, monkeypatch, TWO, code, size, ns)
    assert np.isfinite(state).all() and np.abs(force).max() > 0
    for variant in (ONE, None):
        s1, f1, J1, g1 = _run(eup, monkeypatch, variant, code, size, ns)
        assert np.array_equal(s1, state), variant
        # FP64 sums of at most 4e5 terms in another order, against the largest component
        np.testing.assert_allclose(f1, force, rtol=0, atol=1e-12 * np.abs(force).max())
        assert abs(J1 - J) <= 1e-12 * abs(J)
        assert np.array_equal(g1, grad), variant
