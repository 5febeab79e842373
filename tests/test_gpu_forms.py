"""The forms a step can take, all behind the one-launch halo and against one another bit for bit:
one and two nodes per thread, 16- and 8-byte vectors, kernels chained in graphs of one step and of
sixteen or launched one by one, the halo's blocks apart; and the adjoint step forked over two
streams or in one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# rows shorter and longer than a thread block, one plane, no interior rows, rows a vector kernel takes
SHAPES = [(8, 5, 4), (24, 11, 6), (256, 20, 13), (1024, 6, 5), (40, 2, 5), (16, 9, 1), (37, 9, 5)]
ONE_HALO = 4096
FORMS = {"two nodes": ONE_HALO, "one node": ONE_HALO | 8, "16-byte vectors": ONE_HALO | 1, "8-byte vectors": ONE_HALO | 4,
         "plain launches": ONE_HALO | 2, "one node, plain launches": ONE_HALO | 2 | 8, "seven blocks an SM": ONE_HALO | 64,
         "halo blocks apart": 0}


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_forms_of_a_step(eup, require_gpu, monkeypatch, prec, shape):
    l, m, n = shape
    code = {"fp32": eup.FP32, "fp64": eup.FP64, "fp16": eup.FP16_DEV, "bf16": eup.BF16_DEV}[prec]
    obs = eup.geometry_cylinder_z(l, m, n, l / 3, (m + 1) / 2, max(1.0, min(l, m) / 5))
    obs[:, :, -1] = 0  # none on the outflow plane
    a = eup.init_equilibrium(l, m, n, 0.05, 1e-3, 5, np.float64)
    ref = None
    for name, variant in FORMS.items():
        monkeypatch.setenv("EUP_STEP_VARIANT", str(variant))
        with eup.Solver(eup.Config(l, m, n, bc=(5, 4, 3, 3, 0, 0), svisc=0.05, u_inflow=0.05, precision=code)) as s:
            s.set_obstacles(obs)
            s.upload(a)
            s.step(3)
            s.step(35)  # from the other lattice: two graphs of sixteen and three of one
            got = s.download(np.float64), s.force_series(0, 39)
        ref = ref or got
        assert np.array_equal(got[0], ref[0]), name
        assert np.array_equal(got[1], ref[1]), name


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
def test_forms_of_the_adjoint_step(eup, require_gpu, monkeypatch, prec):
    """On the 192x96x96 channel, where the kernels are long enough to overlap; few checkpoints, so
    that recomputed steps and adjoint steps follow one another in every order."""
    from euplectella_hpc_b200 import workloads
    code, dt = {"fp32": (eup.FP32, np.float32), "fp64": (eup.FP64, np.float64), "fp16": (eup.FP16_DEV, np.float32)}[prec]
    wl = workloads.pbb_cylinder_channel(steps=40, avg_steps=20, precision=code)
    a = wl.initial_state(dt)
    out = {}
    for name, variant in {"serial": ONE_HALO | 262144, "forked": ONE_HALO, "forked, plain launches": ONE_HALO | 2,
                          "serial, halo blocks apart": 262144, "forked, one pass": ONE_HALO | 16384,
                          "forked, two passes": ONE_HALO | 8192}.items():
        monkeypatch.setenv("EUP_STEP_VARIANT", str(variant))
        with eup.Solver(wl.cfg) as s:
            s.set_solid_fraction(wl.ns)
            s.upload(a)
            out[name] = s.adjoint(40, 20, checkpoints=4)[:2]
    J0, g0 = out["serial"]
    assert np.isfinite(g0).all() and np.abs(g0).max() > 0
    for name, (J, g) in out.items():
        # one pass and two add the forces of a step in another order: at most 2^21 terms each way
        assert abs(J - J0) <= (2**22 * 2.0**-53 * abs(J0) if "pass" in name else 0.0), name
        assert np.array_equal(g, g0), name
