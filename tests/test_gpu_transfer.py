"""State transfers through page-locked host memory.  eup_upload and eup_download move the 19
populations through two staging buffers, the host copy of one population on a copy stream
beside the scatter (gather) kernel of the one before, with events ordering each buffer's
reuse.  Copies from pageable arrays are synchronous, so only page-locked arrays exercise that
overlap: here transfers back to back, exact round trips in FP32/FP64, and the stepped state
equal, bit for bit, to the same run uploaded from a pageable array."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L, M, N = 128, 64, 48


def _pinned(shape, dtype):
    import torch
    t = torch.empty(shape, dtype=torch.float64 if dtype == np.float64 else torch.float32, pin_memory=True)
    return t, t.numpy()


def _ptrs(a):
    return [a[q].ctypes.data for q in range(19)]


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
def test_page_locked_transfers_equal_pageable(eup, require_gpu, prec):
    code, dt = {"fp32": (eup.FP32, np.float32), "fp64": (eup.FP64, np.float64), "fp16": (eup.FP16_DEV, np.float32)}[prec]
    eb = np.dtype(dt).itemsize
    cfg = eup.Config(L, M, N, bc=(eup.OUTFLOW, eup.INFLOW, eup.FREESLIP, eup.FREESLIP, eup.PERIODIC, eup.PERIODIC),
                     svisc=0.01, u_inflow=0.05, precision=code)
    obs = eup.geometry_cylinder_z(L, M, N, 40, 32.5, 8)
    a = eup.init_equilibrium(L, M, N, 0.05, 1e-3, 21, dt)
    b = eup.init_equilibrium(L, M, N, 0.05, 1e-3, 22, dt)
    keep = [_pinned(a.shape, dt) for _ in range(4)]  # tensors stay alive with their arrays
    src_a, src_b, out1, out2 = (k[1] for k in keep)
    src_a[...] = a
    src_b[...] = b
    with eup.Solver(cfg) as s:
        s.set_obstacles(obs)
        s.upload_ptrs(_ptrs(src_b), eb)  # a first state, overwritten at once: buffers reused back to back
        s.upload_ptrs(_ptrs(src_a), eb)
        s.download_ptrs(_ptrs(out1), eb)
        s.download_ptrs(_ptrs(out2), eb)
        if prec != "fp16":  # 16-bit storage rounds the deviations
            assert np.array_equal(out1, a)
        assert np.array_equal(out1, out2)
        s.step(6)
        s.download_ptrs(_ptrs(out1), eb)
        f = s.forces()
    with eup.Solver(cfg) as s:
        s.set_obstacles(obs)
        s.upload(a)
        s.step(6)
        ref = s.download(dt)
        f_ref = s.forces()
    assert np.array_equal(out1, ref)
    assert np.array_equal(f, f_ref)


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16"])
@pytest.mark.parametrize("size", [(3, 2, 1), (40, 24, 18), (150, 80, 60)], ids=["3x2x1", "40x24x18", "150x80x60"])
@pytest.mark.parametrize("elem", [4, 8])
def test_state_in_one_piece_and_in_nineteen(eup, require_gpu, prec, size, elem):
    """Arrays one behind the other and arrays apart, small states (one launch and one copy or
    nineteen) and one above the limit for that: what goes up comes down, halo included."""
    l, m, n = size
    code = {"fp32": eup.FP32, "fp64": eup.FP64, "fp16": eup.FP16_DEV}[prec]
    dt = np.float32 if elem == 4 else np.float64
    a = eup.init_equilibrium(l, m, n, 0.05, 1e-3, 21, dt)
    with eup.Solver(eup.Config(l, m, n, svisc=0.05, u_inflow=0.05, precision=code)) as s:
        s.upload(a)
        whole = s.download(dt)
        if prec == "fp64" or elem == 4 and prec == "fp32":
            assert np.array_equal(whole, a)  # no rounding on the way
        apart = [np.ascontiguousarray(a[q]) for q in range(19)]
        s.upload_ptrs([x.ctypes.data for x in apart], elem)
        back = [np.empty_like(a[0]) for _ in range(19)]
        s.download_ptrs([x.ctypes.data for x in back], elem)
        assert np.array_equal(np.stack(back), whole)
        a[7, 0, 0, 0] = np.nan  # a halo value of population 8
        with pytest.raises(eup.EupError, match="a8"):
            s.upload(a)
