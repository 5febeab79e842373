"""Nineteen host arrays that adjoin are not always one allocation: each may be page-locked by
itself, or only some of them may be.  CUDA refuses one copy over several such ranges, and the
transfers take the arrays one by one then."""
import mmap

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = M = N = 14  # 16^3 values: an array is whole pages in both precisions


class _Arrays:
    """19 adjoining arrays in page-aligned memory, those of `ranges` (first, count) registered."""

    def __init__(self, dt, ranges):
        import torch
        self.rt = torch.cuda.cudart()
        self.bytes = 16**3 * np.dtype(dt).itemsize
        assert self.bytes % mmap.PAGESIZE == 0
        self.mem = mmap.mmap(-1, 19 * self.bytes)
        self.a = np.frombuffer(self.mem, dtype=dt).reshape(19, N + 2, M + 2, L + 2)
        self.registered = []
        for first, count in ranges:
            at = self.a.ctypes.data + first * self.bytes
            assert int(self.rt.cudaHostRegister(at, count * self.bytes, 0)) == 0
            self.registered.append(at)

    def ptrs(self):
        return [self.a.ctypes.data + q * self.bytes for q in range(19)]

    def close(self):
        for at in self.registered:
            self.rt.cudaHostUnregister(at)


RANGES = {
    "each by itself": [(q, 1) for q in range(19)],
    "one range": [(0, 19)],
    "two ranges": [(0, 7), (7, 12)],
    "first ten": [(0, 10)],
    "last ten": [(9, 10)],
    "every other": [(q, 1) for q in range(0, 19, 2)],
    "none": [],
}


@pytest.mark.parametrize("ranges", list(RANGES))
@pytest.mark.parametrize("dt", [np.float32, np.float64], ids=["f4", "f8"])
def test_adjoining_arrays_of_several_allocations(eup, require_gpu, ranges, dt):
    start = eup.init_equilibrium(L, M, N, 0.05, 1e-3, 21, dt)
    eb = np.dtype(dt).itemsize
    up, down = _Arrays(dt, RANGES[ranges]), _Arrays(dt, RANGES[ranges])
    try:
        up.a[...] = start
        prec = eup.FP32 if dt == np.float32 else eup.FP64
        with eup.Solver(eup.Config(L, M, N, svisc=0.05, u_inflow=0.05, precision=prec)) as s:
            s.upload_ptrs(up.ptrs(), eb)
            s.download_ptrs(down.ptrs(), eb)
            s.step(2)  # no error is left behind for the next launch to find
            s.synchronize()
        assert np.array_equal(down.a, start)
    finally:
        up.close()
        down.close()


def test_separate_page_locked_arrays(eup, require_gpu):
    import torch
    start = eup.init_equilibrium(L, M, N, 0.05, 1e-3, 21, np.float32)
    up = [torch.from_numpy(start[q].copy()).pin_memory() for q in range(19)]
    down = [torch.empty_like(x).pin_memory() for x in up]
    with eup.Solver(eup.Config(L, M, N, svisc=0.05, u_inflow=0.05)) as s:
        s.upload_ptrs([x.data_ptr() for x in up], 4)
        s.download_ptrs([x.data_ptr() for x in down], 4)
    assert np.array_equal(np.stack([x.numpy() for x in down]), start)


@pytest.mark.parametrize("size", [(70, 50, 24), (96, 48, 40)], ids=["7MB", "16MB"])
@pytest.mark.parametrize("locked", [True, False], ids=["page-locked", "pageable"])
def test_arrays_apart(eup, require_gpu, size, locked):
    """Both sides of the size from which page-locked arrays apart cross population by population."""
    import torch
    l, m, n = size
    start = eup.init_equilibrium(l, m, n, 0.05, 1e-3, 21, np.float32)
    count = start[0].size

    def arrays():
        t = [torch.zeros(count + 4096, pin_memory=locked) for _ in range(19)]  # gaps between them
        return t, [x.numpy()[:count].reshape(start[0].shape) for x in t]

    (keep_up, up), (keep_down, down) = arrays(), arrays()
    for q in range(19):
        up[q][...] = start[q]
    with eup.Solver(eup.Config(l, m, n, svisc=0.05, u_inflow=0.05)) as s:
        s.upload_ptrs([x.ctypes.data for x in up], 4)
        s.download_ptrs([x.ctypes.data for x in down], 4)
    assert np.array_equal(np.stack(down), start)
