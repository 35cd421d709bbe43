"""Calls at the edges of what the entry points take: what the caller reads back whole, memory, launches that fail
on the host, several threads, the largest axes, densities that are not numbers."""
import ctypes

import numpy as np
import pytest

from mocassin_xray_gb300 import abi, configs, Context, Setup

pytestmark = pytest.mark.gpu


class _Dirty:
    """Device allocations of these sizes filled with NaN, every second one given back (the others are held
    until the end, so that the driver keeps the memory in use)."""

    def __init__(self, sizes):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.held = []
        for n in sizes:
            p = ctypes.c_uint64()
            assert self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(n)) == 0
            assert self.cu.cuMemsetD8_v2(p, ctypes.c_ubyte(0xff), ctypes.c_size_t(n)) == 0
            self.held.append(p)
        assert self.cu.cuCtxSynchronize() == 0
        for p in self.held[::2]:
            assert self.cu.cuMemFree_v2(p) == 0

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        for p in self.held[1::2]:
            assert self.cu.cuMemFree_v2(p) == 0


def test_arrays_read_whole_start_at_zero(decks, data_dir, tmp_path):
    """The dump row of the grain CDF and the residuals of cells not evaluated are 0, whatever the device
    memory held before the load."""
    s = Setup(configs.dust_shell(tmp_path / "d", n=9, packets=100), data_dir)
    ctx = Context(0)
    with _Dirty([4 * s.info.nbins * (s.n_cells + 1)] * 64):
        ctx.load(s)
    ctx.opacity(1)
    ctx.emission(1)
    pdf = ctx.get(abi.ARR_DUSTPDF)
    assert np.all(pdf[:, 0] == 0.0) and np.all(pdf[-1, 1:] == 1.0)
    ctx.close()
    s = Setup(decks["h_small"], data_dir)
    ctx = Context(0)
    with _Dirty([8 * (s.n_cells + 1)] * 256):
        ctx.load(s)
    assert np.all(ctx.get(abi.ARR_BAL_RESID) == 0.0)
    ctx.close()
