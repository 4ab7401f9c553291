"""Runs that barely fit the device's memory."""
import ctypes

import numpy as np
import pytest

from glemur_gb300 import Relaxation, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left", [192, 960, 1824])
def test_a_run_that_leaves_no_room_for_the_b_field_uses_the_tile_kernel(left):
    """FP64 stages run as two passes over a B field where that fits.  With the free memory
    at the footprint of such a run and a little below, the run is created and stepped
    all the same, and gives the same grid.  The driver hands memory out in pages of
    2 MB and small buffers from the rest of one (`left` KB of it here)."""
    import torch
    cu = ctypes.CDLL("libcuda.so.1")
    p = configs.random_braid(5, shape=(96, 96, 96), precision=64)
    B0, xb = configs.init_state(p)
    avail = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731

    def steps():
        g = Relaxation(p)
        after = avail()
        try:
            g.upload(xb, B0)
            g.steps_async(3)
            out = g.grid()
            g.refresh()
        finally:
            g.close()
        return out, after

    def small():
        d = ctypes.c_uint64()
        assert cu.cuMemAlloc_v2(ctypes.byref(d), ctypes.c_size_t(32 << 10)) == 0
        return d

    torch.zeros(1, device="cuda")
    steps()                                         # kernels loaded
    torch.cuda.empty_cache()
    before = avail()
    ref, after = steps()
    footprint = before - after
    assert footprint > 4 * 4 * 8 * 96 ** 3          # more than the field
    blocks, page = [], avail()
    try:
        while avail() == page and len(blocks) < 300:
            blocks.append(small())
        blocks += [small() for _ in range((2048 - left) // 32 - 1)]
        for below in range(3):
            torch.cuda.empty_cache()
            hold = torch.empty((avail() - footprint + (below << 21)) >> 21 << 21, dtype=torch.uint8, device="cuda")
            got, _ = steps()
            del hold
            np.testing.assert_array_equal(got, ref)
    finally:
        hold = None
        torch.cuda.empty_cache()
        for d in blocks:
            cu.cuMemFree_v2(d)
