"""Room for the march's second ψ_H set: it never takes the headroom (CPU)."""

from __future__ import annotations

import numpy as np
import pytest

from opencl_fdtd_solver_b200 import CUDAFDTD

SHAPE, NPML = (512, 512, 512), 16
TOTAL = 16 * 1024**3


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_second_set_leaves_the_headroom(dtype):
    item = np.dtype(dtype).itemsize
    own = CUDAFDTD.device_footprint_bytes(SHAPE, NPML, dtype)
    extra = 2 * 3 * 2 * NPML * 512 * 512 * item
    # the footprint holds two such sets, ψ_H and ψ_E
    assert own == 15 * 512**3 * item + 2 * extra

    class Dev:
        global_mem_size = TOTAL

    reserve = TOTAL - CUDAFDTD.device_memory_budget_bytes(Dev())

    def fits(budget, free):
        return CUDAFDTD._second_psi_h_fits(SHAPE, NPML, dtype, budget, free, TOTAL)

    assert fits(own + extra, reserve + extra)
    assert not fits(own + extra - 1, reserve + extra)   # the grid's own budget
    assert not fits(own + extra, reserve + extra - 1)   # other users of the device
