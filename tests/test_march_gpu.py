"""The whole-grid march (CPML inside) against the CPU oracle, bit for bit (GPU).

Grids above the size where ``fdtd_step_swap`` takes the march: extents that end
inside a tile, slabs that end inside a vector (npml not a multiple of 16 bytes of
elements) or a tile, one and several chunks along x, lossy media, sources and
plane DFTs in the CPML; and grids on the other side of each of its lines.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from oracle import dft_oracle as D
from oracle.cpu_fdtd import OracleFDTD
from tests.cases import gaussian_sine

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")

CASES = [
    # shape, npml, lossy
    ((220, 170, 64), 4, False),      # one tile along k
    ((137, 175, 104), 5, True),      # lossy, odd npml: two whole-grid launches
    ((150, 186, 92), 6, False),      # straddling in FP32 only
    ((230, 131, 96), 3, True),       # lossy: two whole-grid launches
    ((26, 680, 140), 2, False),      # few planes; slab ends inside a tile
    ((244, 250, 64), 12, False),     # a rim row in the next tile
    ((1000, 47, 60), 1, False),      # one CPML layer
    ((192, 192, 192), 5, True),      # lossy march (FP32); vectors straddle the z slabs' edges
    ((320, 160, 96), 2, False),      # narrow tile in FP32, many planes: several chunks
    ((72, 224, 160), 4, False),      # padded, few planes: interior march and shell kernels
    ((181, 142, 103), 9, True),      # odd rows: two whole-grid launches
    ((46, 445, 120), 16, True),      # mostly CPML, lossy: two whole-grid launches
    ((90, 320, 84), 12, False),      # mostly CPML, lossless: two whole-grid launches
    ((70, 60, 56), 6, False),        # small: two whole-grid launches
]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,npml,lossy", CASES)
def test_march_vs_oracle(shape, npml, lossy, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, CUDAPlaneDFTMonitor

    nx, ny, nz = shape
    rng = np.random.default_rng(17)
    g = CUDAFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    o = OracleFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    eps = rng.uniform(1, 6, shape).astype(np.float32)
    sig = rng.uniform(0, 50, shape) if lossy else None
    for s in (g, o):
        s.set_epsilon(eps, sigma_array=sig)
        s.add_source(lambda f: f.add_source_Jx(nz // 2, gaussian_sine(f.t, 40e9, 30e9),
                                               i0=0, i1=nx, j0=0, j1=ny, rim_taper=True))
        s.add_source(lambda f: f.add_source_Jx(nz - 1, 0.3 * np.cos(2e11 * f.t), i0=1, i1=nx // 2,
                                               j0=ny // 3, j1=ny))
    # waves everywhere from the first step, in the slabs' first and last layers too
    for n in FIELDS:
        v = rng.standard_normal(shape).astype(dtype) * (1.0 if n[0] == "E" else 1.0 / 377.0)
        setattr(g, n, v)
        getattr(o, n)[...] = v
    planes = [("x", 0, ("Ey", "Hz")), ("y", ny - 1, ("Ex", "Hx")), ("z", npml, ("Ez", "Hy"))]
    mg = [CUDAPlaneDFTMonitor(g, ax, i, [30e9, 35e9], c) for ax, i, c in planes]
    mo = [D.OraclePlaneDFTMonitor(o, ax, i, [30e9, 35e9], c) for ax, i, c in planes]
    g.run(11)  # an odd number of steps: the last ψ_H is in the second set
    o.run(11)
    for n in FIELDS:
        assert np.array_equal(getattr(g, n), getattr(o, n)), n
    for (ax, i, comps), a, b in zip(planes, mg, mo):
        for c in comps:
            assert np.array_equal(a.dft(c), b.dft[c]), (ax, i, c)
    state = g.save_state()
    g.run(3)
    g.load_state(state)
    g.run(2)
    o.run(2)
    for n in FIELDS:
        assert np.array_equal(getattr(g, n), getattr(o, n)), n
    assert g._fused_enabled


def test_march_launches_and_wait_timeout():
    """One launch per step; a zero wait budget gives up, reports and recovers."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, _capi as capi

    g = CUDAFDTD((160, 130, 128), 1e-3, npml=8)
    g.run(2)
    g.synchronize()
    n0 = capi.lib().fdtd_launch_count()
    g.run(3)
    assert capi.lib().fdtd_launch_count() - n0 == 3
    flags = ctypes.c_int32(-1)
    capi.run("fdtd_device_status", ctypes.byref(flags), 1)
    try:
        capi.run("fdtd_set_wait_budget", capi.FDTD_WAIT_INTERIOR, 0)
        g.step()
        g.synchronize()
        capi.run("fdtd_device_status", ctypes.byref(flags), 1)
        assert flags.value & 1
    finally:
        capi.run("fdtd_set_wait_budget", capi.FDTD_WAIT_INTERIOR, -1)
    g.reset_state()
    g.run(3)
    capi.run("fdtd_device_status", ctypes.byref(flags), 0)
    assert flags.value == 0
