"""Forms of the step that need a particular schedule, which each case asserts, against
the CPU oracle bit for bit (GPU): the march's narrow tile in both precisions, vectors
that straddle a z slab's edge in every tile, few planes, the lossy march with whole
vectors; the interior march over partial tiles and several chunks along x; x-slabs with
ghost planes as two whole-grid launches.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from opencl_fdtd_solver_b200 import slabs
from oracle import dft_oracle as D
from oracle.cpu_fdtd import OracleFDTD
from tests.cases import gaussian_sine
from tests.test_schedule_gpu import profile

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")

CASES = [
    # shape, npml, lossy, schedule in FP32 and FP64
    ((320, 160, 96), 1, False, "MARCH", "MARCH"),      # narrow in FP32, slab edges in vectors
    ((384, 128, 48), 4, False, "GRID", "MARCH"),       # narrow in FP64
    ((384, 128, 48), 5, False, "GRID", "MARCH"),       # the same, slab edges in vectors
    ((230, 192, 112), 7, False, "MARCH", "MARCH"),     # wide, slab edges in vectors
    ((26, 640, 192), 2, False, "MARCH", "MARCH"),      # few planes, slabs end inside a tile
    ((30, 512, 192), 5, False, "MARCH", "MARCH"),
    ((192, 192, 192), 8, True, "MARCH", "GRID"),       # lossy, whole vectors
    ((240, 20, 20), 3, False, "INTERIOR", "INTERIOR"),  # several chunks along x
    ((36, 65, 40), 6, True, "INTERIOR", "INTERIOR"),   # partial tiles in j and k
]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,npml,lossy,f32,f64", CASES)
def test_schedule_vs_oracle(shape, npml, lossy, f32, f64, dtype, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, CUDAPlaneDFTMonitor, _capi as capi

    monkeypatch.delenv("FDTD_B200_FACE_E", raising=False)
    nx, ny, nz = shape
    rng = np.random.default_rng(31)
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
    planes = [("x", nx - 1, ("Ey", "Hz")), ("y", npml, ("Ex", "Hx")), ("z", nz - npml, ("Ez", "Hy"))]
    mg = [CUDAPlaneDFTMonitor(g, ax, i, [30e9, 35e9], c) for ax, i, c in planes]
    mo = [D.OraclePlaneDFTMonitor(o, ax, i, [30e9, 35e9], c) for ax, i, c in planes]
    _, sched = profile(g, 9)
    o.run(9)
    assert sched[getattr(capi, "FDTD_SCHEDULE_" + (f32 if dtype == np.float32 else f64))] == 9
    for n in FIELDS:
        assert np.array_equal(getattr(g, n), getattr(o, n)), n
    for (ax, i, comps), a, b in zip(planes, mg, mo):
        for c in comps:
            assert np.array_equal(a.dft(c), b.dft[c]), (ax, i, c)


@pytest.mark.parametrize("lossy", [False, True])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_slabs_as_whole_grid_launches(dtype, lossy):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, _capi as capi

    shape, npml, steps = (96, 52, 56), 5, 25
    nx, ny, nz = shape
    rng = np.random.default_rng(37)
    eps = rng.uniform(1, 6, shape).astype(np.float32)
    sig = rng.uniform(0, 5, shape) if lossy else None
    start = {n: rng.standard_normal(shape).astype(dtype) * (1.0 if n[0] == "E" else 1.0 / 377.0)
             for n in FIELDS}
    plan = slabs.partition(nx, 2, npml)
    o = OracleFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    engines = [CUDAFDTD(shape, 1e-3, npml=npml, dtype=dtype, slab=s) for s in plan]
    for s in (o, *engines):
        s.set_epsilon(eps, sigma_array=sig)
        s.add_source(lambda f: f.add_source_Jx(nz // 4, gaussian_sine(f.t, 60e9, 40e9), i0=4,
                                               i1=nx - 5, j0=5, j1=ny - 6, rim_taper=True))
    for n in FIELDS:
        getattr(o, n)[...] = start[n]
        for g, s in zip(engines, plan):
            setattr(g, n, start[n][s.l0:s.l0 + s.nx_local])
    out = ctypes.c_int32()
    for g in engines:
        for swap in (0, 1):
            capi.run("fdtd_step_schedule", g._grid, swap, ctypes.byref(out))
            assert out.value == capi.FDTD_SCHEDULE_GRID
    views = lambda r: (lambda n, i: engines[r].field_tensor(n)[i])  # noqa: E731
    for _ in range(steps):
        for g in engines:
            g.step()
        slabs.local_exchange(plan, views)
    o.run(steps)
    for n in FIELDS:
        got = np.concatenate([g.field_tensor(n)[s.owned].cpu().numpy()
                              for g, s in zip(engines, plan)])
        assert np.array_equal(got, getattr(o, n)), n
