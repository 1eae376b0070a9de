"""Plane DFTs of the two whole-grid launches against the CPU oracle, bit for bit (GPU).

z planes on both sides of the two lines (9,000 cells, 30,000 cells x frequencies) above
which they are accumulated in a pass of their own, in the first, a CPML, an inner and the
last layer, next to x and y planes that stay with the E launch; up to the four planes that
an engine takes.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import dft_oracle as D
from oracle.cpu_fdtd import OracleFDTD
from tests.cases import gaussian_sine
from tests.test_schedule_gpu import profile

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,nfreqs", [
    ((90, 100, 33), (3, 4, 16)),    # 9,000 cells: below, above the second line, well above
    ((89, 101, 45), (4, 5, 17)),    # 8,989 cells: all with the E launch
    ((100, 100, 35), (3, 2, 1)),    # 30,000 products, below, below
])
def test_z_planes_vs_oracle(shape, nfreqs, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, CUDAPlaneDFTMonitor, _capi as capi

    npml = 5
    nx, ny, nz = shape
    rng = np.random.default_rng(41)
    g = CUDAFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    o = OracleFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    eps = rng.uniform(1, 6, shape).astype(np.float32)
    for s in (g, o):
        s.set_epsilon(eps)
        s.add_source(lambda f: f.add_source_Jx(nz // 2, gaussian_sine(f.t, 40e9, 30e9),
                                               i0=0, i1=nx, j0=0, j1=ny, rim_taper=True))
    for n in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"):
        v = rng.standard_normal(shape).astype(dtype) * (1.0 if n[0] == "E" else 1.0 / 377.0)
        setattr(g, n, v)
        getattr(o, n)[...] = v
    fs = [[25e9 + 1e9 * q for q in range(n)] for n in nfreqs]
    planes = [("z", nz // 2, fs[0], ("Ex", "Hy")), ("z", 0, fs[1], ("Ez", "Hx")),
              ("z", nz - 1, fs[2], ("Ey", "Hz")), ("x", npml, fs[2], ("Ez", "Hy"))]
    mg = [CUDAPlaneDFTMonitor(g, *p) for p in planes]
    mo = [D.OraclePlaneDFTMonitor(o, *p) for p in planes]
    _, sched = profile(g, 7)
    o.run(7)
    assert sched[capi.FDTD_SCHEDULE_GRID] == 7
    for (ax, i, _, comps), a, b in zip(planes, mg, mo):
        for c in comps:
            assert np.array_equal(a.dft(c), b.dft[c]), (ax, i, c)
