"""The second ψ_H set is made only where a step uses it and fits, and the step
without it (``fdtd_step``, ψ_H in place) has the same fields (GPU)."""

from __future__ import annotations

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


@pytest.fixture(scope="module")
def cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import opencl_fdtd_solver_b200 as pkg

    return pkg


@pytest.mark.parametrize("shape,npml,made", [
    ((192, 192, 192), 8, True),     # marches
    ((160, 160, 96), 12, True),     # two whole-grid launches in place of the interior march
    ((181, 160, 155), 8, False),    # odd rows
    ((64, 64, 64), 8, False),       # fits the L2
    ((40, 40, 40), 0, False),       # no CPML
])
def test_second_set_only_where_it_is_used(cuda, shape, npml, made):
    g = cuda.CUDAFDTD(shape, 1e-3, npml=npml)
    assert (g._psi_hn is not None) == made
    assert cuda.CUDAFDTD(shape, 1e-3, npml=npml, fused=False)._psi_hn is None


def test_second_set_asks_for_room_on_a_small_device(cuda, monkeypatch):
    """A grid above an eighth of the budget asks what is free."""
    asked = []
    monkeypatch.setattr(cuda.CUDAFDTD, "_second_psi_h_fits",
                        staticmethod(lambda *a: asked.append(a)))
    assert cuda.CUDAFDTD((192, 192, 192), 1e-3, npml=8)._psi_hn is not None and not asked
    monkeypatch.setattr(cuda.CUDAFDTD, "device_memory_budget_bytes",
                        staticmethod(lambda device: 4 * 10**9))
    assert cuda.CUDAFDTD((192, 192, 192), 1e-3, npml=8)._psi_hn is None
    shape, npml, dtype, budget, free, total = asked[0]
    assert (shape, npml, dtype, budget) == ((192, 192, 192), 8, np.dtype("float32"), 4 * 10**9)
    assert 0 < free <= total


def test_slabs_have_no_second_set(cuda):
    for s in slabs.partition(384, 3, 8):
        g = cuda.CUDAFDTD((384, 192, 192), 1e-3, npml=8, slab=s)
        assert g._psi_hn is None


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape,npml,lossy,schedule", [
    ((192, 160, 120), 8, False, "INTERIOR"),
    ((192, 160, 120), 5, True, "GRID"),
    ((70, 60, 56), 6, False, "GRID"),
])
def test_step_in_place_vs_oracle(cuda, shape, npml, lossy, schedule, dtype, monkeypatch):
    from opencl_fdtd_solver_b200 import _capi as capi

    monkeypatch.setattr(cuda.CUDAFDTD, "_second_psi_h_pays", lambda self: False)
    nx, ny, nz = shape
    rng = np.random.default_rng(23)
    g = cuda.CUDAFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    o = OracleFDTD(shape, 1e-3, npml=npml, dtype=dtype)
    assert g._psi_hn is None
    eps = rng.uniform(1, 6, shape).astype(np.float32)
    sig = rng.uniform(0, 50, shape) if lossy else None
    for s in (g, o):
        s.set_epsilon(eps, sigma_array=sig)
        s.add_source(lambda f: f.add_source_Jx(nz // 2, gaussian_sine(f.t, 40e9, 30e9),
                                               i0=0, i1=nx, j0=0, j1=ny, rim_taper=True))
    for n in FIELDS:
        v = rng.standard_normal(shape).astype(dtype) * (1.0 if n[0] == "E" else 1.0 / 377.0)
        setattr(g, n, v)
        getattr(o, n)[...] = v
    mg = cuda.CUDAPlaneDFTMonitor(g, "z", npml, [30e9, 35e9], ("Ez", "Hy"))
    mo = D.OraclePlaneDFTMonitor(o, "z", npml, [30e9, 35e9], ("Ez", "Hy"))
    _, sched = profile(g, 9)
    o.run(9)
    assert sched[getattr(capi, "FDTD_SCHEDULE_" + schedule)] == 9
    for n in FIELDS:
        assert np.array_equal(getattr(g, n), getattr(o, n)), n
    for c in ("Ez", "Hy"):
        assert np.array_equal(mg.dft(c), mo.dft[c]), c


def test_set_epsilon_gives_the_second_set_up_for_ca(cuda, monkeypatch):
    """Lossy coefficients that do not fit beside the set replace it; the run goes on."""
    shape, npml = (192, 160, 120), 8
    g = cuda.CUDAFDTD(shape, 1e-3, npml=npml)
    o = OracleFDTD(shape, 1e-3, npml=npml)
    rng = np.random.default_rng(29)
    g.Ey = v = rng.standard_normal(shape).astype(np.float32)
    o.Ey[...] = v
    for s in (g, o):
        s.run(3)
    assert g._psi_hn is not None
    empty_like, failed = torch.empty_like, []

    def full_once(t, **kw):
        if not failed:
            failed.append(1)
            raise torch.OutOfMemoryError("device full")
        return empty_like(t, **kw)

    monkeypatch.setattr(torch, "empty_like", full_once)
    eps = rng.uniform(1, 6, shape).astype(np.float32)
    sig = rng.uniform(0, 5, shape)
    for s in (g, o):
        s.set_epsilon(eps, sigma_array=sig)
    assert failed and g._psi_hn is None
    for s in (g, o):
        s.run(4)
    for n in FIELDS:
        assert np.array_equal(getattr(g, n), getattr(o, n)), n
