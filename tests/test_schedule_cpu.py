"""Which schedule a grid's fused step takes (``fdtd_step_schedule``, host only)."""

from __future__ import annotations

import ctypes

import pytest

from opencl_fdtd_solver_b200 import _capi as capi

MARCH, GRID, INTERIOR, FACES = (capi.FDTD_SCHEDULE_MARCH, capi.FDTD_SCHEDULE_GRID,
                                capi.FDTD_SCHEDULE_INTERIOR, capi.FDTD_SCHEDULE_FACES)


def schedule(shape, npml, f64, lossy, swap, slab=None):
    g = capi.Grid(nx=shape[0], ny=shape[1], nz=shape[2], npml=npml,
                  dtype=capi.FDTD_F64 if f64 else capi.FDTD_F32, lossy=lossy)
    if slab is not None:
        g.x_slab, g.pml_x_lo, g.pml_x_hi, g.ghost_lo, g.ghost_hi = 1, *slab
    out = ctypes.c_int32(-1)
    capi.run("fdtd_step_schedule", g, swap, ctypes.byref(out))
    return out.value


@pytest.mark.parametrize("shape,npml,f64,lossy,swapped,in_place", [
    ((512, 512, 512), 16, 0, 0, MARCH, FACES),          # a large shell
    ((256, 256, 256), 12, 0, 0, MARCH, INTERIOR),
    ((192, 192, 192), 5, 0, 1, MARCH, GRID),
    ((192, 192, 192), 5, 1, 1, GRID, GRID),             # no lossy march in FP64
    ((160, 160, 96), 12, 0, 0, GRID, INTERIOR),         # narrow tile
    ((72, 224, 328), 4, 0, 0, INTERIOR, INTERIOR),      # padded, few planes
    ((64, 64, 64), 8, 0, 0, GRID, GRID),                # fits the L2
    ((144, 144, 144), 8, 0, 0, INTERIOR, INTERIOR),     # whole tiles in the interior
    ((118, 448, 152), 16, 0, 0, GRID, INTERIOR),
    ((40, 36, 48), 6, 0, 0, INTERIOR, INTERIOR),
    ((37, 41, 53), 6, 0, 1, GRID, GRID),                # odd rows
    ((181, 230, 155), 10, 0, 0, GRID, GRID),
    ((40, 40, 40), 0, 1, 0, GRID, GRID),                # no CPML
])
def test_schedule_of_a_grid(shape, npml, f64, lossy, swapped, in_place, monkeypatch):
    monkeypatch.delenv("FDTD_B200_FACE_E", raising=False)
    assert schedule(shape, npml, f64, lossy, 1) == swapped
    assert schedule(shape, npml, f64, lossy, 0) == in_place


def test_slabs_never_march_and_bad_calls_are_refused(monkeypatch):
    monkeypatch.delenv("FDTD_B200_FACE_E", raising=False)
    for slab in ((8, 0, 0, 1), (0, 0, 1, 1), (0, 8, 1, 0)):
        for lossy in (0, 1):
            assert schedule((129, 256, 256), 8, 0, lossy, 1, slab) == INTERIOR
            assert schedule((64, 64, 64), 8, 0, lossy, 1, slab) == GRID
    assert capi.call("fdtd_step_schedule", capi.Grid(nx=8, ny=8, nz=8), 0,
                     None) == capi.FDTD_ERR_INVALID
    with pytest.raises(ValueError):
        schedule((0, 8, 8), 1, 0, 0, 0)


def test_forced_face_marches(monkeypatch):
    monkeypatch.setenv("FDTD_B200_FACE_E", "1")
    assert schedule((256, 256, 256), 12, 0, 0, 1) == FACES
    assert schedule((256, 256, 256), 6, 0, 0, 1) == INTERIOR  # not a multiple of 16 bytes
