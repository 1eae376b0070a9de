"""The step profile names what ran: each schedule fills its own slots (GPU)."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def profile(g, n):
    """(summed ms per slot, steps per schedule) of n steps."""
    from opencl_fdtd_solver_b200 import _capi as capi

    capi.run("fdtd_profile_steps", 1)
    g.run(n)
    capi.run("fdtd_profile_steps", 0)
    ms, steps = (ctypes.c_double * 5)(), ctypes.c_int32()
    sched = (ctypes.c_int32 * capi.FDTD_SCHEDULES)()
    capi.run("fdtd_profile_read", ms, ctypes.byref(steps))
    capi.run("fdtd_profile_schedules", sched)
    assert steps.value == n == sum(sched)
    return list(ms), list(sched)


@pytest.mark.parametrize("shape,npml,nfreq,schedule,filled", [
    ((64, 64, 64), 8, 1, "GRID", (0, 4)), ((37, 41, 53), 6, 1, "GRID", (0, 4)),
    ((96, 96, 62), 8, 4, "GRID", (0, 3, 4)),  # a z plane's DFTs after the E launch
    ((192, 160, 192), 8, 1, "MARCH", (2, 3)), ((40, 36, 48), 6, 1, "INTERIOR", (0, 2, 3, 4)),
])
def test_profile_slots_of_each_schedule(shape, npml, nfreq, schedule, filled, monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, CUDAPlaneDFTMonitor, _capi as capi

    monkeypatch.delenv("FDTD_B200_FACE_E", raising=False)
    g = CUDAFDTD(shape, 1e-3, npml=npml, dtype=np.float32)
    CUDAPlaneDFTMonitor(g, 2, shape[2] // 2, [30e9 + 1e9 * q for q in range(nfreq)])
    g.run(2)
    ms, sched = profile(g, 5)
    assert sched[getattr(capi, "FDTD_SCHEDULE_" + schedule)] == 5
    # slot 1 is an empty span of the side stream, not a launch, with the interior march
    assert [q for q in (0, 2, 3, 4) if ms[q] > 0] == list(filled)
    assert ms[1] == 0 or schedule == "INTERIOR"
