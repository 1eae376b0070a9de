"""Float64 far-field sums with separated phases against the oracle's direct sums (GPU).

Enough directions that ``fdtd_farfield`` takes ``k_farfield_nl_sep``, on boxes whose
faces end inside a column group, have an odd row, or are a single sample wide; and
one count of directions below the line, for the direct kernel.

Tolerance: both sides round a phase of up to k·R (about 60 radians here) by a few
ulp, so a sum of n samples differs by at most about 60·2⁻⁵²·few ≈ 5e-14 of the sum
of magnitudes; 1e-11 of the largest far field covers the cancellation between faces.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("span,n_obs", [((22, 17, 9), 401), ((1, 8, 30), 415), ((16, 1, 1), 500),
                                        ((33, 70, 5), 799), ((22, 17, 9), 399)])
def test_separated_sums_vs_oracle(span, n_obs):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from opencl_fdtd_solver_b200 import CUDAFDTD, CUDANear2FarMonitor
    from oracle.cpu_fdtd import OracleFDTD
    from oracle.dft_oracle import OracleNear2FarMonitor

    shape = tuple(s + 7 for s in span)
    dl = 1e-3
    centre = [(3 + (s - 1) / 2) * dl for s in span]
    size = [(s - 1) * dl for s in span]
    freqs = [30e9, 41e9]
    g = CUDAFDTD(shape, dl, npml=1, dtype=np.float64)
    o = OracleFDTD(shape, dl, npml=1, dtype=np.float64)
    mg = CUDANear2FarMonitor(g, centre, size, freqs)
    mo = OracleNear2FarMonitor(o, centre, size, freqs)
    assert (mg.nxf, mg.nyf, mg.nzf) == span
    rng = np.random.default_rng(3)
    acc = rng.standard_normal(tuple(mg.acc.shape))
    mg.acc.copy_(torch.from_numpy(acc))
    for c, name in enumerate(("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")):
        mo.dft[name] = acc[c, ..., 0] + 1j * acc[c, ..., 1]
    v = rng.standard_normal((n_obs, 3))
    pts = 2.0 * v / np.linalg.norm(v, axis=1, keepdims=True)
    pts[0] = (0.0, 0.0, 1.5)
    for fi in (0, 1):
        got, ref = mg.get_farfields(pts, fi), mo.get_farfields(pts, fi)
        assert got.dtype == np.complex128 and got.shape == (n_obs, 6)
        assert np.abs(got - ref).max() <= 1e-11 * np.abs(ref).max(), fi
