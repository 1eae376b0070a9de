"""Split-BF16 contraction of currents whose sums leave float32 (GPU).

The kernel sums up to four currents about the middle of a face before it rounds them,
so finite currents above 8.5e37 overflow there although their far field, in which the
phases cancel, fits float32.  Faces of one to a few rows with such currents beside faces
of ordinary ones, against the float64 direct sums; every result fits float32.

Tolerance: that of the contraction in range (a BF16 pair holds a factor to 2^-17, the
product without lo·lo to 2^-16), 2e-5 of the norm, which the direct sums are well inside.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import n2f_oracle  # noqa: E402

PITCH, FREQ = 6e-3, 0.6 * 299792458.0 / 6e-3  # 0.6 wavelengths a sample


def _face(normal, npp, nqq, nfreq, dtype, peak):
    cur = np.zeros((nfreq, npp, nqq, 4), dtype)
    cur[...] = peak * np.array([1.0, 1j, -1.0, 0.6 + 0.7j])
    return dict(normal=normal, x_n=1e-3, o_p=0.0, o_q=0.0, pitch=PITCH, cur=cur)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("sizes,peaks", [
    ([(2, 2)], [1.5e38]),
    ([(1, 2), (2, 1)], [1.75e38, 1.75e38]),   # two currents a sum
    ([(3, 3)], [1e38]),                     # a middle sample
    ([(2, 2), (40, 36)], [1.5e38, 1.0]),    # beside an ordinary face
])
def test_large_currents_vs_direct_sums(sizes, peaks, dtype):
    from opencl_fdtd_solver_b200.n2f import N2FFace, near2far_contract

    rng = np.random.default_rng(7)
    sign = np.array([[a, b, c] for a in (1, -1) for b in (1, -1) for c in (1, -1)], float)
    dirs = np.concatenate([sign, sign + 0.02 * rng.standard_normal((8, 3)), sign])
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    freqs = np.array([FREQ, 1.02 * FREQ])
    faces = [_face(i, *s, 2, dtype, v) for i, (s, v) in enumerate(zip(sizes, peaks))]
    ref = n2f_oracle.contract(faces, freqs, dirs)
    assert max(np.abs(ref.real).max(), np.abs(ref.imag).max()) < 3.3e38
    dev = [N2FFace(**{**f, "cur": torch.as_tensor(f["cur"], device="cuda")}) for f in faces]
    got = near2far_contract(dev, freqs, dirs, mode="bf16x3").cpu().numpy().astype(np.complex128)
    assert np.isfinite(got).all()
    scale = 1e-38
    err = np.linalg.norm((got - ref) * scale) / np.linalg.norm(ref * scale)
    assert err <= 2e-5, err


def test_currents_that_are_not_finite_stay_so():
    from opencl_fdtd_solver_b200.n2f import N2FFace, near2far_contract

    f = _face(2, 5, 4, 1, np.complex64, 1.0)
    f["cur"][0, 3, 2, 1] = np.inf
    dev = [N2FFace(**{**f, "cur": torch.as_tensor(f["cur"], device="cuda")})]
    got = near2far_contract(dev, [FREQ], [[0.3, 0.5, 0.8]], mode="bf16x3").cpu().numpy()
    assert not np.isfinite(got[0, 0, 1]) and np.isfinite(got[0, 0, [2, 5]]).all()
