"""Near-to-far contraction: the sums folded about the middle of each face, and
several faces per CTA, against the float64 direct sums of ``oracle/n2f_oracle.py``.

Sizes: one and two samples a side, odd and even counts (an odd count's middle sample
pairs with itself), pair counts on both sides of a K step (16 pairs), of a batch of
three K steps and of an n tile (16 pairs); faces of different sizes in one CTA, with a
last group that is not full.

Tolerances, relative to the norm of the result: a BF16 pair holds a factor to 2^-17 and
the product without lo·lo to 2^-16, a TF32 factor to 2^-11; the errors of the two factors
and of many samples add up as random signs, so 2^-15.6 = 2e-5 and 2^-10 = 1e-3 hold them.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from oracle import n2f_oracle  # noqa: E402

TOL = {"bf16x3": 2e-5, "tf32": 1e-3}


def _case(sizes, nfreq, n_obs, dtype, seed=11):
    rng = np.random.default_rng(seed)
    faces = []
    for i, (npp, nqq) in enumerate(sizes):
        cur = (rng.standard_normal((nfreq, npp, nqq, 4)) +
               1j * rng.standard_normal((nfreq, npp, nqq, 4)))
        faces.append(dict(normal=i // 2 % 3, x_n=0.02 * i, o_p=-0.01 + 1e-3 * i, o_q=0.5e-3,
                          pitch=1e-3 * (1 + 0.1 * i), cur=cur.astype(dtype)))
    dirs = rng.standard_normal((n_obs, 3))
    freqs = np.linspace(10e9, 40e9, nfreq)
    return faces, freqs, dirs / np.linalg.norm(dirs, axis=1, keepdims=True)


@pytest.mark.parametrize("sizes,nfreq,n_obs", [
    ([(1, 1)], 1, 1),
    ([(1, 2), (2, 1), (2, 2), (3, 1)], 2, 5),
    ([(31, 32), (32, 33), (33, 34)], 2, 129),
    ([(96, 31), (97, 64), (98, 65)], 1, 128),
    ([(7, 40), (100, 3), (34, 35), (129, 1), (64, 66)], 16, 300),
])
@pytest.mark.parametrize("mode", ["bf16x3", "tf32"])
def test_folded_contraction_vs_direct_sums(sizes, nfreq, n_obs, mode):
    from opencl_fdtd_solver_b200.n2f import N2FFace, near2far_contract

    for dtype in (np.complex64, np.complex128):
        faces, freqs, dirs = _case(sizes, nfreq, n_obs, dtype)
        ref = n2f_oracle.contract(faces, freqs, dirs)
        dev = [N2FFace(**{**f, "cur": torch.as_tensor(f["cur"], device="cuda")}) for f in faces]
        got = near2far_contract(dev, freqs, dirs, mode=mode).cpu().numpy()
        err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
        assert err <= TOL[mode], (dtype, err)
