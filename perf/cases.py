"""Performance cases of the FDTD engine: the calls a simulation program makes.

Four kinds of work, each through the package's public entry points:

* ``run``      : ``CUDAFDTD.run`` for a few steps of a simulation that is under
                 way (fields and DFT accumulators nonzero everywhere), with the
                 source callback and monitors such a program registers
* ``adjoint``  : ``EpsilonAdjoint.value_and_grad``, a whole forward and reverse solve
* ``contract`` : ``near2far_contract``, the far-field sums of many directions and
                 frequencies
* ``farfield`` : ``CUDANear2FarMonitor.get_farfields``, the float64 transform

Sizes are those of the repository's tests and bench configurations, and
generic ones between 32 and 512 cells per axis.  ``exact`` evaluates the same
results in float64 with plain torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from opencl_fdtd_solver_b200 import (CUDAFDTD, CUDANear2FarMonitor, CUDAPlaneDFTMonitor,
                                     DFTObjective, EpsilonAdjoint, N2FFace, near2far_contract)

C0 = 299_792_458.0
MU0 = 4e-7 * math.pi
EPS0 = 1.0 / (MU0 * C0**2)
ETA0 = math.sqrt(MU0 / EPS0)
DL = 1e-3
FIELDS = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


# ------------------------------------------------------------------ the cases
def _run_case(name, nx, ny, nz, npml, steps, *, f64=False, lossy=False, medium="vacuum",
              source="point", monitor="none", nfreq=0, courant=0.0):
    return {"kind": "run", "name": name, "nx": nx, "ny": ny, "nz": nz, "npml": npml,
            "steps": steps, "f64": f64, "lossy": lossy, "medium": medium, "source": source,
            "monitor": monitor, "nfreq": nfreq, "courant": courant}


def listed():
    return [
        # a unit-test sized grid with odd extents: launch latency and host work
        _run_case("run_37x41x53", 37, 41, 53, 6, 20, monitor="x", nfreq=1),
        # the small configuration: a point dipole in vacuum, one mid-plane DFT
        _run_case("run_64", 64, 64, 64, 8, 20, monitor="z", nfreq=3, courant=0.5),
        # an ordinary lossy model with the engine's default CPML thickness, no monitor
        _run_case("run_192_lossy", 192, 192, 192, 20, 8, lossy=True, medium="blocky"),
        # extents as a mesher gives them: nothing is a multiple of anything, lossy block
        _run_case("run_181x230x155_lossy", 181, 230, 155, 10, 8, lossy=True, medium="blocky",
                  source="sheet", monitor="y", nfreq=2),
        # the medium configuration: scattering by a sphere, closed Huygens box at 8 frequencies
        _run_case("run_256_box", 256, 256, 256, 12, 8, medium="sphere", source="sheet",
                  monitor="box", nfreq=8),
        # the double-precision run of the bandwidth configuration
        _run_case("run_384_f64", 384, 384, 384, 16, 4, f64=True, medium="blocky", monitor="z",
                  nfreq=4, courant=0.5),
        # the bandwidth configuration
        _run_case("run_512", 512, 512, 512, 16, 4, medium="blocky", monitor="z", nfreq=4,
                  courant=0.5),
        # one iteration of an inverse design in double precision on a small grid
        {"kind": "adjoint", "name": "adjoint_48_f64", "nx": 48, "ny": 48, "nz": 48, "npml": 8,
         "f64": True, "dx": 16, "dz": 8, "patch": 12, "steps": 100},
        # one iteration of an inverse design at the adjoint configuration
        {"kind": "adjoint", "name": "adjoint_160x160x96", "nx": 160, "ny": 160, "nz": 96,
         "npml": 12, "f64": False, "dx": 96, "dz": 16, "patch": 32, "steps": 1000},
        # a preview of a scatterer's full pattern in TF32
        {"kind": "contract", "name": "contract_89_tf32", "n": 89, "nfreq": 8, "nth": 181,
         "nph": 91, "mode": "tf32"},
        # the near-to-far configuration: a 320-cell box, 32 frequencies, split-BF16
        {"kind": "contract", "name": "contract_320_bf16x3", "n": 320, "nfreq": 32, "nth": 361,
         "nph": 181, "mode": "bf16x3"},
        # the pattern of the medium configuration's box at one frequency, float64 sums
        {"kind": "farfield", "name": "farfield_89", "n": 89, "nfreq": 8, "nth": 181, "nph": 91},
    ]


def draw(rng):
    kind = rng.choice(["run"] * 8 + ["adjoint"] + ["contract"] * 2 + ["farfield"])

    def log_int(lo, hi, p_even=0.5):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        if rng.random() < p_even:  # half the extents people type are multiples of 8
            n = 8 * max(1, round(n / 8))
        return max(lo, min(hi, n))

    if kind == "run":
        f64 = rng.random() < 0.25
        top = 384 if f64 else 512
        dims = [log_int(32, top) for _ in range(3)]
        npml = rng.choice([4, 6, 8, 10, 12, 16, 20])
        npml = min(npml, (min(dims) - 8) // 2)
        monitor = rng.choice(["none", "x", "y", "z", "box"])
        return {k: v for k, v in _run_case(
            "", *dims, npml, 4 if dims[0] * dims[1] * dims[2] > 2e7 else 8, f64=f64,
            lossy=rng.random() < 0.25, medium=rng.choice(["vacuum", "sphere", "blocky"]),
            source=rng.choice(["point", "sheet"]), monitor=monitor,
            nfreq=0 if monitor == "none" else rng.randint(1, 8),
            courant=rng.choice([0.0, 0.5])).items() if k != "name"}
    if kind == "adjoint":
        dims = [log_int(48, 160) for _ in range(2)] + [log_int(48, 96)]
        return {"kind": "adjoint", "nx": dims[0], "ny": dims[1], "nz": dims[2],
                "npml": rng.choice([6, 8, 10, 12]), "f64": rng.random() < 0.25,
                "dx": rng.randint(8, min(dims[:2]) - 30), "dz": rng.randint(4, 12),
                "patch": rng.randint(4, 16), "steps": rng.randint(60, 200)}
    n = log_int(24, 320, 0.3)
    nth = rng.randint(46, 361)
    nfreq = rng.randint(1, 8)
    case = {"kind": kind, "n": n, "nfreq": nfreq, "nth": nth, "nph": nth // 2 + 1}
    if kind == "contract":
        case["mode"] = rng.choice(["bf16x3", "tf32"])
    else:  # the direct sum costs directions x samples
        case["n"] = min(case["n"], 128)
        case["nth"] = min(nth, 181)
        case["nph"] = case["nth"] // 2 + 1
    return case


# -------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _shape(case):
    return case["nx"], case["ny"], case["nz"]


def _media(case, seed):
    """Host εr and σ (or None) of a run case."""
    shape = _shape(case)
    rng = np.random.default_rng([seed, 1])
    if case["medium"] == "blocky":
        vals = rng.uniform(1.0, 12.0, [-(-n // 8) for n in shape]).astype(np.float32)
        eps = vals.repeat(8, 0).repeat(8, 1)[:shape[0], :shape[1]].repeat(8, 2)
        eps = np.ascontiguousarray(eps[:, :, :shape[2]])
    else:
        eps = np.ones(shape, np.float32)
        if case["medium"] == "sphere":
            r = 0.16 * min(shape)
            x, y, z = np.ogrid[tuple(slice(0, n) for n in shape)]
            c = [n // 2 for n in shape]
            inside = (x - c[0])**2 + (y - c[1])**2 + (z - c[2])**2 < r * r
            eps[inside] = rng.uniform(2.0, 6.0)
    sigma = None
    if case["lossy"]:
        sigma = np.zeros(shape, np.float32)
        sl = tuple(slice(n // 4, 3 * n // 4) for n in shape)
        sigma[sl] = rng.uniform(0.01, 0.5)
    return eps, sigma


def _smooth_field(shape, gen, scale, dtype):
    """A wave-filled grid: a few standing waves of 10 to 40 cells and 1 % noise."""
    dev = gen.device
    out = torch.randn(shape, generator=gen, device=dev, dtype=dtype) * (0.01 * scale)
    for _ in range(3):
        u = torch.rand(7, generator=gen, device=dev, dtype=torch.float64)
        w = [torch.cos(2 * math.pi * (torch.arange(n, device=dev, dtype=torch.float64)
                                      / (10.0 + 30.0 * u[a]) + u[3 + a])).to(dtype)
             for a, n in enumerate(shape)]
        out.addcmul_((w[0][:, None] * w[1][None, :])[:, :, None], w[2][None, None, :],
                     value=float(scale * (0.5 + u[6])))
    return out


def _initial_fields(case, seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    dtype = torch.float64 if case["f64"] else torch.float32
    for n in FIELDS:
        yield n, _smooth_field(_shape(case), gen, 1.0 if n[0] == "E" else 1.0 / ETA0, dtype)


def _freqs(case):
    return [30e9] if case["nfreq"] == 1 else [float(f) for f in
                                               np.linspace(20e9, 40e9, case["nfreq"])]


def _sheet(case):
    """(z, i0, i1, j0, j1, taper) of the current source of a run case."""
    nx, ny, nz = _shape(case)
    p = case["npml"]
    if case["source"] == "point":
        return nz // 2, nx // 2, nx // 2 + 1, ny // 2, ny // 2 + 1, False
    return min(p + 3, nz // 2), p, nx - p, p, ny - p, True


def _box(case):
    """Centre and size of the Huygens box of a run case (about a third of the grid)."""
    centre = [n // 2 * DL for n in _shape(case)]
    size = [2 * max(2, int(0.17 * n)) * DL for n in _shape(case)]
    return centre, size


def _amplitude(t):
    return math.sin(2.0 * math.pi * 30e9 * t)


def _directions(case):
    th = np.deg2rad(np.linspace(0.0, 180.0, case["nth"]))
    ph = np.deg2rad(np.linspace(0.0, 180.0, case["nph"], endpoint=False))
    t, p = np.meshgrid(th, ph, indexing="ij")
    return np.stack([np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)], -1).reshape(-1, 3)


def _design(case):
    (nx, ny, nz), d, dz = _shape(case), case["dx"], case["dz"]
    i0, j0, k0 = (nx - d) // 2, (ny - d) // 2, (nz - dz) // 2
    return (i0, i0 + d), (j0, j0 + d), (k0, k0 + dz)


def _patch(case):
    """The objective's plane and patch: above the design box."""
    nx, ny, nz = _shape(case)
    w = case["patch"]
    k = min(nz - case["npml"] - 2, (nz + case["dz"]) // 2 + 4)
    return k, (((nx - w) // 2, (nx + w) // 2), ((ny - w) // 2, (ny + w) // 2))


def _design_eps(case, seed):
    rng = np.random.default_rng([seed, 2])
    shape = tuple(hi - lo for lo, hi in _design(case))
    z = rng.standard_normal(shape)
    for a in range(3):  # a smooth random structure
        for _ in range(4):
            z = 0.5 * z + 0.25 * (np.roll(z, 1, a) + np.roll(z, -1, a))
    return 1.0 + 3.0 / (1.0 + np.exp(-z / z.std()))


def _adjoint_sheet(case):
    nx, ny, nz = _shape(case)
    p = case["npml"]
    return p + 2, p, nx - p, p, ny - p, True


def _face_currents(case, seed):
    """(normal, x_n, o_p, o_q, complex64 [nfreq][n][n][4]) of the six faces of a cubic box."""
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    n, nf = case["n"], case["nfreq"]
    a = torch.arange(n, device=_device(), dtype=torch.float32) / n - 0.5
    env = torch.exp(-6.0 * (a[:, None]**2 + a[None, :]**2)) * DL**2
    for normal in range(3):
        for side in range(2):
            cur = torch.randn((nf, n, n, 4), generator=gen, device=_device(),
                              dtype=torch.complex64)
            yield normal, side * n * DL, 0.5 * DL, 0.5 * DL, cur * env[None, :, :, None]


def _farfield_box(case):
    """Grid extent, centre and size of the box of a farfield case."""
    grid = case["n"] + 23
    return grid, grid // 2 * DL, (case["n"] - 1) * DL


def _face_dft(case, shape, seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    acc = torch.randn(shape, generator=gen, device=_device(), dtype=torch.float64) * 1e-12
    acc[3:] /= ETA0
    return acc


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        fd = CUDAFDTD(_shape(case), DL, npml=case["npml"],
                      dtype=np.float64 if case["f64"] else np.float32,
                      courant=case["courant"] or None)
        if case["medium"] != "vacuum" or case["lossy"]:
            eps, sigma = _media(case, seed)
            fd.set_epsilon(eps, sigma_array=sigma)
        z, i0, i1, j0, j1, taper = _sheet(case)
        fd.add_source(lambda f: f.add_source_Jx(z, _amplitude(f.t), i0, i1, j0, j1,
                                                rim_taper=taper))
        mon = None
        if case["monitor"] == "box":
            centre, size = _box(case)
            mon = CUDANear2FarMonitor(fd, centre, size, _freqs(case))
        elif case["monitor"] != "none":
            axis = "xyz".index(case["monitor"])
            mon = CUDAPlaneDFTMonitor(fd, axis, _shape(case)[axis] // 2, _freqs(case),
                                      ("Ex", "Hy") if case["nfreq"] == 3 else ("Ex",))
        for n, values in _initial_fields(case, seed):
            fd.field_tensor(n).copy_(values)
        return {"case": case, "fd": fd, "mon": mon}
    if kind == "adjoint":
        fd = CUDAFDTD(_shape(case), DL, npml=case["npml"],
                      dtype=np.float64 if case["f64"] else np.float32)
        z, i0, i1, j0, j1, taper = _adjoint_sheet(case)
        fd.add_source(lambda f: f.add_source_Jx(z, _amplitude(f.t), i0, i1, j0, j1,
                                                rim_taper=taper))
        k, patch = _patch(case)
        adj = EpsilonAdjoint(fd, _design(case), case["steps"], DFTObjective("z", k, patch, [30e9]))
        return {"case": case, "adj": adj, "eps": _design_eps(case, seed)}
    if kind == "contract":
        faces = [N2FFace(normal=m, x_n=x, o_p=p, o_q=q, pitch=DL, cur=cur)
                 for m, x, p, q, cur in _face_currents(case, seed)]
        return {"case": case, "faces": faces, "freqs": _freqs(case), "dirs": _directions(case)}
    grid, centre, size = _farfield_box(case)
    fd = CUDAFDTD((grid,) * 3, DL, npml=8)
    mon = CUDANear2FarMonitor(fd, (centre,) * 3, (size,) * 3, _freqs(case))
    mon.acc.copy_(_face_dft(case, mon.acc.shape, seed))
    return {"case": case, "mon": mon, "points": _directions(case)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        fd = state["fd"]
        fd.run(case["steps"])
        out = {n: fd.field_tensor(n) for n in FIELDS}
        if state["mon"] is not None:
            out["dft"] = state["mon"].acc
        return out
    if kind == "adjoint":
        value, grad = state["adj"].value_and_grad(state["eps"])
        return {"value": value, "grad": grad}
    if kind == "contract":
        return near2far_contract(state["faces"], state["freqs"], state["dirs"],
                                 mode=case["mode"])
    return state["mon"].get_farfields(state["points"], case["nfreq"] // 2)


# ---------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind in ("contract", "farfield"):
        n, nf = case["n"], case["nfreq"] if kind == "contract" else 1
        n_obs = case["nth"] * case["nph"]
        samples = 6 * n * n
        item = 8 if kind == "contract" else 16
        # per direction and sample: four complex multiply-adds
        return {"bytes": float(samples * 4 * nf * item + n_obs * nf * 6 * item),
                "flops": 32.0 * n_obs * samples * nf}
    nx, ny, nz = _shape(case)
    p, item, steps = case["npml"], 8 if case["f64"] else 4, case["steps"]
    cells = nx * ny * nz
    psi = 4 * 2 * 2 * p * (ny * nz + nx * nz + nx * ny)  # four arrays a face, read and written
    if kind == "run":
        # per step: six fields read and written, three coefficients (six when lossy)
        per = (12 + 3 * (2 if case["lossy"] else 1)) * cells + psi
        total = float(per * item)
        nf = case["nfreq"]
        if case["monitor"] == "box":
            b = [2 * max(2, int(0.17 * n)) + 1 for n in (nx, ny, nz)]
            face = 2 * (b[0] * b[1] + b[1] * b[2] + b[0] * b[2])
            total += face * (4 * item + 4 * nf * 32)
        elif case["monitor"] != "none":
            plane = cells // (nx, ny, nz)["xyz".index(case["monitor"])]
            total += (2 if nf == 3 else 1) * plane * (item + nf * 32)
        return {"bytes": total * steps, "flops": 36.0 * cells * steps}
    # forward and reverse step alike move the state once; E of the design box is
    # written by the one and read by the other
    box = math.prod(hi - lo + 1 for lo, hi in _design(case))
    per = 2 * ((12 + 3) * cells + psi) + 2 * 3 * box
    return {"bytes": float(per * item + 3 * box * 16) * steps, "flops": 80.0 * cells * steps}


# ------------------------------------------------- the same results in float64
def _profiles(n, npml, dt, offset):
    """(b, c, κ) of one axis (CFS-CPML, cubic grading), float64 on the device."""
    b, c, kappa = np.ones(n), np.zeros(n), np.ones(n)
    smax = 0.8 * 4.0 / (ETA0 * DL)
    for layer in range(npml):
        for lo, i in ((True, layer), (False, n - npml + layer)):
            xi = ((npml - layer - offset) if lo else (layer + 1 - offset)) / npml
            xi = max(xi, 0.0)
            sig, kap, alp = smax * xi**3, 1.0 + 14.0 * xi**3, 0.05 / ETA0 * (1.0 - xi)
            b[i] = math.exp(-((sig / kap + alp) * dt / EPS0))
            den = sig + kap * alp
            c[i] = 0.0 if den == 0 else sig / kap * (b[i] - 1.0) / den / DL
            kappa[i] = kap
    return [torch.from_numpy(v).to(_device()) for v in (b, c, kappa)]


def _edge_mean(a, axis):
    out = a.clone()
    n = a.shape[axis]
    out.narrow(axis, 0, n - 1).copy_(0.5 * (a.narrow(axis, 0, n - 1) + a.narrow(axis, 1, n - 1)))
    return out


def _coefficients(eps, sigma, dt):
    """ca, cb per component from cell-centred εr, σ (float64 device tensors)."""
    ca, cb = [], []
    for a in range(3):
        e = _edge_mean(eps, a)
        if sigma is None:
            ca.append(None)
            cb.append(dt / (EPS0 * e))
        else:
            loss = _edge_mean(sigma, a) * dt / (2.0 * EPS0 * e)
            ca.append((1.0 - loss) / (1.0 + loss))
            cb.append(dt / (EPS0 * e) / (1.0 + loss))
    return ca, cb


class _Exact:
    """The Yee/CPML step on float64 torch tensors."""

    # (component, derivative axis, differentiated component, sign) of curl
    TERMS = ((0, 1, 2, 1), (0, 2, 1, -1), (1, 2, 0, 1), (1, 0, 2, -1), (2, 0, 1, 1), (2, 1, 0, -1))

    def __init__(self, shape, npml, dt):
        self.shape, self.npml, self.dt = shape, npml, dt
        self.ph = [_profiles(n, npml, dt, 0.5) for n in shape]
        self.pe = [_profiles(n, npml, dt, 0.0) for n in shape]

    def zeros(self):
        z = lambda s: torch.zeros(s, device=_device(), dtype=torch.float64)  # noqa: E731
        psi = []
        for _, axis, _, _ in self.TERMS:
            s = list(self.shape)
            s[axis] = 2 * self.npml
            psi.append(z(s))
        return [z(self.shape) for _ in range(6)], psi, [p.clone() for p in psi]

    def _slabs(self, v, axis):
        """v on the two CPML slabs of an axis, low layers first."""
        n, p = v.shape[axis], self.npml
        return torch.cat([v.narrow(axis, 0, p), v.narrow(axis, n - p, p)], axis)

    def _curl(self, field, prof, psi, forward):
        out, new_psi = [0.0, 0.0, 0.0], []
        p = self.npml
        for q, (comp, axis, src, sign) in enumerate(self.TERMS):
            f, n = field[src], self.shape[axis]
            d = f.narrow(axis, 1, n - 1) - f.narrow(axis, 0, n - 1)
            edge = torch.zeros_like(f.narrow(axis, 0, 1))
            d = torch.cat([d, edge] if forward else [edge, d], axis)
            view = [1, 1, 1]
            view[axis] = -1
            b, c, kappa = prof[axis]
            bs, cs = (torch.cat([v[:p], v[n - p:]]).view(view) for v in (b, c))
            ps = bs * psi[q] + cs * self._slabs(d, axis)
            new_psi.append(ps)
            rest = list(self.shape)
            rest[axis] = n - 2 * p
            pad = torch.cat([ps.narrow(axis, 0, p), torch.zeros(rest, device=d.device,
                                                               dtype=d.dtype),
                             ps.narrow(axis, p, p)], axis)
            out[comp] = out[comp] + sign * (d / (kappa * DL).view(view) + pad)
        return out, new_psi

    def step(self, f, psi_h, psi_e, ca, cb, sheet, t):
        """One step from E^n, H^{n-1/2} at time t; returns the advanced state."""
        curl, psi_h = self._curl(f[:3], self.ph, psi_h, True)
        h = [f[3 + c] - self.dt / MU0 * curl[c] for c in range(3)]
        e = [f[0] + self.injection(sheet, t + 0.5 * self.dt, cb[0]), f[1], f[2]]
        curl, psi_e = self._curl(h, self.pe, psi_e, False)
        e = [(e[c] if ca[c] is None else ca[c] * e[c]) + cb[c] * curl[c] for c in range(3)]
        return e + h, psi_h, psi_e

    def injection(self, sheet, t, cb):
        z, i0, i1, j0, j1, taper = sheet
        w = torch.ones((i1 - i0, j1 - j0), device=_device(), dtype=torch.float64)
        if taper:
            w[0] *= 0.8
            w[-1] *= 0.8
            w[:, 0] *= 0.8
            w[:, -1] *= 0.8
            w *= w.numel() / w.sum()
        full = torch.zeros(self.shape, device=_device(), dtype=torch.float64)
        full[i0:i1, j0:j1, z] = w * _amplitude(t)
        return -cb * full


def _exact_box(case, fd_box, f, dt, t, acc, phases):
    """Adds one step's co-located tangential samples to the face DFTs."""
    (x0, x1, y0, y1, z0, z1) = fd_box
    n = _shape(case)
    span = (slice(x0, x1 + 1), slice(y0, y1 + 1), slice(z0, z1 + 1))
    off = 0
    for face, (ax, at) in enumerate(((0, x0), (0, x1), (1, y0), (1, y1), (2, z0), (2, z1))):
        lo = [max(0, s.start - 1) for s in span]
        hi = [min(n[a], s.stop + 1) for a, s in enumerate(span)]
        lo[ax], hi[ax] = max(0, at - 1), at + 1
        win = tuple(slice(a, b) for a, b in zip(lo, hi))
        pick = [slice(s.start - a, s.stop - a) for s, a in zip(span, lo)]
        pick[ax] = at - lo[ax]

        def shift(v, axis):  # v at +1 along axis, clamped at the grid's edge
            k = v.shape[axis]
            return torch.cat([v.narrow(axis, 1, k - 1), v.narrow(axis, k - 1, 1)], axis)

        def back(v, axis):
            return torch.cat([v.narrow(axis, 0, 1), v.narrow(axis, 0, v.shape[axis] - 1)], axis)

        others = [a for a in range(3) if a != ax]
        size = 1
        for a in others:
            size *= span[a].stop - span[a].start
        for comp in others:
            other = others[0] if others[1] == comp else others[1]
            v = f[comp][win]
            e = (0.5 * (v + shift(v, other)))[tuple(pick)].reshape(-1)
            acc[comp, :, off:off + size] += phases[:, None] * e
            v = f[3 + comp][win]
            v = v + back(v, ax)
            # the reference's means: along the component's axis on x and y faces
            h = (0.25 * (v + shift(v, comp if ax < 2 else other)))[tuple(pick)].reshape(-1)
            ph = phases * torch.exp(-0.5j * 2 * math.pi * dt * torch.tensor(
                _freqs(case), device=_device(), dtype=torch.float64))
            acc[3 + comp, :, off:off + size] += ph[:, None] * h
        off += size


def _exact_run(case, seed):
    shape, npml = _shape(case), case["npml"]
    dt = (case["courant"] or 0.99 / math.sqrt(3.0)) * DL / C0
    ex = _Exact(shape, npml, dt)
    _, psi_h, psi_e = ex.zeros()
    f = [v.double() for _, v in _initial_fields(case, seed)]
    eps, sigma = _media(case, seed) if case["medium"] != "vacuum" or case["lossy"] else (
        np.ones(shape, np.float32), None)
    up = lambda a: torch.from_numpy(a).to(_device()).double()  # noqa: E731
    ca, cb = _coefficients(up(eps), None if sigma is None else up(sigma), dt)
    freqs = torch.tensor(_freqs(case) if case["nfreq"] else [], device=_device(),
                         dtype=torch.float64)
    half = torch.exp(-0.5j * 2 * math.pi * freqs * dt)
    acc = box = None
    if case["monitor"] == "box":
        centre, size = _box(case)
        box = []
        for a, n in enumerate(shape):
            box += [max(0, round((centre[a] - size[a] / 2) / DL)),
                    min(n - 1, round((centre[a] + size[a] / 2) / DL))]
        e = [box[2 * a + 1] - box[2 * a] + 1 for a in range(3)]
        acc = torch.zeros((6, len(freqs), 2 * (e[0] * e[1] + e[1] * e[2] + e[0] * e[2])),
                          device=_device(), dtype=torch.complex128)
    t = 0.0
    plane = None
    if case["monitor"] in ("x", "y", "z"):
        axis = "xyz".index(case["monitor"])
        plane = axis, shape[axis] // 2, (0, 4) if case["nfreq"] == 3 else (0,)
        rest = [n for a, n in enumerate(shape) if a != axis]
        acc = torch.zeros((len(plane[2]), len(freqs), *rest), device=_device(),
                          dtype=torch.complex128)
    for _ in range(case["steps"]):
        f, psi_h, psi_e = ex.step(f, psi_h, psi_e, ca, cb, _sheet(case), t)
        t += dt
        ph = torch.exp(2j * math.pi * freqs * t) * dt
        if plane is not None:
            for q, comp in enumerate(plane[2]):
                w = ph if comp < 3 else ph * half
                acc[q] += w[:, None, None] * f[comp].select(plane[0], plane[1])
        elif box is not None:
            _exact_box(case, box, f, dt, t, acc, ph)
    out = {n: f[c] for c, n in enumerate(FIELDS)}
    if acc is not None:
        out["dft"] = torch.view_as_real(acc)
    return out


def _exact_adjoint(case, seed):
    """Objective and gradient by torch autograd, in segments from saved states."""
    shape, npml, steps = _shape(case), case["npml"], case["steps"]
    dt = 0.99 * DL / (C0 * math.sqrt(3.0))
    ex = _Exact(shape, npml, dt)
    design = tuple(slice(lo, hi) for lo, hi in _design(case))
    eps_d = torch.from_numpy(_design_eps(case, seed)).to(_device()).requires_grad_(True)
    with torch.enable_grad():
        full = torch.ones(shape, device=_device(), dtype=torch.float64)
        full[design] = eps_d
        edges = []
        for a in range(3):
            n = shape[a]
            m = 0.5 * (full.narrow(a, 0, n - 1) + full.narrow(a, 1, n - 1))
            edges.append(dt / (EPS0 * torch.cat([m, full.narrow(a, n - 1, 1)], a)))
    cb = [e.detach().requires_grad_(True) for e in edges]
    ca = [None] * 3
    k, ((a0, a1), (b0, b1)) = _patch(case)
    sheet = _adjoint_sheet(case)
    omega = 2.0 * math.pi * 30e9

    def advance(state, n):
        f, ph_, pe_ = ex.step(state[:6], state[6:12], state[12:], ca, cb, sheet, n * dt)
        return f + ph_ + pe_

    def sample(state, n):
        w = complex(math.cos(omega * (n + 1) * dt), math.sin(omega * (n + 1) * dt)) * dt
        return w * state[0][a0:a1, b0:b1, k]

    seg = 20
    f, psi_h, psi_e = ex.zeros()
    state, saved, D = f + psi_h + psi_e, [], 0.0
    with torch.no_grad():
        for n in range(steps):
            if n % seg == 0:
                saved.append(state)
            state = advance(state, n)
            D = D + sample(state, n)
    value = float((D.real**2 + D.imag**2).sum())
    seed_D = 2.0 * D  # dJ/dRe + i dJ/dIm
    grad_cb = [torch.zeros_like(c) for c in cb]
    bar = [torch.zeros_like(s) for s in state]
    for s in range(len(saved) - 1, -1, -1):
        n0, n1 = s * seg, min(steps, (s + 1) * seg)
        with torch.enable_grad():
            start = [v.detach().requires_grad_(True) for v in saved[s]]
            state, d = start, 0.0
            for n in range(n0, n1):
                state = advance(state, n)
                d = d + sample(state, n)
            total = (seed_D.conj() * d).real.sum()
            for v, g in zip(state, bar):
                total = total + (v * g).sum()
            grads = torch.autograd.grad(total, start + cb)
        bar = [g for g in grads[:len(start)]]
        for c in range(3):
            grad_cb[c] += grads[len(start) + c]
        saved[s] = None
    (g,) = torch.autograd.grad(edges, eps_d, grad_cb)
    return {"value": value, "grad": g.cpu().numpy()}


def _phases(gamma, n):
    """e^{j2π γ m} for m < n: [len(gamma)][n] complex128."""
    t = gamma[:, None] * torch.arange(n, device=gamma.device, dtype=torch.float64)
    t = t - torch.round(t)
    return torch.polar(torch.ones_like(t), 2.0 * math.pi * t)


def _face_sums(normal, x_n, o_p, o_q, cur, freq, dirs):
    """Σ_pq e^{jk r̂·r'} cur[p][q][4] for every direction: [n_obs][4] complex128."""
    ip, iq = [a for a in range(3) if a != normal]
    g = freq / C0 * dirs
    lead = g[:, normal] * x_n + g[:, ip] * o_p + g[:, iq] * o_q
    n_p, n_q = cur.shape[:2]
    out = []
    for s in range(0, dirs.shape[0], 8192):
        u = _phases(g[s:s + 8192, ip] * DL, n_p)
        v = _phases(g[s:s + 8192, iq] * DL, n_q)
        T = (u @ cur.reshape(n_p, n_q * 4)).reshape(-1, n_q, 4)
        out.append((v[:, :, None] * T).sum(1))
    return torch.cat(out) * _phases(lead, 2)[:, 1:]


def _exact_contract(case, seed):
    dirs = torch.from_numpy(_directions(case)).to(_device())
    dirs = dirs / torch.linalg.vector_norm(dirs, dim=1, keepdim=True)
    freqs = _freqs(case)
    out = torch.zeros((len(freqs), dirs.shape[0], 6), device=_device(), dtype=torch.complex128)
    for normal, x_n, o_p, o_q, cur in _face_currents(case, seed):
        ip, iq = [a for a in range(3) if a != normal]
        for fi, freq in enumerate(freqs):
            nl = _face_sums(normal, x_n, o_p, o_q, cur[fi].to(torch.complex128), freq, dirs)
            out[fi][:, [ip, iq, 3 + ip, 3 + iq]] += nl
    return out


def _exact_farfield(case, seed):
    n, nf = case["n"], case["nfreq"]
    fi = nf // 2
    freq = _freqs(case)[fi]
    _, centre, size = _farfield_box(case)
    lo, hi = round((centre - size / 2) / DL), round((centre + size / 2) / DL)
    assert hi - lo + 1 == n
    acc = torch.view_as_complex(_face_dft(case, (6, nf, 6 * n * n, 2), seed))[:, fi]
    pts = torch.from_numpy(_directions(case).astype(np.float32).astype(np.float64)).to(_device())
    r = torch.linalg.vector_norm(pts, dim=1, keepdim=True)
    rh = pts / r
    w = torch.ones(n, device=_device(), dtype=torch.float64)
    w[0] = w[-1] = 0.5
    w = (w[:, None] * w[None, :] * DL**2)[:, :, None]
    nl = torch.zeros((pts.shape[0], 6), device=_device(), dtype=torch.complex128)
    for face in range(6):
        normal, out = face // 2, 1.0 if face % 2 else -1.0
        ip, iq = [a for a in range(3) if a != normal]
        v = acc[:, face * n * n:(face + 1) * n * n].reshape(6, n, n)
        nrm = torch.zeros(3, device=_device(), dtype=torch.complex128)
        nrm[normal] = out
        # the solver's signs: J = -n x H, M = n x E
        j = -torch.linalg.cross(nrm.expand(n, n, 3), v[3:].permute(1, 2, 0))
        m = torch.linalg.cross(nrm.expand(n, n, 3), v[:3].permute(1, 2, 0))
        cur = torch.stack([j[..., ip], j[..., iq], m[..., ip], m[..., iq]], -1) * w
        s = _face_sums(normal, (lo, hi)[face % 2] * DL, (lo + 0.5) * DL, (lo + 0.5) * DL,
                       cur.contiguous(), freq, rh)
        nl[:, [ip, iq, 3 + ip, 3 + iq]] += s
    k = 2.0 * math.pi * freq / C0
    N, L = nl[:, :3], nl[:, 3:]
    rc = rh.to(torch.complex128)
    trans = N - (rc * N).sum(1, keepdim=True) * rc
    pref = -1j * k * torch.exp(-1j * k * r) / (4.0 * math.pi * r)
    E = pref * (ETA0 * trans - torch.linalg.cross(rc, L))
    H = -torch.linalg.cross(rc, E) / ETA0
    return torch.cat([E, H], 1).cpu().numpy()


def exact(case, seed):
    with torch.no_grad():
        return {"run": _exact_run, "adjoint": _exact_adjoint, "contract": _exact_contract,
                "farfield": _exact_farfield}[case["kind"]](case, seed)
