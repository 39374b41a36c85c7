"""Performance cases of the engine: what a user's program does with it, through its public entry points.

A case is a dict of plain values; ``kind`` says which part of a program it stands for:

  run        the main loop between two outputs: ``NSVEparticles_step`` (or ``step`` without tracers) once per
             iteration, then the checkpoint (vorticity, tracer positions and rhs history) into pinned host memory
  ensemble   many instances of mixed sizes advanced together, then the members' fields and positions read back
  ift, dft   ``field::ift`` / ``field::dft`` on the caller's device buffers
  stats      ``do_stats``: spectra, moments and histograms of velocity and vorticity
  sample     the tracer output of ``NSVEparticles::do_stats``: velocity and Lagrangian acceleration at the tracers
  rspace     real-space moments and histogram of a caller's device field, any grid size

Grids are the powers of two that the engine takes, 16^3 to 512^3; the real-space statistics take any sizes.
"""
import ctypes
import math
from fractions import Fraction

import numpy as np
import torch

from bfps_b200 import _lib
from bfps_b200._lib import check, lib, ptr
from bfps_b200.solver import NSVEparticles_step, ensemble, particles_system, vorticity_equation

# viscosity and time step by grid size: resolved flows of kinetic energy 0.5 at a CFL number below 0.5
NU = {16: 0.1, 32: 0.1, 64: 0.02, 128: 0.01, 256: 0.005, 512: 0.002}
DT = {16: 0.01, 32: 0.01, 64: 0.008, 128: 0.004, 256: 0.002, 512: 0.001}
NBINS = 256
MAX_VELOCITY, MAX_VORTICITY = 8.0, 80.0


def listed():
    return [
        # the smallest production run: a regression-sized FP64 box, 32 iterations between checkpoints; latency and
        # launches count
        dict(name="run_32_f64", kind="run", n=32, bits=64, dealias="two_thirds", forcing="linear", steps=32,
             tracers=1024, neighbours=2, smoothness=0, order=2),
        # a small FP32 box without tracers (NSVE)
        dict(name="run_64_f32", kind="run", n=64, bits=32, dealias="smooth", forcing="linear", steps=32, tracers=0,
             neighbours=1, smoothness=0, order=1),
        # an FP64 box with an odd number of spline tracers and Kolmogorov forcing
        dict(name="run_128_f64", kind="run", n=128, bits=64, dealias="smooth", forcing="Kolmogorov", steps=16,
             tracers=10007, neighbours=1, smoothness=1, order=4),
        # the benchmark's middle size
        dict(name="run_256_f32", kind="run", n=256, bits=32, dealias="smooth", forcing="linear", steps=16,
             tracers=100000, neighbours=2, smoothness=2, order=4),
        # FP64 with the two-thirds rule, wide stencils
        dict(name="run_256_f64", kind="run", n=256, bits=64, dealias="two_thirds", forcing="linear", steps=8,
             tracers=50001, neighbours=4, smoothness=1, order=3),
        # the headline workload: 512^3 FP32 with 4e6 tracers
        dict(name="run_512_f32", kind="run", n=512, bits=32, dealias="smooth", forcing="linear", steps=8,
             tracers=4000000, neighbours=3, smoothness=2, order=3),
        # the benchmark's batched ensemble: 40 x 32^3, 16 x 64^3, 8 x 128^3, 1e4 tracers each
        dict(name="ensemble_mixed", kind="ensemble", m32=40, m64=16, m128=8, steps=25, tracers=10000, neighbours=2,
             smoothness=0, order=4),
        # one inverse and one forward transform of a 3-vector field in device memory
        dict(name="ift_128_f64", kind="ift", n=128, bits=64),
        dict(name="dft_256_f32", kind="dft", n=256, bits=32),
        # the statistics of one output step
        dict(name="stats_256_f32", kind="stats", n=256, bits=32, dealias="smooth"),
        # the tracer output of one output step
        dict(name="sample_256_f32", kind="sample", n=256, bits=32, dealias="smooth", forcing="linear",
             tracers=100003, neighbours=2, smoothness=2),
        # statistics of a caller's field with odd, unequal sizes
        dict(name="rspace_odd_f64", kind="rspace", nx=190, ny=161, nz=133, bits=64, nbins=500),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "ensemble", "ift", "dft", "stats", "sample", "rspace"])
    bits = rng.choice([32, 32, 64])
    if kind == "rspace":
        nx, ny, nz = (2 * int(math.exp(rng.uniform(math.log(8), math.log(160)))) + rng.randrange(2) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, bits=bits, nbins=rng.randrange(16, 2049))
    interp = dict(neighbours=rng.randrange(1, 6), smoothness=rng.randrange(3))
    tracers = int(math.exp(rng.uniform(math.log(3), math.log(500000)))) | 1
    if kind == "ensemble":
        return dict(kind=kind, m32=rng.randrange(1, 33), m64=rng.randrange(1, 13), m128=rng.randrange(1, 7),
                    steps=rng.randrange(3, 21), tracers=int(math.exp(rng.uniform(math.log(10), math.log(10000)))) | 1,
                    order=rng.randrange(1, 7), **interp)
    n = 2 ** rng.randrange(4, 9)
    if kind in ("ift", "dft"):
        return dict(kind=kind, n=n, bits=bits)
    dealias = rng.choice(["smooth", "two_thirds"])
    if kind == "stats":
        return dict(kind=kind, n=n, bits=bits, dealias=dealias)
    forcing = rng.choice(["none", "linear", "Kolmogorov"])
    if kind == "sample":
        return dict(kind=kind, n=n, bits=bits, dealias=dealias, forcing=forcing, tracers=tracers, **interp)
    return dict(kind=kind, n=n, bits=bits, dealias=dealias, forcing=forcing,
                steps=rng.randrange(1, {16: 65, 32: 49, 64: 49, 128: 25, 256: 9}[n]),
                tracers=rng.choice([0, tracers, tracers]), order=rng.randrange(1, 7), **interp)


# ---- inputs -------------------------------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _real(case):
    return torch.float32 if case["bits"] == 32 else torch.float64


def _complex(case):
    return torch.complex64 if case["bits"] == 32 else torch.complex128


class _Modes:
    """Wavenumbers of the [ky][kz][kx] half spectrum of an n^3 box of side 2 pi, in 64 bits."""

    def __init__(self, n, dealias="smooth"):
        self.n, self.smooth = n, dealias == "smooth"
        i = torch.arange(n, dtype=torch.float64, device=_device())
        k = torch.where(i <= n // 2, i, i - n)
        self.k = (i[: n // 2 + 1].view(1, 1, -1), k.view(-1, 1, 1), k.view(1, -1, 1))  # kx, ky, kz
        self.k2 = (self.k[0] ** 2 + self.k[1] ** 2) + self.k[2] ** 2
        self.kM = n // 2 - 1 if self.smooth else n // 3 - 1
        self.kM2 = float(self.kM * self.kM)
        self.safe = torch.where(self.k2 > 0, self.k2, torch.ones_like(self.k2))
        self.inside = self.k2 <= self.kM2

    def curl(self, a):
        kx, ky, kz = self.k
        return torch.stack([1j * (ky * a[2] - kz * a[1]), 1j * (kz * a[0] - kx * a[2]), 1j * (kx * a[1] - ky * a[0])])

    def divfree(self, a):
        t = sum(k * a[c] for c, k in enumerate(self.k)) / self.safe
        a = torch.stack([a[c] - t * k for c, k in enumerate(self.k)])
        a[:, 0, 0, 0] = 0
        return a

    def dealias(self, a):
        if self.smooth:
            return a * torch.exp(-36.0 * (self.k2 / self.kM2) ** 18)
        return a * (self.k2 < self.kM2)


def _vorticity(n, seed, dealias="smooth"):
    """Random solenoidal vorticity with E(k) ~ k^4 exp(-2 (k/k0)^2), energy 0.5, as 64-bit modes [c][ky][kz][kx]."""
    m = _Modes(n, dealias)
    g = _generator(seed)
    u = torch.stack([torch.fft.rfftn(torch.randn(n, n, n, dtype=torch.float64, device=_device(), generator=g))
                     for _ in range(3)])
    k0 = 4.0 if n >= 512 else 3.0
    u = m.divfree(u * (torch.sqrt(m.k2) * torch.exp(-((torch.sqrt(m.k2) / k0) ** 2)) * (m.k2 < m.kM2)))
    weight = torch.full_like(m.k[0], 2.0)
    weight[..., 0] = 1.0
    energy = 0.5 * float((weight * (u.real ** 2 + u.imag ** 2).sum(0)).sum())
    return m.curl(u) * math.sqrt(0.5 / energy)


def _layout(a, dtype):
    """[c][ky][kz][kx] modes in the engine's layout [ky][kz][kx][c], in its precision."""
    return a.permute(1, 2, 3, 0).to(dtype).contiguous()


def _positions(count, seed):
    r = torch.rand(count, 3, dtype=torch.float64, device=_device(), generator=_generator(seed + 1000003))
    return (r * (2 * math.pi)).cpu().numpy()


def _solver(case, seed, n=None):
    n = case["n"] if n is None else n
    fs = vorticity_equation(n, precision="single" if case.get("bits", 32) == 32 else "double",
                            dealias_type=_lib.TWO_THIRDS if case.get("dealias") == "two_thirds" else _lib.SMOOTH)
    fs.nu, fs.fk0, fs.fk1, fs.famplitude, fs.fmode = NU[n], 1.5, 3.0, 0.5, 2
    fs.forcing_type = case.get("forcing", "linear")
    return fs


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


def _member_seeds(case, seed):
    sizes = [32] * case["m32"] + [64] * case["m64"] + [128] * case["m128"]
    return [(n, seed * 1009 + i) for i, n in enumerate(sizes)]


def prepare(case, seed):
    kind, s = case["kind"], {"case": dict(case)}
    if kind == "rspace":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        s["field"] = torch.randn(nz, ny, 2 * (nx // 2 + 1), 3, dtype=_real(case), device="cuda",
                                 generator=_generator(seed))
        s["moments"] = torch.zeros(10, 4, dtype=torch.float64, device="cuda")
        s["hist"] = torch.zeros(case["nbins"], 4, dtype=torch.int64, device="cuda")
        return s
    if kind == "ensemble":
        s["ens"], s["members"], at = ensemble(), [], {32: 0, 64: 0, 128: 0}
        s["fields"] = {"w%d" % n: _pinned((case["m%d" % n], n, n, n // 2 + 1, 3), torch.complex64)
                       for n in (32, 64, 128)}
        s["pos"] = _pinned((case["m32"] + case["m64"] + case["m128"], case["tracers"], 3), torch.float64)
        for i, (n, sd) in enumerate(_member_seeds(case, seed)):
            fs = _solver(case, sd, n)
            fs.set_cvorticity(_layout(_vorticity(n, sd), torch.complex64).cpu().numpy())
            ps = particles_system(fs, _positions(case["tracers"], sd), case["neighbours"], case["smoothness"],
                                  case["order"])
            s["ens"].add(fs, DT[n], ps)
            s["members"].append((fs, ps, s["fields"]["w%d" % n][at[n]].data_ptr(), s["pos"][i].numpy()))
            at[n] += 1
        return s
    n = case["n"]
    fs = s["fs"] = _solver(case, seed)
    if kind == "ift":
        s["in"] = _layout(_vorticity(n, seed), _complex(case))
        s["out"] = torch.zeros(n, n, n + 2, 3, dtype=_real(case), device="cuda")
        return s
    if kind == "dft":
        s["in"] = torch.randn(n, n, n + 2, 3, dtype=_real(case), device="cuda", generator=_generator(seed))
        s["out"] = torch.zeros(n, n, n // 2 + 1, 3, dtype=_complex(case), device="cuda")
        return s
    # as a run starts: the field of a checkpoint, then the tracers
    fs.io_checkpoint_read(_layout(_vorticity(n, seed, case["dealias"]), _complex(case)).cpu().numpy())
    s["ps"] = None
    if case.get("tracers"):
        order = case.get("order", 1)
        s["ps"] = particles_system(fs, _positions(case["tracers"], seed), case["neighbours"], case["smoothness"], order)
    if kind == "run":
        s["out"] = {"vorticity": _pinned(fs.cshape, _complex(case))}
        if s["ps"] is not None:
            s["out"]["pos"] = _pinned((case["tracers"], 3), torch.float64)
            s["out"]["rhs"] = _pinned((case["order"], case["tracers"], 3), torch.float64)
            s["host"] = (s["out"]["pos"].numpy(), s["out"]["rhs"].numpy())
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "run":
        fs, ps, dt = s["fs"], s["ps"], DT[case["n"]]
        for _ in range(case["steps"]):
            if ps is not None:
                NSVEparticles_step(fs, ps, dt, 1)
            else:
                fs.step(dt, 1)
        check(lib().bfg_field_download(fs.handle, _lib.FIELD_VORTICITY, s["out"]["vorticity"].data_ptr()), fs.handle)
        if ps is not None:
            check(lib().bfg_particles_download(ps.handle, ptr(s["host"][0]), ptr(s["host"][1]), None), fs.handle)
        return s["out"]
    if kind == "ensemble":
        s["ens"].step(case["steps"])
        for fs, ps, field, pos in s["members"]:
            check(lib().bfg_field_download(fs.handle, _lib.FIELD_VORTICITY, field), fs.handle)
            check(lib().bfg_particles_download(ps.handle, ptr(pos), None, None), fs.handle)
        return dict(s["fields"], pos=s["pos"])
    if kind == "ift":
        check(lib().bfg_ift(s["fs"].handle, s["in"].data_ptr(), s["out"].data_ptr()), s["fs"].handle)
        return s["out"]
    if kind == "dft":
        check(lib().bfg_dft(s["fs"].handle, s["in"].data_ptr(), s["out"].data_ptr()), s["fs"].handle)
        return s["out"]
    if kind == "stats":
        st = s["fs"].do_stats(MAX_VELOCITY, MAX_VORTICITY, NBINS)
        # counts as numbers: a value next to a bin's edge may fall on either side of it
        return {f: (spec, mom, hist.astype(np.float64)) for f, (spec, mom, hist) in st.items()}
    if kind == "sample":
        s["fs"].velocity_rspace()
        velocity = s["ps"].sample_velocity()
        return {"velocity": velocity, "acceleration": s["ps"].sample_acceleration()}
    check(lib().bfg_rspace_stats_noalloc(s["field"].data_ptr(), case["nx"], case["ny"], case["nz"], case["bits"] // 8,
                                         4.0, case["nbins"], s["moments"].data_ptr(), s["hist"].data_ptr(),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"moments": s["moments"], "hist": s["hist"]}


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def _transforms(n, fields):
    """Operations of that many real transforms of n^3 points (5/2 n log2 n each)."""
    return fields * 2.5 * n ** 3 * 3 * math.log2(n)


def _step_work(n, bits, steps, tracers, neighbours, order):
    field = 3 * n * n * (n + 2) * bits // 8  # a complex 3-vector field
    # every step: the state in and out, the tracers' positions and rhs history in, positions and rhs out
    moved = steps * (2 * field + tracers * 24 * (order + 2))
    done = steps * (_transforms(n, 27) + tracers * 6 * (2 * neighbours + 2) ** 3)
    return moved, done, field


def work(case):
    kind = case["kind"]
    if kind == "rspace":
        points = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": points * 3 * case["bits"] // 8 + 320 + 32 * case["nbins"], "flops": points * 80}
    if kind == "ensemble":
        moved = done = 0
        for n in (32, 64, 128):
            m, d, field = _step_work(n, 32, case["steps"], case["tracers"], case["neighbours"], case["order"])
            moved += case["m%d" % n] * (m + field + 24 * case["tracers"])
            done += case["m%d" % n] * d
        return {"bytes": moved, "flops": done}
    n, bits = case["n"], case["bits"]
    if kind == "run":
        moved, done, field = _step_work(n, bits, case["steps"], case["tracers"], case["neighbours"], case["order"])
        return {"bytes": moved + field + 24 * case["tracers"] * (1 + case["order"]), "flops": done}
    field = 3 * n * n * (n + 2) * bits // 8
    if kind in ("ift", "dft"):
        return {"bytes": 2 * field, "flops": _transforms(n, 3)}
    if kind == "stats":  # the vorticity in; two inverse transforms, 80 operations a point and field
        return {"bytes": field, "flops": _transforms(n, 6) + 160 * n ** 3}
    # sample: the vorticity in, two samples of the tracers out; u, the six products and the acceleration transformed
    return {"bytes": field + case["tracers"] * 72,
            "flops": _transforms(n, 12) + case["tracers"] * 12 * (2 * case["neighbours"] + 2) ** 3}


def tolerance(case):
    """About four times the distance from 64-bit arithmetic that was measured at the listed cases and over draws
    (runs: 1.9e-6 in 32 bits, 4e-15 in 64; transforms 1.8e-7; statistics and samples 4.8e-6)."""
    kind = case["kind"]
    if kind == "rspace":
        return {"rel": 1e-13, "max": 1e-12}
    if kind != "ensemble" and case["bits"] == 64:
        return {"rel": 3e-14, "max": 3e-12}
    if kind in ("ift", "dft"):
        return {"rel": 1e-6, "max": 1e-5}
    if kind in ("stats", "sample"):
        return {"rel": 2e-5, "max": 1e-4}
    return {"rel": 1e-5, "max": 1e-4}


# ---- the same in 64 bits, by plain torch --------------------------------------------------------------------------

def _to_real(a):
    """Unnormalised inverse transform of [c][ky][kz][kx] to [c][y][z][x]."""
    n = a.shape[1]
    return torch.stack([torch.fft.irfft(torch.fft.ifft2(f, dim=(0, 1), norm="forward"), n=n, dim=2, norm="forward")
                        for f in a])


def _to_modes(r):
    return torch.stack([torch.fft.fft2(torch.fft.rfft(f, dim=2), dim=(0, 1)) for f in r])


def _symmetrize(a):
    """The kx = 0 plane made Hermitian, rows ky > n/2 (and kz > n/2 on ky = 0) from their mirror images."""
    n = a.shape[1]
    p = a[:, :, :, 0]
    flip = (-torch.arange(n, device=a.device)) % n
    mirror = p[:, flip][:, :, flip].conj()
    q = p.clone()
    q[:, n // 2 + 1:] = mirror[:, n // 2 + 1:]
    q[:, 0, n // 2 + 1:] = mirror[:, 0, n // 2 + 1:]
    q[:, 0, 0] = q[:, 0, 0].real.to(a.dtype)
    a = a.clone()
    a[:, :, :, 0] = q
    return a


class _Flow:
    """The vorticity equation in 64 bits: third-order integrating-factor Runge-Kutta steps of the modes w."""

    def __init__(self, case, w, n):
        self.case, self.n, self.m = case, n, _Modes(n, case.get("dealias", "smooth"))
        self.w, self.dt, self.nu = w, DT[n], NU[n]
        k = torch.sqrt(self.m.k2)
        self.band = (k >= 1.5) & (k <= 3.0)
        self.forcing = case.get("forcing", "linear")

    def velocity(self, w):
        m = self.m
        return _symmetrize(m.curl(w) / m.safe * (m.inside & (m.k2 > 0)))

    def nonlinear(self, w):
        u, o = _to_real(self.velocity(w)), _to_real(w)
        p = torch.stack([u[(c + 1) % 3] * o[(c + 2) % 3] - u[(c + 2) % 3] * o[(c + 1) % 3] for c in range(3)])
        t = self.m.curl(self.m.dealias(_to_modes(p / self.n ** 3)))
        if self.forcing == "linear":
            t = t + 0.5 * w * self.band
        elif self.forcing == "Kolmogorov":
            t[2, 2, 0, 0] -= 0.25
            t[2, self.n - 2, 0, 0] -= 0.25
        return self.m.divfree(t)

    def step(self):
        m, dt, v0 = self.m, self.dt, self.w
        full = torch.exp(-self.nu * m.k2 * dt)
        half = torch.exp(-self.nu * m.k2 * dt / 2)
        v1 = (v0 + dt * self.nonlinear(v0)) * full * m.inside
        v2 = (3 * v0 * half + (v1 + dt * self.nonlinear(v1)) / half) * 0.25 * m.inside
        v3 = (v0 * half + 2 * (v2 + dt * self.nonlinear(v2))) * half / 3
        self.w = _symmetrize(m.divfree(torch.where(m.inside, v3, v0)))

    def acceleration(self):
        m = self.m
        u = self.velocity(self.w)
        r = _to_real(u)
        k = m.k
        g = m.dealias(_to_modes(r * r))
        p = -sum(k[c] * k[c] * g[c] for c in range(3))
        g = m.dealias(_to_modes(torch.stack([r[c] * r[(c + 1) % 3] for c in range(3)])))
        p = p - 2 * sum(k[c] * k[(c + 1) % 3] * g[c] for c in range(3))
        p = p / (self.n ** 3 * m.safe) * (m.inside & (m.k2 > 0))
        a = -self.nu * m.k2 * u
        if self.forcing == "linear":
            a = a + 0.5 * u * self.band
        return torch.stack([a[c] - 1j * k[c] * p for c in range(3)]) * m.inside


def _weight_polynomials(n, m):
    """Coefficients (increasing powers) of the 2n+2 interpolation weights: Lagrange (m = 0), or the Hermite
    polynomials of degree 2m+1 with centred differences over 2n+1 nodes for the derivatives."""
    def lagrange(nodes):
        out = []
        for j in nodes:
            p = [Fraction(1)]
            for k in nodes:
                if k != j:
                    p = [Fraction(a) / (j - k) for a in
                         [x - k * y for x, y in zip([Fraction(0)] + p, p + [Fraction(0)])]]
            out.append(p)
        return out

    if m == 0:
        return [[float(a) for a in p] for p in lagrange(range(-n, n + 2))]
    at0 = {1: [[1, 0, -3, 2], [0, 1, -2, 1]],
           2: [[1, 0, 0, -10, 15, -6], [0, 1, 0, -6, 8, -3],
               [0, 0, Fraction(1, 2), Fraction(-3, 2), Fraction(3, 2), Fraction(-1, 2)]]}[m]
    at1 = []  # (-1)^d times the polynomial of 1 - x
    for d, p in enumerate(at0):
        q = [Fraction(0)] * len(p)
        for i, a in enumerate(p):
            for j in range(i + 1):
                q[j] += (-1) ** d * Fraction(a) * math.comb(i, j) * (-1) ** j
        at1.append(q)
    rows = [[Fraction(0)] * (2 * m + 2) for _ in range(2 * n + 2)]
    basis = lagrange(range(-n, n + 1))
    for d in range(m + 1):
        for j in range(2 * n + 1):
            c = (Fraction(int(j == n)) if d == 0 else basis[j][d] * math.factorial(d))
            rows[j] = [a + c * b for a, b in zip(rows[j], at0[d])]
            rows[j + 1] = [a + c * b for a, b in zip(rows[j + 1], at1[d])]
    return [[float(a) for a in p] for p in rows]


def _interpolate(r, pos, neighbours, smoothness):
    """The field r [c][y][z][x] at the positions (count, 3)."""
    n = r.shape[1]
    h = 2 * math.pi / n
    flat = r.permute(2, 1, 3, 0).reshape(-1, 3)  # [z][y][x]
    polys = _weight_polynomials(neighbours, smoothness)
    out = []
    for p in pos.split(500000):
        cell = torch.floor(p / h)
        frac = (p - cell * h) / h
        weights = []
        for c in polys:
            v = torch.zeros_like(frac)
            for a in reversed(c):
                v = v * frac + a
            weights.append(v)
        weights = torch.stack(weights)  # (2n+2, count, 3)
        grid = torch.stack([(cell.long() - neighbours + i) % n for i in range(len(polys))])
        total = torch.zeros_like(p)
        for z in range(len(polys)):
            for y in range(len(polys)):
                row = (grid[z, :, 2] * n + grid[y, :, 1]) * n
                line = (flat[row[:, None] + grid[:, :, 0].T] * weights[:, :, 0].T[..., None]).sum(1)
                total += (weights[z, :, 2] * weights[y, :, 1])[:, None] * line
        out.append(total)
    return torch.cat(out)


_ADAMS = {1: [1], 2: [3 / 2, -1 / 2], 3: [23 / 12, -16 / 12, 5 / 12], 4: [55 / 24, -59 / 24, 37 / 24, -9 / 24],
          5: [v / 720 for v in (1901, -2774, 2616, -1274, 251)],
          6: [v / 1440 for v in (4277, -7923, 9982, -7298, 2877, -475)]}


def _advance(flow, case, pos, steps):
    """`steps` NSVEparticles steps: positions and rhs history (newest first, slot 0 empty) after them."""
    order = case["order"]
    rhs = [torch.zeros_like(pos) for _ in range(order)] if pos is not None else []
    for i in range(steps):
        if pos is not None:
            rhs[0] = _interpolate(_to_real(flow.velocity(flow.w)), pos, case["neighbours"], case["smoothness"])
            pos = pos + flow.dt * sum(a * r for a, r in zip(_ADAMS[min(i + 1, order)], rhs))
            rhs = [torch.zeros_like(pos)] + rhs[:-1]
        flow.step()
    return pos, torch.stack(rhs) if rhs else None


def _moments(v, estimates, nbins):
    """min, <v^1..8>, max (10, 4) and histogram (nbins, 4) of three components and the magnitude; v is (points, 3)."""
    v = torch.cat([v, torch.sqrt((v[:, 0] ** 2 + v[:, 1] ** 2) + v[:, 2] ** 2)[:, None]], 1)
    e = torch.tensor(estimates, dtype=torch.float64, device=v.device)
    low, high = torch.zeros_like(e), torch.zeros_like(e)
    low[3] = e[3]
    rows = [torch.minimum(low, v.amin(0))] + [(v ** k).mean(0) for k in range(1, 9)]
    rows.append(torch.maximum(high, v.amax(0)))
    hist = torch.zeros(nbins, 4, dtype=torch.int64, device=v.device)
    for i in range(4):
        size = 2 * estimates[i] / nbins
        b = torch.floor(v[:, 3] * 2 / size if i == 3 else (v[:, i] + estimates[i]) / size).long()
        hist[:, i] = torch.bincount(b[(b >= 0) & (b < nbins)], minlength=nbins)
    return torch.stack(rows), hist


def _field_stats(m, a, estimate):
    k = torch.sqrt(m.k2)
    shells = m.kM + 2
    shell = k.long()[m.inside]
    weight = torch.full_like(m.k[0], 2.0)
    weight[..., 0] = 1.0
    weight = weight.expand_as(m.k2)[m.inside]
    spec = torch.zeros(shells, 3, 3, dtype=torch.float64, device=a.device)
    for i in range(3):
        for j in range(3):
            v = weight * (a[i].real * a[j].real + a[i].imag * a[j].imag)[m.inside]
            spec[:, i, j] = torch.bincount(shell, weights=v, minlength=shells)[:shells]
    mom, hist = _moments(_to_real(a).reshape(3, -1).T, [estimate] * 3 + [estimate * math.sqrt(3.0)], NBINS)
    return spec.cpu(), mom.cpu(), hist.double().cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind == "rspace":
        f = torch.randn(case["nz"], case["ny"], 2 * (case["nx"] // 2 + 1), 3, dtype=_real(case), device=_device(),
                        generator=_generator(seed))
        mom, hist = _moments(f[:, :, : case["nx"]].reshape(-1, 3).double(), [4.0] * 3 + [4.0 * math.sqrt(3.0)],
                             case["nbins"])
        return {"moments": mom, "hist": hist}
    if kind == "ensemble":
        out, where = {"w32": [], "w64": [], "w128": []}, []
        for n, sd in _member_seeds(case, seed):
            flow = _Flow(case, _vorticity(n, sd).to(torch.complex64).to(torch.complex128), n)
            pos, _ = _advance(flow, case, torch.from_numpy(_positions(case["tracers"], sd)).to(_device()),
                              case["steps"])
            out["w%d" % n].append(_layout(flow.w, torch.complex128).cpu())
            where.append(pos.cpu())
        return dict({f: torch.stack(v) for f, v in out.items()}, pos=torch.stack(where))
    n = case["n"]
    if kind == "ift":
        r = _to_real(_vorticity(n, seed).to(_complex(case)).to(torch.complex128))
        return torch.nn.functional.pad(r.permute(2, 1, 3, 0), (0, 0, 0, 2))
    if kind == "dft":
        r = torch.randn(n, n, n + 2, 3, dtype=_real(case), device=_device(), generator=_generator(seed))
        return _layout(_to_modes(r[:, :, :n].double().permute(3, 1, 0, 2).contiguous()), torch.complex128)
    w = _symmetrize(_vorticity(n, seed, case["dealias"]).to(_complex(case)).to(torch.complex128))
    m = _Modes(n, case["dealias"])
    w = m.divfree(w * (m.k2 < m.kM2))
    flow = _Flow(case, w, n)
    if kind == "stats":
        return {"vorticity": _field_stats(m, w, MAX_VORTICITY / math.sqrt(3.0)),
                "velocity": _field_stats(m, flow.velocity(w), MAX_VELOCITY / math.sqrt(3.0))}
    pos = torch.from_numpy(_positions(case["tracers"], seed)).to(_device()) if case["tracers"] else None
    if kind == "sample":
        at = (pos, case["neighbours"], case["smoothness"])
        return {"velocity": _interpolate(_to_real(flow.velocity(w)), *at).cpu(),
                "acceleration": _interpolate(_to_real(flow.acceleration()), *at).cpu()}
    pos, rhs = _advance(flow, case, pos, case["steps"])
    out = {"vorticity": _layout(flow.w, torch.complex128).cpu()}
    if pos is not None:
        out["pos"], out["rhs"] = pos.cpu(), rhs.cpu()
    return out
