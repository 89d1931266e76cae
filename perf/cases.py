"""Performance cases of the solver: what a user's program has it do, over the range it is used in.

Each case runs a box through the public Python interface (spns_b200.hit): time steps of DNS
and LES boxes in both precisions, ensembles, the energy spectrum and the velocity-gradient
spectra.  Inputs are synthetic: solenoidal Gaussian fields with a developed (von Karman)
spectrum and energy in every retained mode, made from the seed alone.

`exact` restates the step on the padded FFT grid with torch.fft in 64 bits: advective
nonlinear term with 3/2-rule padding, Smagorinsky stress, rotation, constant-power and
spectrum forcing, Adams-Bashforth and the self-adaptive one-leg scheme.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from spns_b200 import hit
from spns_b200.params import HitArgs

# FFT grid sizes of the solver (M; the retained modes per axis are N <= 2 M / 3)
LENGTHS = (48, 72, 96, 144, 192, 288, 384, 768)

# One box: what a case holds unless it says otherwise.  nx, ny, nz are the retained modes of
# the true grid, mx, my, mz its FFT sizes, lx, ly, lz the wavenumber steps of a non-cubic box.
BOX = dict(kind="step", prec=64, les=0.0, adv=False, kappa=False, eps=0.0, fixed_dt=0.0, omega=0.0, nu=1e-3, c_at=0.5,
           lx=1, ly=1, lz=1, steps=1, tune=False)


def _box(n, **more):
    n = (n, n, n) if isinstance(n, int) else n
    c = dict(BOX, nx=n[0], ny=n[1], nz=n[2], mx=3 * n[0] // 2, my=3 * n[1] // 2, mz=3 * n[2] // 2)
    c.update(more)
    return c


def listed():
    return [
        # Plain decaying DNS, 64^3, fixed dt, one step a call and the time read back after it, as the
        # driver's loop does: launches and host latency count.
        dict(_box(64, kind="driver", nu=1e-2, fixed_dt=1e-3), name="dns_64_f64_driver"),
        # The smallest served run: a chunk of 25 asynchronous steps of an LES box with tuned launch shapes.
        dict(_box(32, prec=32, les=0.16, nu=1e-4, steps=25, tune=True), name="les_32_f32_chunk"),
        # Spectrum-forced LES as in the decaying-grid-turbulence setup: step, then E(K) set on the given shells.
        dict(_box(64, kind="forced", les=0.16, nu=7.787e-4), name="les_64_f64_spectrum_forced"),
        # Boxes with odd and unequal mode counts in the advective form, self-adaptive step, rotating frame.
        dict(_box((95, 64, 121), mx=144, my=96, mz=192, adv=True, kappa=True, omega=1.0), name="dns_95x64x121_f64_advective"),
        # Rotating LES on a non-cubic box.
        dict(_box(128, lz=2, prec=32, les=0.17, omega=1.0, nu=1e-4), name="les_noncubic_128_f32"),
        # The large sizes of the served mix, and the LES in the plain double-precision form.
        dict(_box(256, prec=32, nu=2e-3), name="dns_256_f32"),
        dict(_box(256, prec=32, les=0.15, nu=5e-4), name="les_256_f32"),
        dict(_box(256, les=0.15, nu=5e-4), name="les_256_f64"),
        # The batched workload: 64 independent LES boxes of 32..96 modes, one step of each.
        dict(kind="ensemble", boxes=64, lo=32, hi=96, prec=32, name="ensemble_64_les_f32"),
        # The headline workload: forced DNS, 512^3, self-adaptive step, in both precisions.
        dict(_box(512, kappa=True, eps=0.1, nu=4.9e-4), name="dns_512_f64_forced"),
        dict(_box(512, prec=32, kappa=True, eps=0.1, nu=4.9e-4), name="dns_512_f32_forced"),
        # Post-processing: spectra of the velocity-gradient invariants.
        dict(_box(128, kind="invariants"), name="invariants_128_f64"),
    ]


def _axis(rng, cap):
    """A grid size up to `cap` and a mode count that goes with it: 2/3 of it, or a few less (odd ones among them)."""
    m = rng.choice([v for v in LENGTHS if v <= cap])
    n = 2 * m // 3
    return (n if rng.random() < 0.6 else n - rng.randint(1, n // 4)), m


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["driver", "forced", "ensemble", "invariants", "spectrum"])
    if kind == "ensemble":
        return dict(kind=kind, boxes=rng.randint(4, 60), lo=32, hi=rng.choice([48, 64, 96]), prec=rng.choice([32, 32, 64]))
    prec = 64 if kind in ("driver", "forced", "invariants", "spectrum") else rng.choice([32, 64])
    les = rng.uniform(0.1, 0.2) if kind == "forced" or (kind == "step" and rng.random() < 0.5) else 0.0
    cap = 192 if kind in ("driver", "forced", "invariants") else 384 if les or kind == "spectrum" else 768
    top = rng.choice([v for v in LENGTHS if v <= cap])
    if rng.random() < 0.5:   # a cubic box
        n, m = _axis(rng, top)
        n, m = (n, n, n), (m, m, m)
    else:
        n, m = zip(*(_axis(rng, top) for _ in range(3)))
    points = m[0] * m[1] * m[2]
    more = dict(mx=m[0], my=m[1], mz=m[2], kind=kind, prec=prec, les=round(les, 3), nu=round(10 ** rng.uniform(-4, -2), 6))
    if kind == "step":
        more["kappa"] = rng.random() < 0.4
        more["adv"] = not les and rng.random() < 0.2 and points <= 384 ** 3
        more["eps"] = 0.1 if rng.random() < 0.3 else 0.0
        more["omega"] = rng.choice([0.0, 0.0, 1.0])
        more["lz"] = rng.choice([1, 1, 1, 2])
        more["steps"] = rng.randint(2, 25) if points <= 96 ** 3 else 1
        more["tune"] = points <= 192 ** 3 and rng.random() < 0.5
    return _box(n, **more)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _boxes(case, seed):
    """The boxes of a case, each with a seed of its own."""
    if case["kind"] != "ensemble":
        return [(case, seed)]
    r = np.random.default_rng([seed, 5])
    sizes = [n for n in (32, 48, 64, 96) if case["lo"] <= n <= case["hi"]]
    # the same grids for every seed, so that passes on several inputs are the same work
    grids = [sizes[i % len(sizes)] for i in range(case["boxes"])]
    return [(_box(n, prec=case["prec"], les=float(r.uniform(0.10, 0.20)), nu=1e-4, tune=True), seed * 1009 + 17 * i) for i, n in enumerate(grids)]


def _modes(case, device="cuda"):
    """Wavenumbers ky, kx, kz of the compact layout [ky][kx][kz], shaped to broadcast."""
    def full(n, s):
        h = n // 2
        i = torch.arange(2 * h + 1, device=device, dtype=torch.float64)
        return s * torch.where(i <= h, i, i - (2 * h + 1))
    kz = case["lz"] * torch.arange(case["nz"] // 2 + 1, device=device, dtype=torch.float64)
    return full(case["ny"], case["ly"])[:, None, None], full(case["nx"], case["lx"])[None, :, None], kz[None, None, :]


def _field(case, seed):
    """Solenoidal Gaussian field, energy spectrum k^4 / (k^2 + k0^2)^(17/6) with a viscous tail, u_rms = 1."""
    ky, kx, kz = _modes(case)
    k2 = ky * ky + kx * kx + kz * kz
    shape = (3,) + tuple(k2.shape)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    u = torch.empty(shape, device="cuda", dtype=torch.complex128)
    for c in range(3):
        u[c] = torch.complex(torch.randn(shape[1:], device="cuda", dtype=torch.float64, generator=g),
                             torch.randn(shape[1:], device="cuda", dtype=torch.float64, generator=g))
    safe = torch.where(k2 > 0, k2, torch.ones_like(k2))
    kmax = max(case["nx"] * case["lx"], case["ny"] * case["ly"], case["nz"] * case["lz"]) / 2.0
    amp = torch.where(k2 > 0, k2.sqrt() / (k2 + 9.0) ** (17.0 / 12.0) * torch.exp(-3.0 * k2.sqrt() / kmax), torch.zeros_like(k2))
    for c in range(3):
        u[c] *= amp
    d = (kx * u[0] + ky * u[1] + kz * u[2]) / safe
    for c, k in enumerate((kx, ky, kz)):
        u[c] -= d * k
    # Hermitian kz = 0 plane: u(-kx, -ky) = conj u(kx, ky)
    p = u[:, :, :, 0].clone()
    q = torch.roll(torch.flip(p, (1, 2)), (1, 1), (1, 2))
    u[:, :, :, 0] = 0.5 * (p + q.conj())
    e = u.real.square().sum() + u.imag.square().sum()
    e0 = u[:, :, :, 0].real.square().sum() + u[:, :, :, 0].imag.square().sum()
    u *= torch.sqrt(3.0 / (2.0 * e - e0))
    return u if case["prec"] == 64 else u.to(torch.complex64)


def _target(case):
    """The spectrum that a spectrum-forced run is held to, on the shells the box resolves."""
    k = np.arange(min(case["nx"], case["ny"], case["nz"]) // 2 + 1, dtype=np.float64)
    return 0.2 * k ** 4 / (k * k + 9.0) ** (17.0 / 6.0)


# ---------------------------------------------------------------------------
# The solver's side
# ---------------------------------------------------------------------------
class _State:
    """The device-resident spectral state of a box as a tensor [3][ky][kx][kz] (no copy)."""

    def __init__(self, box, ptr):
        self.box = box
        self.__cuda_array_interface__ = {"shape": tuple(box.spectral_shape), "typestr": "<c16" if box.precision == hit.SPNS_FP64 else "<c8",
                                         "data": (ptr, False), "version": 2}


def _state(s):
    """The box's current state; the self-adaptive scheme alternates between two buffers."""
    p = ctypes.c_void_p()
    hit.lib().spns_device_state(s["box"]._h, ctypes.byref(p), None, None)
    if p.value not in s["views"]:
        s["views"][p.value] = torch.as_tensor(_State(s["box"], p.value), device="cuda")
    return s["views"][p.value]


def _make(case, seed):
    n = [case["n" + a] for a in "xyz"]
    m = [case["m" + a] for a in "xyz"]
    f = [case["l" + a] for a in "xyz"]
    ex = [v * k if v % 2 == 0 else (v - 1) * k + 1 for v, k in zip(n, f)]
    em = [v * k for v, k in zip(m, f)]
    args = HitArgs(Nx=ex[0], Ny=ex[1], Nz=ex[2], Mx=em[0], My=em[1], Mz=em[2], nu=case["nu"], C_Smag=case["les"], C_At=case["c_at"],
                   Lx=f[0], Ly=f[1], Lz=f[2], omega_x=0.0, omega_y=0.0, omega_z=case["omega"], Nx_file=-1, Ny_file=-1, Nz_file=-1,
                   isReLambda=False, isInitialFieldFromBinaryFile=False, isInitialFieldFromASCIIFile=False, isNotCubic=max(f) > 1,
                   isRotating=case["omega"] != 0.0, isLES=case["les"] > 0, isComplexConjugateCorrected=False, isSelfAdaptive=case["kappa"])
    box = hit.HIT(args, precision=hit.SPNS_FP64 if case["prec"] == 64 else hit.SPNS_FP32_HILO, k41_ranks=-1, fixed_dt=case["fixed_dt"],
                  eps_forcing=case["eps"], nonlinear_form=2 if case["adv"] else 0)
    s = {"box": box, "views": {}}
    _state(s).copy_(_field(case, seed))
    torch.cuda.synchronize()
    box.Recalculate_Velocity_Antitransform()
    box.Recalculate_TimeStep()
    if case["tune"]:
        box.autotune(steps=2)
    box.synchronize()
    return s


def prepare(case, seed):
    s = {"case": case, "boxes": [_make(c, d) for c, d in _boxes(case, seed)], "target": None}
    if case["kind"] == "ensemble":
        s["ensemble"] = hit.Ensemble([b["box"] for b in s["boxes"]])
    if case["kind"] == "forced":
        s["target"] = _target(case)
    torch.cuda.empty_cache()
    return s


def run(s):
    case, b = s["case"], s["boxes"][0]
    box, kind = b["box"], case["kind"]
    if kind == "ensemble":
        s["ensemble"].step(1)
        return [_state(x) for x in s["boxes"]]
    if kind == "spectrum":
        return box.Recalculate_Energy_Cascade()
    if kind == "invariants":
        return box.Recalculate_Invariants_Distribution()
    if kind == "forced":
        box.New_Fractional_Step_Method()
        box.Forcing_Energy_Cascade(s["target"], len(s["target"]) - 1, False)
        return _state(b)
    if kind == "driver":
        box.New_Fractional_Step_Method()
        return {"time": box.gettime(), "state": _state(b)}
    if case["steps"] > 1:
        box.step_async(case["steps"])
        box.synchronize()
    else:
        box.New_Fractional_Step_Method()
    return _state(b)


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    total = {"bytes": 0.0, "flops": 0.0}
    for c, _ in _boxes(case, 0):
        modes = (2 * (c["nx"] // 2) + 1) * (2 * (c["ny"] // 2) + 1) * (c["nz"] // 2 + 1)
        points = c["mx"] * c["my"] * c["mz"]
        word = 16 if c["prec"] == 64 else 8
        fft = 2.5 * points * math.log2(points)      # one real 3-D transform
        steps = c["steps"]
        if c["kind"] == "spectrum":
            total["bytes"] += 3 * modes * word
            total["flops"] += 12 * modes
            continue
        if c["kind"] == "invariants":
            total["bytes"] += 3 * modes * word
            total["flops"] += 14 * fft
            continue
        # u^n and R^{n-1} read, u^{n+1} and R^n written, u^{n-1} read by the self-adaptive scheme;
        # the compensated single-precision state is a pair
        state = (2 if c["prec"] == 64 else 4) + (0 if not c["kappa"] else 1 if c["prec"] == 64 else 2)
        total["bytes"] += steps * 3 * modes * word * (state + 2)
        # 12 (advective, LES) or 6 (rotational) inverse transforms, 3 forward and 6 of the stress
        total["flops"] += steps * fft * (21 if c["les"] else 15 if c["adv"] else 9)
        if c["kind"] == "forced":
            total["bytes"] += 3 * modes * word * 3
    return total


# ---------------------------------------------------------------------------
# The same results in 64 bits, by torch.fft
# ---------------------------------------------------------------------------
class _Exact:
    def __init__(self, case):
        self.c = c = case
        self.k = dict(zip("yxz", _modes(c)))
        self.k2 = self.k["x"] ** 2 + self.k["y"] ** 2 + self.k["z"] ** 2
        self.M = (c["my"], c["mx"], c["mz"])
        self.h = (c["ny"] // 2, c["nx"] // 2, c["nz"] // 2)
        self.A = {a: 2 * math.pi / c["m" + a] / c["l" + a] for a in "xyz"}

    def grid(self, f):
        (hy, hx, hz), (My, Mx, Mz) = self.h, self.M
        p = torch.zeros((My, Mx, Mz // 2 + 1), device=f.device, dtype=torch.complex128)
        for dy, sy in ((slice(0, hy + 1), slice(0, hy + 1)), (slice(My - hy, My), slice(hy + 1, 2 * hy + 1))):
            for dx, sx in ((slice(0, hx + 1), slice(0, hx + 1)), (slice(Mx - hx, Mx), slice(hx + 1, 2 * hx + 1))):
                p[dy, dx, :hz + 1] = f[sy, sx]
        p = torch.fft.ifftn(p, dim=(0, 1), norm="forward")
        return torch.fft.irfft(p, n=Mz, dim=2, norm="forward")

    def modes(self, q):
        (hy, hx, hz), (My, Mx, Mz) = self.h, self.M
        p = torch.fft.rfft(q, dim=2, norm="forward")[:, :, :hz + 1]
        p = torch.fft.fftn(p, dim=(0, 1), norm="forward")
        p = torch.cat((p[:hy + 1], p[My - hy:]), 0)
        return torch.cat((p[:, :hx + 1], p[:, Mx - hx:]), 1)

    def d(self, f, a):
        return self.grid(1j * self.k[a] * f)

    def time_step(self, v):
        """Step size and scheme parameter from the grid velocity."""
        c = self.c
        if c["fixed_dt"] > 0:
            return c["fixed_dt"], 0.5
        A = [self.A[a] for a in "xyz"]
        if not c["kappa"]:
            top = max(float(v[i].abs().max()) / A[i] for i in range(3))
            return c["c_at"] * min(0.2 * min(a * a for a in A) / c["nu"], 0.35 / top), 0.5
        top = float((v[0].abs() / A[0] + v[1].abs() / A[1] + v[2].abs() / A[2]).max())
        Ah, nu, half = sum(A) / 3.0, c["nu"], math.pi / 2
        phi = math.atan(top * Ah * Ah / (0.35 * nu * 12.0))
        p = (math.atan(164.0 / 99.0), math.pi / 3.0, math.pi * 9.0 / 25.0)

        def arc(q, x0, x1, f0, f1):
            return (q[0] * phi * phi + q[1] * phi + q[2]) * (phi - x0) * (phi - x1) + f0 + (phi - x0) * (f1 - f0) / (x1 - x0)
        t = (arc((0.0, 0.0647998, -0.386022), 0.0, p[0], 4.0 / 3.0, 0.9302468) if phi < p[0]
             else arc((3.72945, -9.38143, 7.06574), p[0], half, 0.9302468, 1.0))
        k1, k2 = 0.73782212, 0.44660387
        kap = (1.0 if phi <= p[0] else arc((2403400.0, -5018490.0, 2620140.0), p[0], p[1], 1.0, k1) if phi <= p[1]
               else arc((2945.0, -6665.76, 3790.54), p[1], p[2], k1, k2) if phi <= p[2]
               else arc((4.80513, -16.9473, 15.0155), p[2], half, k2, 0.0))
        return c["c_at"] * t / math.sqrt(top * top / 0.35 ** 2 + 144.0 * nu * nu / Ah ** 4), kap

    def shells(self):
        K = self.k2.sqrt().round().to(torch.int64)
        w = torch.where(torch.arange(self.k2.shape[2], device=self.k2.device) > 0, 2.0, 1.0).to(torch.float64).expand(self.k2.shape)
        return K, w

    def last_shell(self):
        c = self.c
        n = [(c["n" + a] if c["n" + a] % 2 == 0 else c["n" + a] - 1) * c["l" + a] + c["n" + a] % 2 for a in "xyz"]
        return int(math.ceil(math.sqrt(sum(float(v // 2) ** 2 for v in n))))

    def spectrum(self, e):
        K, w = self.shells()
        n = self.last_shell() + 1
        keep = K < n
        return torch.zeros(n, device=e.device, dtype=torch.float64).index_add_(0, K[keep], (w * e)[keep])

    def energy(self, u):
        return self.spectrum(0.5 * (u.real.square() + u.imag.square()).sum(0))

    def nonlinear(self, u, v):
        """Modes of u_j d_j u_i [+ d_j tau_ij], zero at k = 0."""
        c, out = self.c, []
        les = c["les"] > 0
        strain = {}
        for i in range(3):
            conv = torch.zeros_like(v[0])
            for j, a in enumerate("xyz"):
                g = self.d(u[i], a)
                conv += v[j] * g
                if les:
                    key = (min(i, j), max(i, j))
                    strain[key] = strain[key] + g if key in strain else g
                del g
            out.append(self.modes(conv))
            del conv
        if les:
            mx = [c["m" + a] * c["l" + a] for a in "xyz"]
            delta = 2.0 * math.pi / float(mx[0] * mx[1] * mx[2]) ** (1.0 / 3.0)
            nut = sum((2.0 if i == j else 1.0) * s * s for (i, j), s in strain.items()).sqrt_() * (c["les"] * delta) ** 2
            for (i, j), s in strain.items():
                t = self.modes((-2.0 if i == j else -1.0) * nut * s)
                out[i] += 1j * self.k["xyz"[j]] * t
                if i != j:
                    out[j] += 1j * self.k["xyz"[i]] * t
        for f in out:
            f[0, 0, 0] = 0.0
        return torch.stack(out)

    def step(self, n, u):
        c = self.c
        v = [self.grid(u[i]) for i in range(3)]
        dt, kap = self.time_step(v)
        old, R0, time = u, torch.zeros_like(u), 0.0
        K, _ = self.shells()
        for s in range(n):
            if s:
                v = [self.grid(u[i]) for i in range(3)]
            R = self.nonlinear(u, v).neg_()
            R -= c["nu"] * self.k2 * u
            if c["omega"]:
                R[0] += 2 * c["omega"] * u[1]
                R[1] -= 2 * c["omega"] * u[0]
            if c["eps"] > 0:
                e = self.energy(u)[1:3].sum()
                R += torch.where((K >= 1) & (K <= 2), c["eps"] / (2.0 * e), torch.zeros_like(e)) * u
                R[:, 0, 0, 0] = 0.0
            if c["kappa"]:
                new = (2.0 * kap * u + dt * ((1.0 + kap) * R - kap * R0) - (kap - 0.5) * old) / (kap + 0.5)
            else:
                new = u + dt * (1.5 * R - 0.5 * R0)
            div = (self.k["x"] * new[0] + self.k["y"] * new[1] + self.k["z"] * new[2]) / torch.where(self.k2 > 0, self.k2, torch.ones_like(self.k2))
            for i, a in enumerate("xyz"):
                new[i] -= div * self.k[a]
            old, u, R0 = u, new, R
            dt, kap = self.time_step(v)
            time += dt
        return u, time

    def forced(self, u, target):
        E = self.energy(u)
        last = min(len(target) - 1, (min(self.c["n" + a] for a in "xyz") - 1) // 2)
        f = torch.ones_like(E)
        T = torch.as_tensor(target[:last + 1], device=E.device)
        f[:last + 1] = torch.where(E[:last + 1] > 0, (T / E[:last + 1].clamp_min(1e-300)).sqrt(), torch.zeros_like(T))
        K, _ = self.shells()
        return u * f[K.clamp_max(len(E) - 1)]

    def invariants(self, u):
        G = [[self.d(u[i], a) for a in "xyz"] for i in range(3)]
        S = [[0.5 * (G[i][j] + G[j][i]) for j in range(3)] for i in range(3)]
        O = [[0.5 * (G[i][j] - G[j][i]) for j in range(3)] for i in range(3)]

        def mul(a, b):
            return [[sum(a[i][k] * b[k][j] for k in range(3)) for j in range(3)] for i in range(3)]

        def tr(a):
            return a[0][0] + a[1][1] + a[2][2]

        def det(t):
            return (t[0][0] * (t[1][1] * t[2][2] - t[1][2] * t[2][1]) - t[0][1] * (t[1][0] * t[2][2] - t[1][2] * t[2][0])
                    + t[0][2] * (t[1][0] * t[2][1] - t[1][1] * t[2][0]))
        QG, QS = 0.5 * (tr(G) ** 2 - tr(mul(G, G))), 0.5 * (tr(S) ** 2 - tr(mul(S, S)))
        V2 = 4.0 * (tr(mul(mul(S, S), mul(O, O))) - 2.0 * QS * (QG - QS))
        out = []
        for q in (QG, QS, det(G), det(S), V2):
            f = self.modes(q)
            out.append(self.spectrum(f.real.square() + f.imag.square()))
        return torch.stack(out)


def exact(case, seed):
    out = []
    for c, d in _boxes(case, seed):
        x = _Exact(c)
        u = _field(c, d).to(torch.complex128)
        if c["kind"] == "spectrum":
            out.append(x.energy(u).cpu().numpy())
        elif c["kind"] == "invariants":
            out.append(x.invariants(u).cpu().numpy())
        else:
            u, time = x.step(c["steps"], u)
            if c["kind"] == "forced":
                u = x.forced(u, _target(c))
            out.append({"time": time, "state": u} if c["kind"] == "driver" else u)
    return out if case["kind"] == "ensemble" else out[0]
