"""Measured cases of the TD step: what a program of this library's users has it do.

A case is one measurement block of a run (``TDRun.steps``, on small systems with the energies
that a driver prints after each block), or one optimal-control gradient (``TDRun.adjoint``).
The states, densities and potentials come back as the context's own device arrays, as programs
that keep their data on the GPU read them.

``exact`` restates the step in plain torch (complex128, cuFFT): the same functional, H, ABM and
density formulas, without the library.
"""
import ctypes
import math

import numpy as np
import torch

from wslda_b200 import FP64, MIXED_H32, MIXED_H64, TDRun
from wslda_b200.projects import Project

PRECISIONS = {"fp64": FP64, "h64": MIXED_H64, "h32": MIXED_H32}

# runtime parameters of the projects' hooks where they are not the project's own defaults: the
# td-gauss stirrer with the values its process_params makes of its inputs (amplitude, 1/(2 w^2)
# per axis, start, stop and ramp times)
GAUSS = {0: 0.25, 1: -0.125, 2: -0.125, 3: 0.0, 4: -3.0, 5: 1.0e6, 6: 4.0}
# the 14 stirrer parameters of the 2D optimal-control workload (path coefficients, A, w)
STIRRER = [0.55, 0.31, 0.72, 0.18, 0.44, 0.63, 0.27, 0.81, 0.39, 0.52, 0.66, 0.23, 0.48, 0.74]


def _case(name, project, precision, nwf, steps, energy=False, gradient=0):
    """gradient: checkpoint interval of a gradient call, 0 for a block of steps"""
    return {"name": name, "project": project, "precision": precision, "nwf": nwf, "steps": steps,
            "energy": energy, "gradient": gradient}


def listed():
    return [
        # the 1D ASLDA run of the td-gauss test family: 12 points, 312 plane-wave states with
        # (k_y, k_z) and degeneracies; a block with its energies. The smallest call: launches
        _case("1d-aslda-312", "gauss_aslda_1d", "fp64", 312, 10, energy=True),
        # the 1D BdG workload (128 points, 256 states): a block of a long small run
        _case("1d-bdg-256", "c1_bdg1d", "fp64", 256, 20),
        # the 3D BdG run of the td-gauss family (12^3, 895 states), a block with its energies
        _case("3d-bdg-12-895", "gauss_bdg_3d", "fp64", 895, 10, energy=True),
        # the same lattice with variable effective mass and currents, an odd share of the states
        _case("3d-aslda-12-447", "gauss_aslda_3d", "fp64", 447, 6, energy=True),
        # the 2D SLDA workload at its full state count, FP64 ...
        _case("2d-slda-64-8192", "c2_slda2d", "fp64", 8192, 3),
        # ... and in the FP32-mixed form with complex64 history
        _case("2d-slda-64-8192-h32", "c2_slda2d", "h32", 8192, 3),
        # a 2D lattice beyond one CTA with variable mass (160x96): a rank's share of the states
        _case("2d-aslda-160x96-301", "t2d_big", "fp64", 301, 3),
        # the optimal-control gradient of the 2D BdG workload: loss and 14 derivatives
        _case("2d-bdg-48-gradient", "c4_bdg2d", "fp64", 4608, 12, gradient=4),
        # the 3D ASLDA workload (32^3, gradients every half step): a rank's share of its 12,000
        # states in FP64, and more of them in the FP32-mixed form
        _case("3d-aslda-32-1500", "c3_aslda3d", "fp64", 1500, 2),
        _case("3d-aslda-32-3000-h32", "c3_aslda3d", "h32", 3000, 2),
        # the 3D SLDA vortex workload (48^3): a rank's share in FP64 and in the all-FP32 form
        _case("3d-slda-48-601", "c5_slda3d", "fp64", 601, 2),
        _case("3d-slda-48-1001-h32", "c5_slda3d", "h32", 1001, 2),
    ]


# what draw() takes from: project, precisions, states, steps, largest states x steps, with energies
_RANGES = [
    ("gauss_aslda_1d", ("fp64",), (40, 1500), (1, 12), 15000, True),
    ("c1_bdg1d", ("fp64", "h64", "h32"), (30, 3000), (1, 20), 60000, False),
    ("t2d_slda", ("fp64", "h32"), (24, 2000), (1, 10), 20000, True),
    ("gauss_bdg_3d", ("fp64", "h64"), (60, 3456), (1, 10), 20000, True),
    ("gauss_aslda_3d", ("fp64",), (60, 2000), (1, 6), 6000, True),
    ("c2_slda2d", ("fp64", "h64", "h32"), (40, 8192), (1, 4), 24576, False),
    ("c4_bdg2d", ("fp64", "h32"), (40, 4608), (1, 6), 24576, False),
    ("t2d_big", ("fp64", "h64"), (8, 600), (1, 3), 900, False),
    ("c3_aslda3d", ("fp64", "h64", "h32"), (8, 3000), (1, 3), 3000, False),
    ("c5_slda3d", ("fp64", "h64", "h32"), (4, 900), (1, 3), 1200, False),
]


def draw(rng):
    project, precisions, (lo, hi), (s0, s1), most, energy = rng.choice(_RANGES)
    nwf = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    steps = rng.randint(s0, s1)
    gradient = 0
    if project == "c4_bdg2d" and rng.random() < 0.5:
        gradient, steps = rng.randint(1, 4), rng.randint(2, 8)
    steps = max(1, min(steps, most // nwf))
    return {"project": project, "precision": "fp64" if gradient else rng.choice(precisions), "nwf": nwf, "steps": steps,
            "energy": energy and rng.random() < 0.5, "gradient": gradient}


def _params(name):
    p = Project(name).params
    for k, v in (GAUSS if name.startswith("gauss_") else {}).items():
        p[k] = v
    if name == "c4_bdg2d":
        p[:14] = STIRRER
    return p


def _inputs(case, seed):
    """states [2, S, N] in the form's storage type, occupations, and for 1D the plane-wave
    momenta and degeneracies"""
    proj = Project(case["project"])
    S, N = case["nwf"], proj.numel
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (seed % (1 << 30)) + S)
    dtype = torch.complex128 if case["precision"] == "fp64" else torch.complex64
    y = torch.empty((2, S, N), dtype=dtype, device="cuda")
    chunk = max(1, (1 << 24) // N)
    for a in range(0, S, chunk):
        b = min(S, a + chunk)
        z = torch.randn((2, b - a, N), dtype=torch.complex128, device="cuda", generator=g)
        z /= torch.linalg.vector_norm(z, dim=(0, 2), keepdim=True) * math.sqrt(proj.dv)
        y[:, a:b] = z
    rng = np.random.default_rng(seed)
    # occupations of a system at a small temperature: near 1 and near 0 with a smooth edge
    occ = 1.0 / (1.0 + np.exp((np.arange(S) - 0.5 * S) / (0.05 * S) + 0.3 * rng.standard_normal(S)))
    kky = kkz = cnt = None
    if case["project"] == "gauss_aslda_1d":
        dk = 2.0 * math.pi / (12 * 1.15)
        ny, nz = rng.integers(0, 4, S), rng.integers(0, 4, S)
        kky, kkz = dk * ny, dk * nz
        cnt = ((ny > 0) + 1) * ((nz > 0) + 1)
    return proj, y, occ, kky, kkz, cnt


class _DeviceArray:
    """an array of a context as the CUDA array interface describes it; holds the context"""

    def __init__(self, run, pointer, shape, typestr):
        self.run = run
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(pointer), False), "version": 2}


def prepare(case, seed):
    proj, y, occ, kky, kkz, cnt = _inputs(case, seed)
    N, S = proj.numel, case["nwf"]
    run_ = TDRun(proj, S, precision=PRECISIONS[case["precision"]])
    states, dens, pots = ctypes.c_void_p(), ctypes.POINTER(ctypes.c_double)(), ctypes.POINTER(ctypes.c_double)()
    run_._check(run_.lib.wtd_device_pointers(run_.h, ctypes.byref(states), ctypes.byref(dens), ctypes.byref(pots)))
    view = lambda p, shape, t: torch.as_tensor(_DeviceArray(run_, p, shape, t), device="cuda")  # noqa: E731
    d_states = view(states.value, (2, S, N), "<c16" if case["precision"] == "fp64" else "<c8")
    d_states.copy_(y)
    del y
    p0 = np.zeros(12 * N)
    p0[4 * N:6 * N] = 1.0
    run_.setup_fields(p0, occ, _params(proj.name), kky=kky, kkz=kkz, cnt=cnt)
    torch.cuda.synchronize()
    if not case["gradient"]:
        run_.initial_measurement()
    run_.sync()
    state = {"run": run_, "steps": case["steps"], "energy": case["energy"], "gradient": case["gradient"],
             "stream": torch.cuda.ExternalStream(run_.stream()),
             "states": d_states,
             "densities": view(ctypes.addressof(dens.contents), (12 * N,), "<f8"),
             "potentials": view(ctypes.addressof(pots.contents), (12 * N,), "<f8")}
    torch.cuda.synchronize()
    return state


def run(state):
    r = state["run"]
    here = torch.cuda.current_stream()
    # the context's work comes after the caller's, and the caller's next after the context's
    state["stream"].wait_stream(here)
    out = {}
    if state["gradient"]:
        loss, grad = r.adjoint(state["steps"], nparam=14, checkpoint_every=state["gradient"])
        out["loss"], out["gradient"] = loss, grad
    else:
        r.steps(state["steps"])
        if state["energy"]:
            out["energy"] = r.energy()
    here.wait_stream(state["stream"])
    out["states"], out["densities"], out["potentials"] = state["states"], state["densities"], state["potentials"]
    return out


def work(case):
    """The ABM stream: per step and state the predictor reads y and q history arrays and writes
    f_k, y_pred and P, the corrector reads y_pred and P and writes y.  Operations: the spectral
    derivatives (5 n log2 n per complex transform)."""
    proj = Project(case["project"])
    S, N, steps = case["nwf"], proj.numel, case["steps"]
    size = 16 if case["precision"] == "fp64" else 8
    hist = 8 if case["precision"] == "h32" else 16
    q = proj.nhist - 1
    step_bytes = S * 2 * N * (size * 4 + hist * (q + 3))
    fft = 5.0 * N * math.log2(N)
    # per component and half step: forward, laplacian back (constant mass); variable mass adds
    # the first derivatives, the transform pair of alpha psi and the gradient densities
    d = proj.codedim
    per_half = 2 * fft if proj.const_mass else (2 + d + 2 + 2 + d) * fft
    step_flops = S * 2 * 2 * per_half
    sweeps = 1.0
    if case["gradient"]:
        sweeps = 3.0  # the forward, and a reverse sweep of twice its arrays
    return {"bytes": sweeps * steps * step_bytes, "flops": sweeps * steps * step_flops}


def tolerance(case):
    # about four times what the outputs differ by from exact(): FP64 up to 1.3e-15 per block (a few
    # times more where the densities' sums cancel), complex64 states 1.3e-7; the gradient takes
    # dv_ext/dtheta by central differences with step 1e-6, 1e-10 in FP64
    if case["gradient"]:
        return {"rel": 5e-10}
    if case["precision"] == "fp64":
        return {"rel": 2e-14}
    return {"rel": 5e-7}


# ---------------------------------------------------------------------------------------------
# the step in plain torch
# ---------------------------------------------------------------------------------------------
NMIN, NMAX, DENSEPS, GAMMA0, G0, G1 = 1.0e-7, 1.0e-5, 1.0e-8, -11.11, 0.357, 0.642
R0, R1 = 1.0 / (2.0 * math.pi ** 2), 0.5
PREDICT = {3: [23 / 12, -16 / 12, 5 / 12], 4: [55 / 24, -59 / 24, 37 / 24, -9 / 24],
           5: [1901 / 720, -2774 / 720, 2616 / 720, -1274 / 720, 251 / 720]}
CORRECT = {3: (9 / 24, [19 / 24, -5 / 24, 1 / 24]), 4: (251 / 720, [646 / 720, -264 / 720, 106 / 720, -19 / 720]),
           5: (251 / 720, [646 / 720, -264 / 720, 106 / 720, -19 / 720])}


class _Exact:
    def __init__(self, case, seed, params=None):
        self.case = case
        proj, y, occ, kky, kkz, cnt = _inputs(case, seed)
        self.proj, self.dims = proj, [proj.nx, proj.ny, proj.nz][: proj.codedim]
        self.y = y.to(torch.complex128)
        self.S, self.N = case["nwf"], proj.numel
        self.f = torch.tensor(occ, device="cuda")
        self.kp2 = torch.zeros(self.S, dtype=torch.float64, device="cuda")
        self.w = torch.ones(self.S, dtype=torch.float64, device="cuda")
        if kky is not None:
            self.kp2 = torch.tensor(kky ** 2 + kkz ** 2, device="cuda")
            self.w = torch.tensor(cnt, dtype=torch.float64, device="cuda")
        self.d = [proj.dx, proj.dy, proj.dz]
        full = [proj.nx, proj.ny, proj.nz]
        self.L = [a * b for a, b in zip(self.d, full)]
        self.lperp = math.prod(self.L[proj.codedim:])
        self.volel = math.prod(self.d) * math.prod(full[proj.codedim:])
        self.dv = proj.dv
        self.c = proj.constants()
        self.p = torch.tensor(_params(proj.name), device="cuda") if params is None else params
        self.var = not proj.const_mass
        self.A = (1.094, 0.156, -0.532) if self.var else (1.0, 0.0, 0.0)
        self.mf = proj.name.startswith("t2d_")
        k, kn = [], []
        for n, L in zip(self.dims, self.L):
            m = torch.arange(n, device="cuda")
            kk = (2.0 * math.pi / L) * torch.where(m < n // 2, m, m - n).double()
            k.append(kk)
            kn.append(torch.where(m == n // 2, 0.0, kk))
        shape = lambda v, a: v.reshape([-1 if b == a else 1 for b in range(len(self.dims))])  # noqa: E731
        self.k2 = sum(shape(v * v, a) for a, v in enumerate(k))
        self.kd = [shape(v, a) for a, v in enumerate(kn)]
        x = [(torch.arange(n, device="cuda") - n // 2).double() * s for n, s in zip(full, self.d)]
        grids = torch.meshgrid(*x[: proj.codedim], indexing="ij")
        self.x = [g.reshape(-1) for g in grids] + [torch.full((self.N,), -(n // 2) * s, dtype=torch.float64, device="cuda")
                                                   for n, s in list(zip(full, self.d))[proj.codedim:]]
        z = lambda: torch.zeros(self.N, dtype=torch.float64, device="cuda")  # noqa: E731
        self.V = [z(), z()]
        self.delta = z().to(torch.complex128)
        self.al = [z() + 1.0, z() + 1.0]
        self.Acur = [[z(), z(), z()], [z(), z(), z()]]
        self.it = 0
        self.hist = [torch.zeros_like(self.y) for _ in range(proj.nhist - 1)]  # f_{k-1}, f_{k-2}, ...
        self.f1 = torch.zeros_like(self.y)
        self.coef_ready = False
        self.axes = tuple(range(-len(self.dims), 0))

    # spectral operators on [..., N]
    def fft(self, a):
        return torch.fft.fftn(a.reshape(*a.shape[:-1], *self.dims), dim=self.axes)

    def ifft(self, a):
        return torch.fft.ifftn(a, dim=self.axes).reshape(*a.shape[: a.dim() - len(self.dims)], self.N)

    def lap(self, a):
        return self.ifft(-self.k2 * self.fft(a))

    def lap_real(self, a):
        return self.lap(a.to(torch.complex128)).real

    def grad(self, a, axis):
        return self.ifft(1j * self.kd[axis] * self.fft(a))

    # hooks
    def v_ext(self, spin):
        name, p, t = self.proj.name, self.p, self.c["dt"] * self.it
        x, y, z = self.x
        if name.startswith("gauss_"):
            a, b, r = float(p[4]), float(p[5]), float(p[6])
            ramp = lambda s: 0.5 * (1.0 + math.tanh(math.tan(math.pi / 2 * (2.0 * s / r - 1.0))))  # noqa: E731
            s = 0.0 if t <= a or t >= b else 1.0 if a + r <= t <= b - r else ramp(t - a) if t < a + r else 1.0 - ramp(t - b + r)
            return -p[0] * s * torch.exp(p[1] * x * x + p[2] * y * y + p[3] * z * z)
        if name == "c1_bdg1d":
            return 0.5 * p[1] ** 2 * x * x
        if name == "c2_slda2d":
            return 0.5 * p[0] ** 2 * (x * x + y * y)
        if name == "c3_aslda3d":
            return torch.zeros_like(x)
        if name == "c4_bdg2d":
            sx = sum(p[2 * h - 2] * torch.cos(h * p[16] * t) + p[2 * h - 1] * torch.sin(h * p[16] * t) for h in (1, 2, 3))
            sy = sum(p[4 + 2 * h] * torch.cos(h * p[16] * t) + p[5 + 2 * h] * torch.sin(h * p[16] * t) for h in (1, 2, 3))
            w = p[17] * p[13]
            return p[12] * torch.exp(-((x - p[15] * sx) ** 2 + (y - p[15] * sy) ** 2) / (2.0 * w * w))
        if name == "c5_slda3d":
            x0, y0 = p[4] * torch.cos(p[5] * t), p[4] * torch.sin(p[5] * t)
            return p[2] * torch.exp(-((x - x0) ** 2 + (y - y0) ** 2) / (2.0 * p[3] ** 2))
        v = 0.5 * p[0] ** 2 * (x * x + y * y + z * z) + p[1] * math.sin(float(p[2]) * t) * x / self.L[0]
        return v + 0.01 * p[1] if spin else v

    def delta_ext(self):
        name, p = self.proj.name, self.p
        x, y, _ = self.x
        if name in ("c2_slda2d", "c5_slda3d"):
            d0, xi = (p[1], p[2]) if name == "c2_slda2d" else (p[0], p[1])
            r = torch.sqrt(x * x + y * y)
            a = torch.where(r == 0.0, 0.0, d0 * torch.tanh(r / xi) / torch.where(r == 0.0, 1.0, r))
            return torch.complex(a * x, a * y)
        if name.startswith("t2d_"):
            c = torch.cos(2.0 * math.pi * y / self.L[1])
            return torch.complex(p[3] * c, p[3] * 0.5 * torch.sin(2.0 * math.pi * x / self.L[0]) * c)
        return torch.zeros(self.N, dtype=torch.complex128, device="cuda")

    # local functional
    @staticmethod
    def p_reg(n):
        a = torch.tan(math.pi * (n.clamp(NMIN, NMAX) - NMIN) / (NMAX - NMIN) - math.pi / 2)
        return torch.where(n <= NMIN, 0.0, torch.where(n >= NMAX, 1.0, 0.5 + 0.5 * torch.tanh(a)))

    @staticmethod
    def dp_reg(n):
        inside = (n > NMIN) & (n < NMAX)
        a = math.pi * (torch.where(inside, n, 0.5 * (NMIN + NMAX)) - NMIN) / (NMAX - NMIN) - math.pi / 2
        c = torch.cosh(torch.tan(a)) * torch.cos(a)
        return torch.where(inside, 0.5 * math.pi / (c * c) / (NMAX - NMIN), 0.0)

    def alpha(self, p):
        a0, a1, a2 = self.A
        return a0 + a1 * p * (1 - 2 / 3 * p ** 2 + p ** 4 / 5) + a2 * p ** 2 * (1 - p ** 2 + p ** 4 / 3)

    def potentials(self):
        va, vb = self.v_ext(0), self.v_ext(1)
        func, c = self.proj.functional, self.c
        rho, nu = self.rho, self.nu
        if func == "CUSTOMEDF":
            g = self.p[0] if self.proj.name == "c1_bdg1d" else self.p[14]
            self.V, self.delta = [va, vb], -g * nu
            return
        sqrt = lambda v: torch.sqrt(v.to(torch.complex128))  # noqa: E731

        def regular(mu, ap):
            p0 = sqrt(2.0 * mu / ap)
            p0 = torch.where(p0.imag < 0, -p0, p0)
            kc = sqrt(2.0 * (c["ec"] + mu) / ap)
            kc = torch.where(kc.imag < 0, -kc, kc)
            z = torch.log((kc + p0) / (kc - p0))
            z = torch.where(z.imag < 0, z + 2j * math.pi, z)
            return p0, kc * R0 * (1.0 - (p0 / kc) * R1 * z)

        if func == "BDG":
            ap = 0.5 * (self.al[0] + self.al[1])
            mu = (c["mu_a"] - self.V[0] + c["mu_b"] - self.V[1]) / 2
            _, lam = regular(mu, torch.ones_like(mu))
            geff = 1.0 / (1.0 / (4 * math.pi * c["sclgth"] * ap) - lam / ap)
            self.V, self.delta = [va, vb], -geff.real * nu
            return
        na, nb = rho
        n = na + nb
        pr, dpr = self.p_reg(n), self.dp_reg(n)
        p = pr * (na - nb) / n
        dpol = [pr * 2 * nb / n ** 2 + dpr * (na - nb) / n, -pr * 2 * na / n ** 2 + dpr * (na - nb) / n]
        a0, a1, a2 = self.A
        aa, ab = self.alpha(p), self.alpha(-p)
        ap, am = 0.5 * (aa + ab), 0.5 * (aa - ab)
        dap = 2 * a2 * p * (1 - p ** 2 + p ** 4 / 3) - 2 * a2 * p ** 3 * (1 - 2 / 3 * p ** 2)
        dam = a1 * (1 - 2 / 3 * p ** 2 + p ** 4 / 5) - 4 * a1 * p ** 2 * (1 / 3 - p ** 2 / 5)
        G = G0 + G1 * p ** 2
        P5, M5 = ((1 + p) / 2) ** (5 / 3), ((1 - p) / 2) ** (5 / 3)
        P2, M2 = ((1 + p) / 2) ** (2 / 3), ((1 - p) / 2) ** (2 / 3)
        brk = G - aa * P5 - ab * M5
        six = 6 * math.pi ** 2 * n
        const = [0.5 * six ** (2 / 3) * brk + six ** (5 / 3) / (20 * math.pi ** 2) *
                 (2 * G1 * p - (dam + dap) * P5 - 5 / 6 * aa * P2 - (-dam + dap) * M5 + 5 / 6 * ab * M2) * dpol[s] for s in (0, 1)]
        const = [va + const[0], vb + const[1]]
        dams = dap_s = [torch.zeros_like(n)] * 2
        if self.var:
            self.al = [aa, ab]
            j = self.j
            for s, a in ((0, aa), (1, ab)):
                t = self.p_reg(rho[s])
                self.Acur[s] = [torch.where(t == 0, 0.0, t * (1 - a) * j[s][q] / rho[s]) for q in range(len(self.dims))]
            dams, dap_s = [dam * d for d in dpol], [dap * d for d in dpol]
            for s in (0, 1):
                const[s] = const[s] + dams[s] * (self.tau[0] - self.tau[1]) / 2 + dap_s[s] * (self.tau[0] + self.tau[1]) / 2
            ja2, jb2 = (sum(q * q for q in j[s]) for s in (0, 1))
            t = self.p_reg(na)
            t7 = torch.where(t != 0, t * ja2 / (2 * na), 0.0)
            const[0] = const[0] + ((ap + am - 1) / na - (dap_s[0] + dams[0])) * t7 - torch.where(t != 0, self.dp_reg(na) * (ap + am - 1) * ja2 / (2 * na), 0.0)
            const[1] = const[1] - (dap_s[1] + dams[1]) * t7
            t = self.p_reg(nb)
            t7 = torch.where(t != 0, t * jb2 / (2 * nb), 0.0)
            const[0] = const[0] - (dap_s[0] - dams[0]) * t7
            const[1] = const[1] + ((ap - am - 1) / nb - (dap_s[1] - dams[1])) * t7 - torch.where(t != 0, self.dp_reg(nb) * (ap - am - 1) * jb2 / (2 * nb), 0.0)
        ne = n + DENSEPS
        dC = [(dap * dpol[s] * ne ** (1 / 3) + ap * ne ** (-2 / 3) / 3) / GAMMA0 for s in (0, 1)]
        tC = ap * ne ** (1 / 3) / GAMMA0
        Vn = list(self.V)
        kF = (3 * math.pi ** 2 * n) ** (1 / 3)
        for _ in range(15):
            mu = (c["mu_a"] - Vn[0] + c["mu_b"] - Vn[1]) / 2
            p0, lam = regular(mu, ap)
            geff = (ap / (tC - lam)).real
            ld = -geff * nu
            dn, d2 = (ld.conj() * nu).real, ld.abs() ** 2
            new = [const[s] - dap_s[s] / ap * dn - dC[s] / ap * d2 for s in (0, 1)]
            if self.mf:
                bc = (p0 / (kF + 1e-12)).real
                lx = bc * kF * self.d[0] / math.pi
                ok = (geff < -1e-10) & (lx > 1e-10)
                q = torch.where(ok, lx, 0.5)
                l0 = bc * R0 / q * (1 - R1 * q * torch.log((1 + q) / (1 - q)))
                dl0 = -2 * bc * R0 * R1 / (1 - q * q) - bc * R0 / q / q
                dl = torch.where(ok, kF / (3 * n * ap) * (l0 + dl0 * bc * self.d[0] * kF / math.pi), 0.0)
                new = [v + dl * d2 for v in new]
            Vn = [0.75 * b + 0.25 * a for a, b in zip(Vn, new)]
        self.V, self.delta = Vn, ld

    def coefficients(self):
        self.D = self.delta + self.delta_ext()
        self.va = [self.V[0] - self.c["mu_a"], self.V[1] - self.c["mu_b"]]
        if self.var:
            self.na = [0.25 * self.lap_real(a) for a in self.al]
            self.div = [-0.5 * sum(self.grad(a.to(torch.complex128), q).real for q, a in enumerate(A)) for A in self.Acur]
        self.coef_ready = True

    def chunks(self):
        c = max(1, (1 << 23) // self.N)
        return [slice(a, min(self.S, a + c)) for a in range(0, self.S, c)]

    def apply(self, u, v, kp2):
        """(H - <H>) of a chunk of states"""
        kp = kp2[:, None]
        out = []
        for s, (a, b) in enumerate(((u, v), (v, u))):
            F = self.fft(a)
            lap = self.ifft(-self.k2 * F)
            if self.var:
                al = self.al[s]
                h = (self.va[s] + 0.5 * al * kp + (1j if s == 0 else -1j) * self.div[s] + self.na[s]) * a
                h = h - 0.25 * al * lap - 0.25 * self.lap(al * a)
                h = -h if s else h
                for q in range(len(self.dims)):
                    h = h - 1j * self.Acur[s][q] * self.ifft(1j * self.kd[q] * F)
            else:
                h = (self.va[s] + 0.5 * kp) * a - 0.5 * lap
                h = -h if s else h
            out.append(h + (self.D.conj() if s else self.D) * b)
        e = ((u.conj() * out[0]).real.sum(-1) + (v.conj() * out[1]).real.sum(-1)) * self.dv
        return out[0] - e[:, None] * u, out[1] - e[:, None] * v

    def H(self, y):
        parts = [torch.stack(self.apply(y[0, c], y[1, c], self.kp2[c])) for c in self.chunks()]
        return torch.cat(parts, 1)

    def normalise(self, y):
        return y / torch.sqrt((y.real ** 2 + y.imag ** 2).sum((0, 2)) * self.dv)[None, :, None]

    def measure(self, y, full):
        f, w = self.f, self.w
        rho = [(f * w) @ (y[0].real ** 2 + y[0].imag ** 2), ((1 - f) * w) @ (y[1].real ** 2 + y[1].imag ** 2)]
        self.rho = [r / self.lperp for r in rho]
        fn = (0.5 * (1 - 2 * f) * w).to(torch.complex128)
        self.nu = sum(fn[c] @ (y[0, c] * y[1, c].conj()) for c in self.chunks()) / self.lperp
        zero = torch.zeros(self.N, dtype=torch.float64, device="cuda")
        self.tau, self.j = [zero, zero], [[zero] * len(self.dims), [zero] * len(self.dims)]
        if not full:
            return
        for s, weight in ((0, f * w), (1, (1 - f) * w)):
            t, j = zero, [zero] * len(self.dims)
            for c in self.chunks():
                a = y[s, c]
                F = self.fft(a)
                lap = self.ifft(-self.k2 * F) - self.kp2[c][:, None] * a
                t = t + weight[c] @ (a.conj() * lap).real
                for q in range(len(self.dims)):
                    j[q] = j[q] + (1 - 2 * s) * (weight[c] @ (a.conj() * self.ifft(1j * self.kd[q] * F)).imag)
            self.tau[s] = (0.5 * self.lap_real(self.rho[s]) - t / self.lperp).clamp(min=0.0)
            self.j[s] = [q / self.lperp for q in j]

    def start(self):
        self.y = self.normalise(self.y)
        self.measure(self.y, True)

    def predict(self, y, f0, hist):
        b = PREDICT[self.proj.nhist]
        s = b[0] * f0
        for k, h in enumerate(hist):
            s = s + b[k + 1] * h
        return self.normalise(y - 1j * self.c["dt"] * s)

    def correct(self, y, f0, hist, fp):
        c, a = CORRECT[self.proj.nhist]
        s = a[0] * f0 + c * fp
        for k, h in enumerate(hist):
            if k + 1 < len(a):
                s = s + a[k + 1] * h
        return self.normalise(y - 1j * self.c["dt"] * s)

    def step(self, last):
        f0 = self.H(self.y) if self.coef_ready else self.f1
        yp = self.predict(self.y, f0, self.hist)
        self.it += 1
        self.measure(yp, self.var)
        self.potentials()
        self.coefficients()
        self.y = self.correct(self.y, f0, self.hist, self.H(yp))
        self.hist = [f0] + self.hist[:-1]
        self.measure(self.y, self.var or last)
        self.potentials()
        self.coefficients()

    def energy(self):
        func, n = self.proj.functional, self.rho[0] + self.rho[1]
        j2 = [sum(q * q for q in self.j[s]) for s in (0, 1)]
        pr = [self.p_reg(r) for r in self.rho]
        e = [0.0] * 11
        if func == "CUSTOMEDF":
            e[0] = 0.5 * (self.al[0] * self.tau[0] + self.al[1] * self.tau[1]).sum()
            e[2] = -0.5 * (self.delta * self.nu.conj()).real.sum()
        else:
            t = [self.tau[s] - pr[s] * j2[s] / self.rho[s] for s in (0, 1)]
            e[2] = -(self.delta * self.nu.conj()).real.sum()
            e[3] = sum((pr[s] * j2[s] / (2 * self.rho[s])).sum() for s in (0, 1))
            if func == "BDG":
                e[0] = 0.5 * (self.al[0] * t[0] + self.al[1] * t[1]).sum()
            else:
                p = self.p_reg(n) * (self.rho[0] - self.rho[1]) / n
                aa, ab = self.alpha(p), self.alpha(-p)
                e[0] = 0.5 * (aa * t[0] + ab * t[1]).sum()
                e[1] = ((6 * math.pi ** 2 * n) ** (5 / 3) / (20 * math.pi ** 2) *
                        (G0 + G1 * p ** 2 - aa * ((1 + p) / 2) ** (5 / 3) - ab * ((1 - p) / 2) ** (5 / 3))).sum()
        e[4] = (self.rho[0] * self.v_ext(0) + self.rho[1] * self.v_ext(1)).sum()
        e[5] = -2.0 * (self.nu.conj() * self.delta_ext()).real.sum()
        e[7], e[8] = self.rho[0].sum(), self.rho[1].sum()
        if len(self.dims) > 1:
            e[9], e[10] = ((self.x[0] * self.j[s][1] - self.x[1] * self.j[s][0]).sum() for s in (0, 1))
        return np.array([float(v) * self.volel for v in e])

    def outputs(self):
        zero = torch.zeros(self.N, dtype=torch.float64, device="cuda")
        pad = lambda v: list(v) + [zero] * (3 - len(v))  # noqa: E731
        d = [torch.view_as_real(self.nu).reshape(-1)]
        for s in (0, 1):
            d += [self.rho[s], self.tau[s]] + pad(self.j[s])
        p = self.V + [torch.view_as_real(self.delta).reshape(-1)] + self.al
        for s in (0, 1):
            p = p + pad(self.Acur[s][: len(self.dims)])
        return {"states": self.y.detach(), "densities": torch.cat(d).detach(), "potentials": torch.cat(p).detach()}


def _exact_gradient(case, seed):
    """loss and gradient by autograd through the same step, one half step at a time"""
    from torch.utils.checkpoint import checkpoint
    params = torch.tensor(_params(case["project"]), device="cuda", requires_grad=True)
    x = _Exact(case, seed, params)
    with torch.no_grad():
        x.start()
    zero = torch.zeros_like(x.y)
    y, hist, n = x.y, [zero, zero], case["steps"]
    D = Va = None

    def fields(yy, p, it):
        x.p, x.it = p, it
        x.measure(yy, False)
        x.potentials()
        return x.delta, x.V[0]

    def first(y, h0, h1, D, Va, p, it, have):
        if have:
            x.D, x.va = D, [Va - x.c["mu_a"], Va - x.c["mu_b"]]
            f0 = x.H(y)
        else:
            f0 = zero
        yp = x.predict(y, f0, [h0, h1])
        return (yp, f0) + fields(yp, p, it)

    def second(y, yp, f0, h0, h1, D, Va, p, it):
        x.D, x.va = D, [Va - x.c["mu_a"], Va - x.c["mu_b"]]
        yn = x.correct(y, f0, [h0, h1], x.H(yp))
        return (yn,) + fields(yn, p, it)

    for k in range(n):
        yp, f0, D1, V1 = checkpoint(first, y, *hist, D, Va, params, k + 1, k > 0, use_reentrant=False)
        yn, D, Va = checkpoint(second, y, yp, f0, *hist, D1, V1, params, k + 1, use_reentrant=False)
        y, hist = yn, [f0, hist[0]]
    loss = (D.real ** 2 + D.imag ** 2).sum() * x.dv
    loss.backward()
    with torch.no_grad():
        x.p, x.it, x.y = params, n, y.detach()
        x.measure(x.y, True)
        x.potentials()
    out = x.outputs()
    return {"loss": float(loss), "gradient": params.grad[:14].cpu().numpy(), **out}


def exact(case, seed):
    if case["gradient"]:
        return _exact_gradient(case, seed)
    with torch.no_grad():
        x = _Exact(case, seed)
        x.start()
        for k in range(case["steps"]):
            x.step(k == case["steps"] - 1)
        out = {"energy": x.energy()} if case["energy"] else {}
        out.update(x.outputs())
    return out
