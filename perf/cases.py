"""The work that programs have this library do, as cases to be timed.

A case is one pass of a program over the public entry points, in one of five forms ("kind"):

* march      a GPU program that keeps prob.sol in its own device array (a CuArray, a torch tensor):
             push the array, take `steps` steps, write the array back, all on the caller's stream;
* integrate  the same around TimeIntegrator: fixed steps with volume penalisation and its
             divergence corrections, or on-device CFL steps with recorded diagnostics;
* session    a short program on host data: initial fields from host arrays, diagnostics between
             single steps, physical fields back to the host;
* host       the C ABI on page-locked host arrays: set_state, step, get_state;
* ensemble   size classes of independent boxes advanced together, one device array per box.

Sizes, schemes, viscosities and spectra are those of the repository's benchmark configurations and
tests: the seeded spectrum E(k) ~ k^4 exp(-2 (k/kpeak)^2) and Taylor-Green fields, 16^3 to 512^3.
"""
import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import load_package

L = 2 * math.pi
SIZES = (16, 32, 48, 64, 96, 128, 256, 512)
FORMS = ("mhd", "hd")


def _case(kind, n=0, steps=1, scheme="RK4", form="mhd", **kw):
    c = {"kind": kind, "n": n, "steps": steps, "scheme": scheme, "form": form, "ic": "random", "kpeak": 4.0,
         "nu": 1e-3, "eta": 1e-3, "b_ratio": 0.3, "dt": 0.2 * L / max(n, 1), "vp": "none", "forced": False, "cfl": False,
         "tuned": True}
    c.update(kw)
    return c


def listed():
    return [
        # one stepforward! of the smallest benchmark grid on the program's own device array: launch latency
        dict(_case("march", 32, 1, ic="tg", nu=1e-2, eta=1e-2, dt=1e-3), name="stepforward_32"),
        # the CPU reference configuration, Taylor-Green 32^3, 100 RK4 steps between two looks at the spectra
        dict(_case("march", 32, 100, ic="tg", nu=1e-2, eta=1e-2, dt=1e-3), name="tg_32_x100"),
        # a small low-storage run, as in the serving mix
        dict(_case("march", 64, 20, "LSRK4", nu=2e-3, eta=5e-4), name="lsrk4_64_x20"),
        # host initial conditions, a diagnostic after every step, fields back for a snapshot
        dict(_case("session", 96, 10), name="session_96"),
        # TimeIntegrator! without a fixed dt: getCFL! on the device and recorded energies
        dict(_case("integrate", 128, 20, cfl=True), name="cfl_128_x20"),
        # A99-forced turbulence
        dict(_case("march", 128, 5, "LSRK4", forced=True), name="forced_128_x5"),
        # a penalised obstacle with moving walls, corrected to solenoidal fields after each step
        dict(_case("integrate", 128, 10, vp="walls"), name="vp_128_x10"),
        # hydrodynamics (B_field = false), a program that never calls the autotuner
        dict(_case("march", 256, 2, form="hd", tuned=False), name="hd_256_x2"),
        # the headline configuration, 256^3 RK4
        dict(_case("march", 256, 5, dt=5e-4), name="rk4_256_x5"),
        # one step between host arrays: the end-to-end benchmark
        dict(_case("host", 256, 1, dt=5e-4), name="host_256"),
        # the largest grid, one stepforward! on the program's own device array
        dict(_case("march", 512, 1, nu=5e-4, eta=5e-4, dt=2.5e-4), name="rk4_512"),
        # the batched-ensemble configuration: 64 uneven boxes, LSRK4
        dict(_case("ensemble", 0, 10, "LSRK4", n32=24, n48=20, n64=12, n96=8), name="ensemble_x10"),
    ]


def draw(rng):
    """A case of the same ranges; at most about 512^3 point-steps."""
    log = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    nu = log(5e-4, 5e-3)
    kw = {"nu": nu, "eta": rng.choice((nu, log(5e-4, 5e-3))), "kpeak": rng.uniform(2.0, 6.0),
          "b_ratio": rng.uniform(0.1, 1.0), "tuned": rng.random() < 0.6}
    scheme = rng.choice(("RK4", "LSRK4"))
    kind = rng.choice(("march", "march", "march", "integrate", "session", "host", "ensemble", "ensemble"))

    def steps_for(n, most):
        cost = 1.2e-10 * n ** 3 + 1.2e-4  # about a step's seconds
        return max(1, int(log(1.0, max(1.5, min(most, 0.02 / cost)))))

    if kind == "ensemble":
        counts = {"n32": rng.randint(0, 24), "n48": rng.randint(0, 20), "n64": rng.randint(1, 12), "n96": rng.randint(0, 8)}
        return _case("ensemble", 0, rng.randint(2, 10), scheme, **counts, **kw)
    if kind == "integrate":
        n = rng.choice((32, 48, 64, 96, 128))
        if rng.random() < 0.5:
            return _case("integrate", n, steps_for(n, 25), scheme, cfl=True, **kw)
        return _case("integrate", n, steps_for(n, 20), scheme, vp=rng.choice(("mask", "walls")), form=rng.choice(FORMS), **kw)
    if kind == "session":
        n = rng.choice((32, 48, 64, 96))
        return _case("session", n, rng.randint(2, 10), scheme, **kw)
    if kind == "host":
        n = rng.choice((48, 64, 96, 128, 256))
        return _case("host", n, rng.randint(1, 3), scheme, **kw)
    n = rng.choice(SIZES[:7])
    form = rng.choice(("mhd", "mhd", "hd"))
    forced = form == "mhd" and n <= 128 and rng.random() < 0.3
    return _case("march", n, steps_for(n, 100), scheme, form, forced=forced, **kw)


# ---------------------------------------------------------------------------------------------
# Inputs (torch on the GPU, from the seed alone)
# ---------------------------------------------------------------------------------------------
def _kept(n):
    """2/3 rule: kept modes of the half axis, and kept non-negative / negative ones of a full axis."""
    lo, hi = (1 - 1 / 3) / 2 * n, (1 + 1 / 3) / 2 * n
    return math.floor(lo), math.floor(lo), n - math.ceil(hi)


def _waves(n, dtype):
    kx = torch.arange(n // 2 + 1, device="cuda", dtype=dtype).reshape(1, 1, -1)
    k = (torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)).to(dtype)
    return kx, k.reshape(1, n, 1), k.reshape(n, 1, 1)


def _mask(n):
    kx, kp, kn = _kept(n)
    m = torch.zeros((n, n, n // 2 + 1), dtype=torch.bool, device="cuda")
    for z in (slice(0, kp), slice(n - kn, n)):
        for y in (slice(0, kp), slice(n - kn, n)):
            m[z, y, :kx] = True
    return m


def _project(f, ks, inv):
    p = (ks[0] * f[0] + ks[1] * f[1] + ks[2] * f[2]) * inv
    for a in range(3):
        f[a] -= ks[a] * p


def _random_sol(n, nf, seed, kpeak, b_ratio):
    """Solenoidal random-phase state (nf, n, n, n/2+1) complex64 on the retained band."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    ks = _waves(n, torch.float32)
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    inv = torch.where(k2 > 0, 1.0 / k2.clamp(min=1.0), torch.zeros_like(k2))
    shape = torch.sqrt(k2) * torch.exp(-k2 / kpeak ** 2) * _mask(n)
    sol = torch.empty((nf, n, n, n // 2 + 1), dtype=torch.complex64, device="cuda")
    w = torch.full((n // 2 + 1,), 2.0, device="cuda")
    w[0] = 1.0
    for h in range(nf // 3):
        f = sol[3 * h:3 * h + 3]
        for a in range(3):
            f[a] = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device="cuda")) * shape
        _project(f, ks, inv)
        ms = sum(float((w * (torch.view_as_real(f[a]) ** 2).sum(-1)).sum(dtype=torch.float64)) for a in range(3)) / float(n) ** 6
        f *= (1.0 if h == 0 else b_ratio) / math.sqrt(ms)
    return sol


def _tg_phys(n, nf, seed):
    """Taylor-Green u and B (amplitude 0.5) about a seeded origin, float32 (nf, z, y, x)."""
    r = np.random.default_rng(seed)
    o, amp = r.uniform(0, L, 3), r.uniform(0.8, 1.2)
    g = [torch.arange(n, device="cuda", dtype=torch.float64) * (L / n) + o[a] for a in range(3)]
    z, y, x = torch.meshgrid(g[2], g[1], g[0], indexing="ij")
    f = [torch.sin(x) * torch.cos(y) * torch.cos(z), -torch.cos(x) * torch.sin(y) * torch.cos(z), torch.zeros_like(x),
         0.5 * torch.cos(x) * torch.sin(y) * torch.sin(z), -0.5 * torch.sin(x) * torch.cos(y) * torch.sin(z), torch.zeros_like(x)]
    return (amp * torch.stack(f[:nf])).float()


def _sol(case, seed):
    nf = 6 if case["form"] == "mhd" else 3
    if case["ic"] == "tg":
        return torch.fft.rfftn(_tg_phys(case["n"], nf, seed), dim=(1, 2, 3)) * _mask(case["n"])
    return _random_sol(case["n"], nf, seed, case["kpeak"], case["b_ratio"])


def _obstacle(case, seed):
    """A smooth ball obstacle chi and, with walls, its velocity and field (3, z, y, x) each."""
    n = case["n"]
    r = np.random.default_rng(seed + 1)
    c, rad, v = r.uniform(-1, 1, 3), r.uniform(0.6, 1.2), r.uniform(-0.5, 0.5, 6)
    g = torch.arange(n, device="cuda", dtype=torch.float64) * (L / n) - math.pi
    z, y, x = torch.meshgrid(g, g, g, indexing="ij")
    d = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2)
    chi = (0.5 - 0.5 * torch.tanh((d - rad) * n / (2 * L))).float()
    wall = None
    if case["vp"] == "walls":
        wall = torch.stack([v[a] * (1 + 0.5 * torch.cos(z + a)) for a in range(6)]).float()
    return chi, wall


def _power(n):
    """Injected power of the forcing: an acceleration of about one at every grid size."""
    return 320.0 / n ** 3


def _boxes(case, seed):
    """(n, nu, seed) of each box of an ensemble; viscosities log-uniform about the case's."""
    r = np.random.default_rng(seed)
    out = []
    for n in (32, 48, 64, 96):
        for _ in range(case["n%d" % n]):
            out.append((n, case["nu"] * math.exp(r.uniform(-1, 1)), int(r.integers(1 << 40))))
    return out


# ---------------------------------------------------------------------------------------------
# The program's side
# ---------------------------------------------------------------------------------------------
def _problem(pkg, case):
    p = pkg.Problem(pkg.GPU(0), nx=case["n"], Lx=L, nu=case["nu"], eta=case["eta"], dt=case["dt"], stepper=case["scheme"],
                    B_field=case["form"] == "mhd", VP_method=case["vp"] != "none")
    return p


def prepare(case, seed):
    pkg = load_package()
    s = {"case": case, "pkg": pkg, "lib": pkg._lib.load()}
    kind = case["kind"]
    if kind == "ensemble":
        classes, boxes = {}, _boxes(case, seed)
        for n, nu, bs in boxes:
            if n not in classes:
                count = case["n%d" % n]
                nk = n // 2 + 1
                classes[n] = {"batch": pkg.Batch(n, count, stepper=case["scheme"]), "slots": [],
                              "sol": torch.empty((count, 6, n, n, nk), dtype=torch.complex64, device="cuda"),
                              "out": torch.empty((count, 6, n, n, nk), dtype=torch.complex64, device="cuda")}
            c = classes[n]
            c["sol"][len(c["slots"])] = _random_sol(n, 6, bs, case["kpeak"], case["b_ratio"])
            c["slots"].append(c["batch"].add(nu, nu, 0.2 * L / n))
        if case["tuned"]:
            for c in classes.values():
                pkg.autotune(c["batch"], persist=False)
        s["classes"] = classes
        s["ensemble"] = pkg.Ensemble([c["batch"] for c in classes.values()])
        return s
    prob = s["prob"] = _problem(pkg, case)
    if case["vp"] != "none":
        chi, wall = _obstacle(case, seed)
        w = None if wall is None else [a.cpu().numpy().T for a in wall]
        prob.set_vp(chi.cpu().numpy().T, None if w is None else w[:3], None if w is None else w[3:])
    if case["forced"]:
        pkg.SetUpFk(prob, kf=2.0, P=_power(case["n"]), sigma=1.0, b=1.0, seed=seed)
    if case["tuned"]:
        pkg.autotune(prob, persist=False)
    sol = _sol(case, seed)
    if kind == "session":
        phys = torch.fft.irfftn(sol, s=(case["n"],) * 3, dim=(1, 2, 3))
        names = pkg.FIELDS[:prob.nfields]
        s["fields"] = {f: phys[i].cpu().numpy().T for i, f in enumerate(names)}
    elif kind == "host":
        s["sol"] = sol.cpu().pin_memory()
        s["out"] = torch.empty_like(s["sol"]).pin_memory()
    else:
        s["sol"], s["out"] = sol, torch.empty_like(sol)
    return s


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    case, pkg, lib = s["case"], s["pkg"], s["lib"]
    kind, check = case["kind"], pkg._lib.check
    if kind == "ensemble":
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for c in s["classes"].values():
            h = c["batch"].handle
            for i, slot in enumerate(c["slots"]):
                check(lib.mhd_slot_set_state_device(h, slot, _ptr(c["sol"][i]), stream))
        s["ensemble"].step(case["steps"])
        for c in s["classes"].values():
            h = c["batch"].handle
            for i, slot in enumerate(c["slots"]):
                check(lib.mhd_slot_get_state_device(h, slot, _ptr(c["out"][i]), stream))
        return {n: c["out"] for n, c in s["classes"].items()}
    prob = s["prob"]
    if kind == "session":
        pkg.SetUpProblemIC(prob, **s["fields"])
        energies = []
        for _ in range(case["steps"]):
            pkg.stepforward(prob)
            d = prob.diagnostics()
            energies.append((d.E_u, d.E_B, d.H_c))
        pkg.updatevars(prob)
        return {"energies": np.array(energies, dtype=np.float32), **{f: getattr(prob.vars, f) for f in s["fields"]}}
    if kind == "host":
        check(lib.mhd_set_state(prob.handle, _ptr(s["sol"])))
        pkg.stepforward(prob, case["steps"])
        check(lib.mhd_get_state(prob.handle, _ptr(s["out"])))
        return s["out"]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check(lib.mhd_set_state_device(prob.handle, _ptr(s["sol"]), stream))
    history = None
    if kind == "integrate":
        if case["cfl"]:
            freq = max(1, case["steps"] // 4)
            prob.clock.t = 0.0
            pkg.TimeIntegrator(prob, math.inf, case["steps"] - 1, diag_freq=freq)
            history = prob.diagnostic_history()[:, 1:5].astype(np.float32)  # t, E_u, E_B, H_c
        else:
            pkg.TimeIntegrator(prob, math.inf, case["steps"] - 1, usr_dt=case["dt"])
    else:
        if case["forced"]:
            prob.clock.step = 0  # the forcing draws by the step count
        pkg.stepforward(prob, case["steps"])
    check(lib.mhd_get_state_device(prob.handle, _ptr(s["out"]), stream))
    return s["out"] if history is None else [s["out"], history]


def work(case):
    def one(n, nf, stages):
        state = 8.0 * nf * n * n * (n // 2 + 1)
        kx, kp, kn = _kept(n)
        band = 8.0 * nf * (kp + kn) ** 2 * kx
        transforms = 14 if nf == 6 else 8
        flops = stages * (transforms * 2.5 * n ** 3 * math.log2(n) + 40.0 * n ** 3)
        return state, band, flops

    stages = 4 if case["scheme"] == "RK4" else 5
    st = case["steps"]
    if case["kind"] == "ensemble":
        b = f = 0.0
        for n in (32, 48, 64, 96):
            s, r, fl = one(n, 6, stages)
            b += case["n%d" % n] * (2 * s + 2 * r * st)
            f += case["n%d" % n] * fl * st
        return {"bytes": b, "flops": f}
    n, nf = case["n"], 6 if case["form"] == "mhd" else 3
    s, r, fl = one(n, nf, stages)
    io = 2.0 * 4 * nf * n ** 3 if case["kind"] == "session" else 2 * s
    mask = 0.0 if case["vp"] == "none" else 4.0 * n ** 3 * (1 if case["vp"] == "mask" else 1 + nf)
    return {"bytes": io + 2 * r * st + mask * stages * st, "flops": fl * st}


# ---------------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------
_LS_A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
         -1275806237668 / 842570457699)
_LS_B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
         3134564353537 / 4481467310338, 2277821191437 / 14882151754819)


def _mix64(z):
    def shr(v, s):
        return (v >> s) & ((1 << (64 - s)) - 1)

    z = z + (0x9E3779B97F4A7C15 - (1 << 64))
    z = (z ^ shr(z, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ shr(z, 27)) * (0x94D049BB133111EB - (1 << 64))
    return z ^ shr(z, 31)


class _Exact:
    """Pseudospectral MHD / HD in float64 over a leading box dimension: X is (boxes, fields, z, y, kx)."""

    def __init__(self, n, nf, nu, eta, dt, scheme, chi=None, wall=None, forcing=None):
        self.n, self.nf, self.scheme, self.dt = n, nf, scheme, dt
        self.nu, self.eta = ([v] if isinstance(v, float) else v for v in (nu, eta))
        self.ks = _waves(n, torch.float64)
        self.k2 = self.ks[0] ** 2 + self.ks[1] ** 2 + self.ks[2] ** 2
        self.inv = torch.where(self.k2 > 0, 1.0 / self.k2.clamp(min=1.0), torch.zeros_like(self.k2))
        self.mask = _mask(n)
        self.chi, self.wall, self.forcing = chi, wall, forcing
        self.step, self.vmax = 0, 0.0

    def phys(self, c):
        c = torch.fft.ifftn(c, dim=(-3, -2))
        c[..., 0] = c[..., 0].real.to(c.dtype)
        return torch.fft.irfft(c, n=self.n, dim=-1)

    def spec(self, a):
        return torch.fft.rfftn(a, dim=(-3, -2, -1)) * self.mask

    def solenoidal(self, f):
        _project(f, self.ks, self.inv)
        return f

    def rhs(self, X, stage):
        N = torch.empty_like(X)
        for b in range(X.shape[0]):
            self.rhs_one(X[b], N[b], self.nu[b], self.eta[b], stage)
        return N

    def rhs_one(self, X, N, nu, eta, stage):
        ks, mhd = self.ks, self.nf == 6
        f = [self.phys(X[c]) for c in range(self.nf)]
        self.vmax = max(float(a.abs().max()) for a in f)
        u, B = f[:3], f[3:]
        N.zero_()
        for i in range(3):
            for j in range(i, 3):
                T = self.spec(B[i] * B[j] - u[i] * u[j] if mhd else -u[i] * u[j])
                N[i] += 1j * ks[j] * T
                if i != j:
                    N[j] += 1j * ks[i] * T
        self.solenoidal(N[:3])
        if mhd:
            for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):  # E_k = u_i B_j - u_j B_i
                E = self.spec(u[i] * B[j] - u[j] * B[i])
                N[3 + i] += 1j * ks[j] * E
                N[3 + j] -= 1j * ks[i] * E
        for c in range(self.nf):
            N[c] -= (nu if c < 3 else eta) * self.k2 * self.spec(f[c])
        if self.chi is not None:
            for h in range(self.nf // 3):
                F = torch.stack([self.spec(self.chi / (13 * self.dt / 7) * (
                    f[3 * h + a] - (0 if self.wall is None else self.wall[3 * h + a]))) for a in range(3)])
                N[3 * h:3 * h + 3] -= self.solenoidal(F)
        if self.forcing is not None:
            self.force(N, 8 * self.step + stage)

    def force(self, N, call):
        seed, n = self.forcing, self.n
        dx, sigma, b, kf, P = L / n, 1.0, 1.0, 2.0, _power(n)
        k = torch.sqrt(self.k2)
        A = math.sqrt(P * 3 * n ** 3 / float((torch.exp(-(k - kf) ** 2 / sigma ** 2) / (k + 1) ** 2).sum()) / dx ** 3)
        wrap = lambda v: v - (1 << 64) if v >= 1 << 63 else v  # noqa: E731
        i64 = lambda v: torch.tensor(wrap(v), dtype=torch.int64, device="cuda")  # noqa: E731
        key = _mix64(i64(seed) ^ _mix64(i64(call)))
        index = torch.arange(N[0].numel(), device="cuda").reshape(N[0].shape)
        draws = [((_mix64(key ^ (index * 4 + d)) >> 40) & 0xFFFFFF).double() / 16777216.0 for d in range(3)]
        kx, ky, kz = self.ks
        kp = torch.sqrt(kx ** 2 + kz ** 2).expand_as(k)
        ki, pi = (torch.where(v > 0, 1 / v.clamp(min=0.5), torch.zeros_like(v)) for v in (k, kp))
        Fk = A * torch.sqrt(torch.exp(-(k - b) ** 2 / sigma ** 2) / 2 / math.pi) * ki
        phi = draws[1] * math.pi
        gi = (-torch.tanh(b * (phi - math.pi / 2)) / math.tanh(b * math.pi / 2)).clamp(-1, 1)
        a1 = A * Fk * gi * torch.exp(2j * math.pi * draws[0])
        a2 = A * Fk * torch.sqrt(1 - gi ** 2) * torch.exp(2j * math.pi * draws[2])
        N[0] += (a1 * kz * pi + a2 * kx * ky * pi * ki) * self.mask
        N[1] += (-a2 * kp * ki) * self.mask
        N[2] += (-a1 * kx * pi + a2 * kz * ky * pi * ki) * self.mask
        N[:3, ..., 0] = N[:3, ..., 0].real.to(N.dtype)

    def advance(self, X):
        dt = self.dt
        if self.scheme == "RK4":
            R = self.rhs(X, 0)
            acc = R / 6
            for stage, (frac, w) in enumerate(((0.5, 3), (0.5, 3), (1.0, 6)), 1):
                R = self.rhs(X + (frac * dt) * R, stage)
                acc += R / w
            X = X + dt * acc
        else:
            dU = torch.zeros_like(X)
            X = X.clone()
            for i in range(5):
                R = self.rhs(X, i)
                dU = _LS_A[i] * dU + dt * R
                X += _LS_B[i] * dU
        self.step += 1
        return X

    def energies(self, X):
        w = torch.full((X.shape[-1],), 2.0, dtype=torch.float64, device="cuda")
        w[0] = 1.0
        sc = (L / self.n) ** 3 / self.n ** 3
        dot = lambda a, b: float((w * (a.real * b.real + a.imag * b.imag)).sum()) * sc  # noqa: E731
        u, b = X[0, :3], X[0, 3:]
        return [dot(u, u), dot(b, b), dot(u, b)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = {}
        boxes = _boxes(case, seed)
        for n in (32, 48, 64, 96):
            mine = [b for b in boxes if b[0] == n]
            if not mine:
                continue
            nus = [float(b[1]) for b in mine]
            e = _Exact(n, 6, nus, nus, 0.2 * L / n, case["scheme"])
            X = torch.stack([_random_sol(n, 6, b[2], case["kpeak"], case["b_ratio"]) for b in mine]).to(torch.complex128)
            for _ in range(case["steps"]):
                X = e.advance(X)
            out[n] = X
        return out
    chi = wall = None
    if case["vp"] != "none":
        chi, wall = _obstacle(case, seed)
        chi, wall = chi.double(), None if wall is None else wall.double()
    nf = 6 if case["form"] == "mhd" else 3
    e = _Exact(case["n"], nf, float(case["nu"]), float(case["eta"]), case["dt"], case["scheme"], chi, wall,
               seed if case["forced"] else None)
    sol = _sol(case, seed)
    if kind == "session":
        X = e.spec(torch.fft.irfftn(sol, s=(case["n"],) * 3, dim=(1, 2, 3)).double())[None]
        energies = []
        for _ in range(case["steps"]):
            X = e.advance(X)
            energies.append(e.energies(X))
        names = ("ux", "uy", "uz", "bx", "by", "bz")
        return {"energies": torch.tensor(energies, dtype=torch.float64),
                **{f: e.phys(X[0, i]).permute(2, 1, 0).contiguous() for i, f in enumerate(names)}}
    X = sol.to(torch.complex128)[None]
    del sol
    history = []
    if case["cfl"]:
        dx, t, freq = L / case["n"], 0.0, max(1, case["steps"] // 4)
        limit = 0.25 * dx * dx / max(case["nu"], case["eta"])
        e.vmax = max(float(e.phys(X[0, c]).abs().max()) for c in range(nf))
    if case["vp"] != "none":
        for h in range(nf // 3):
            e.solenoidal(X[0, 3 * h:3 * h + 3])
    for i in range(case["steps"]):
        if case["cfl"]:
            e.dt = min(0.25 * dx / e.vmax, limit)
        X = e.advance(X)
        if case["vp"] != "none":
            for h in range(nf // 3):
                e.solenoidal(X[0, 3 * h:3 * h + 3])
        if case["cfl"]:
            t += e.dt
            if (i + 1) % freq == 0:
                history.append([t] + e.energies(X))
    return X[0] if not case["cfl"] else [X[0], torch.tensor(history, dtype=torch.float64)]
