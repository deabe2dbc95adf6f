"""The work that users of dns_b200 have it do, as cases to be timed.

Three kinds of program, each through the library's public entry points:

* ``run``: the reference's own loop (main.c): a velocity field is loaded, the
  time step is repeated, energy and enstrophy are printed and the real fields
  are dumped.  One pass is the stretch between two dumps: ``steps`` RK4 steps,
  the diagnostics, and the fields in the program's own pinned host buffer.
  With ``fresh`` the pass also loads the field again, as a program does that
  runs one short case after another; with ``pressure`` the dump holds P too.
* ``ens``: an ensemble of runs of two grid sizes and of many viscosities
  stepped together, with every run's diagnostics and spectra read at the end.
* ``adj``: the gradient of the final energy with respect to the initial
  velocity and to the viscosity.

Fields are Taylor-Green plus a seeded solenoidal perturbation with
E(k) ~ k^4 exp(-2 (k/4)^2), as the library's ensembles start from.  What a
mixed-precision context returns is kept in float32, which is all the
precision that it has.
"""
import ctypes
import math

import numpy as np
import torch

import dns_b200

FP64, MIXED = dns_b200.DNS_PREC_FP64, dns_b200.DNS_PREC_MIXED


def _run(name, n, prec, steps, nu=1 / 1600, dt=0.0025, fresh=False, pressure=False):
    return {"name": name, "kind": "run", "n": n, "precision": prec, "steps": steps, "nu": nu,
            "dt": dt, "fresh": fresh, "pressure": pressure}


def listed():
    return [
        # the smallest calls: a test or a teaching run, one print interval
        _run("run32_fp64", 32, "fp64", 10, nu=0.01, dt=0.01),
        # short runs one after another (load, ten steps, dump with pressure)
        _run("run64_fp64_dump", 64, "fp64", 10, nu=0.01, dt=0.01, fresh=True, pressure=True),
        # the same size in mixed precision, an odd number of steps
        _run("run64_mixed", 64, "mixed", 25, nu=0.003, dt=0.005),
        # the reference's published 128^3 runs
        _run("run128_fp64", 128, "fp64", 20),
        _run("run128_mixed", 128, "mixed", 41, dt=0.005),
        # the benchmark's grid, both precisions
        _run("run256_fp64", 256, "fp64", 20, nu=1 / 3000),
        _run("run256_mixed", 256, "mixed", 40, nu=1 / 3000),
        # the largest grid
        _run("run512_fp64", 512, "fp64", 9, nu=1 / 3000),
        _run("run512_mixed", 512, "mixed", 16, nu=1 / 3000),
        # the ensemble of the benchmark: 32 runs at 64^3 and 16 at 128^3
        {"name": "ens_64_128_mixed", "kind": "ens", "n": 64, "runs": 32, "n2": 128, "runs2": 16,
         "precision": "mixed", "steps": 40, "dt": 0.005},
        # gradients: the benchmark's grid, and a small one in mixed precision
        {"name": "adj128_fp64", "kind": "adj", "n": 128, "precision": "fp64", "steps": 20,
         "snapshots": 6, "nu": 0.005, "dt": 0.005},
        {"name": "adj64_mixed", "kind": "adj", "n": 64, "precision": "mixed", "steps": 33,
         "snapshots": 5, "nu": 0.005, "dt": 0.005},
    ]


def draw(rng):
    def log_int(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    prec = rng.choice(["fp64", "mixed"])
    share = 1.0 if prec == "fp64" else 0.5
    nu, dt = math.exp(rng.uniform(math.log(1 / 3000), math.log(1 / 100))), rng.choice([0.002, 0.0025, 0.005])
    kind = rng.choice(["run"] * 4 + ["ens", "adj"])
    if kind == "run":
        n = rng.choice([16, 32, 64, 64, 128, 128, 256, 256, 512])
        most = max(1, min(60, int(6 * 512 ** 3 / n ** 3 / share)))
        return {"kind": "run", "n": n, "precision": prec, "steps": log_int(1, most), "nu": nu, "dt": dt,
                "fresh": rng.random() < 0.3, "pressure": rng.random() < 0.3}
    if kind == "ens":
        n, n2 = rng.choice([(32, 64), (64, 128), (16, 64)])
        return {"kind": "ens", "n": n, "runs": log_int(1, 24), "n2": n2, "runs2": log_int(1, 9),
                "precision": prec, "steps": log_int(1, 20), "dt": dt}
    n = rng.choice([16, 32, 64, 128])
    return {"kind": "adj", "n": n, "precision": prec, "steps": log_int(2, 20 if n == 128 else 40),
            "snapshots": log_int(1, 12), "nu": nu, "dt": dt}


# ---------------------------------------------------------------- inputs


def _wave(n, device):
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=device)
    kz = torch.arange(n // 2 + 1, dtype=torch.float64, device=device)
    return k.view(n, 1, 1), k.view(1, n, 1), kz.view(1, 1, -1)


def _field(n, seed, amplitude=0.05):
    """Taylor-Green plus a solenoidal perturbation of `amplitude` times its
    rms: float64 [3][n][n][n] on the GPU."""
    dev = torch.device("cuda")
    x = 2 * math.pi / n * torch.arange(n, dtype=torch.float64, device=dev)
    s, c = torch.sin(x), torch.cos(x)
    kx, ky, kz = _wave(n, dev)
    kk = kx ** 2 + ky ** 2 + kz ** 2
    amp = torch.sqrt(kk) * torch.exp(-kk / 16.0)
    amp[n // 2], amp[:, n // 2], amp[:, :, n // 2] = 0, 0, 0
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    hats = [torch.fft.rfftn(torch.randn((n, n, n), generator=gen, dtype=torch.float64, device=dev)) * amp
            for _ in range(3)]
    div = (kx * hats[0] + ky * hats[1] + kz * hats[2]) / torch.where(kk > 0, kk, torch.ones_like(kk))
    u = torch.stack([torch.fft.irfftn(h - k * div, s=(n, n, n)) for h, k in zip(hats, (kx, ky, kz))])
    u *= amplitude * 0.5 / math.sqrt(float(u.square().sum()) / n ** 3)
    u[0] += s.view(n, 1, 1) * c.view(1, n, 1) * c.view(1, 1, n)
    u[1] -= c.view(n, 1, 1) * s.view(1, n, 1) * c.view(1, 1, n)
    return u


def _sizes(case):
    return [case["n"]] * case["runs"] + [case["n2"]] * case["runs2"]


def _viscosities(case, seed):
    rng = np.random.default_rng(seed)
    return np.exp(rng.uniform(math.log(1 / 3000), math.log(1 / 100), case["runs"] + case["runs2"]))


def _prec(case):
    return FP64 if case["precision"] == "fp64" else MIXED


class _Handle:
    """A handle of the C library, given back with the object."""

    def __init__(self, create, destroy, *args):
        self.lib = dns_b200.load_library()
        self.destroy = getattr(self.lib, destroy)
        self.h = ctypes.c_void_p()
        self.call(create, *args, ctypes.byref(self.h), plain=True)

    def call(self, name, *args, plain=False):
        st = getattr(self.lib, name)(*(args if plain else (self.h, *args)))
        if st != dns_b200.DNS_OK:
            raise dns_b200.DNSError(st, self.lib.dns_last_error().decode())

    def __del__(self):
        if getattr(self, "h", None):
            self.destroy(self.h)
            self.h = None


def _at(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    prec = _prec(case)
    n = case["n"]
    if case["kind"] == "run":
        flags = dns_b200.DNS_FLAG_PRESSURE if case["pressure"] else 0
        ctx = _Handle("dns_create", "dns_destroy", n, prec, flags)
        fields = torch.empty((4 if case["pressure"] else 3, n, n, n), dtype=torch.float64, pin_memory=True)
        fields[:3].copy_(_field(n, seed))
        ctx.call("dns_set_velocity", *[_at(fields[f]) for f in range(3)])
        kept = torch.empty(fields.shape, dtype=torch.float32) if prec == MIXED else None
        first = fields[:3].clone().pin_memory() if case["fresh"] else None
        return {"case": case, "ctx": ctx, "fields": fields, "kept": kept, "first": first}
    if case["kind"] == "ens":
        sizes = _sizes(case)
        ens = _Handle("dns_ens_create", "dns_ens_destroy", len(sizes), (ctypes.c_long * len(sizes))(*sizes), prec, 0)
        for r, m in enumerate(sizes):
            u = _field(m, seed * 1000 + r).cpu()
            ens.call("dns_ens_set_velocity", r, *[_at(u[f]) for f in range(3)])
        nu, dt = _viscosities(case, seed), np.full(len(sizes), case["dt"])
        ens.call("dns_ens_set_params", nu.ctypes.data, dt.ctypes.data)
        spectra = [torch.empty((k, 3, m, m, m // 2 + 1), dtype=torch.complex128, pin_memory=True)
                   for m, k in ((n, case["runs"]), (case["n2"], case["runs2"]))]
        kept = [torch.empty(s.shape, dtype=torch.complex64) for s in spectra] if prec == MIXED else None
        return {"case": case, "ens": ens, "spectra": spectra, "kept": kept, "sums": np.empty(4 * len(sizes))}
    u = _field(n, seed).cpu().numpy()
    return {"case": case, "u": [u[f] for f in range(3)]}


# ---------------------------------------------------------------- one pass


def run(state):
    case = state["case"]
    if case["kind"] == "run":
        ctx, fields = state["ctx"], state["fields"]
        if case["fresh"]:
            ctx.call("dns_set_velocity", *[_at(state["first"][f]) for f in range(3)])
        ctx.call("dns_step", case["nu"], case["dt"], case["steps"])
        v = [ctypes.c_double() for _ in range(4)]
        ctx.call("dns_diagnostics", *[ctypes.byref(x) for x in v])
        E, Om = dns_b200.scale_diagnostics(*[x.value for x in v], case["n"])
        ctx.call("dns_get_fields", *[_at(f) for f in fields], *[None] * (4 - len(fields)))
        if state["kept"] is not None:
            fields = state["kept"].copy_(fields)
        return {"E": float(E), "Om": float(Om), "fields": fields}
    if case["kind"] == "ens":
        ens, sums = state["ens"], state["sums"]
        ens.call("dns_ens_step", case["steps"])
        ens.call("dns_ens_diagnostics", sums.ctypes.data)
        run_ = 0
        for s in state["spectra"]:
            for q in range(len(s)):
                ens.call("dns_ens_get_spectral", run_, _at(s[q]))
                run_ += 1
        spectra = state["spectra"]
        if state["kept"] is not None:
            spectra = [k.copy_(s) for k, s in zip(state["kept"], spectra)]
        d = [dns_b200.scale_diagnostics(*sums[4 * r:4 * r + 4], m) for r, m in enumerate(_sizes(case))]
        d = np.array(d, dtype=np.float64)
        return {"diagnostics": d if state["kept"] is None else d.astype(np.float32), "spectra": spectra}
    J, g, gnu = dns_b200.adjoint_energy(*state["u"], case["nu"], case["dt"], case["steps"],
                                        case["snapshots"], _prec(case))
    g = [a if case["precision"] == "fp64" else a.astype(np.float32) for a in g]
    return {"J": J, "grad": g, "grad_nu": gnu}


# ---------------------------------------------------------------- what it takes


def work(case):
    """Bytes: every step reads its state (three half spectra and the real
    velocity that the first stage takes over) and writes the next one, and
    what is loaded and dumped moves once more.  Operations: nine real 3-D
    transforms and about 120 operations a point for each of the four stages."""
    def step(n, size):
        state = 3 * (2 * n * n * (n // 2 + 1) + n ** 3) * size
        return 2 * state, 4 * (9 * 2.5 * n ** 3 * math.log2(n ** 3) + 120 * n ** 3 / 2)

    size = 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "run":
        b, f = step(case["n"], size)
        moved = (3 + case["pressure"] + 3 * case["fresh"]) * 8 * case["n"] ** 3
        return {"bytes": case["steps"] * b + moved, "flops": case["steps"] * f}
    if case["kind"] == "ens":
        per = [step(m, size) for m in _sizes(case)]
        moved = sum(3 * 16 * m * m * (m // 2 + 1) for m in _sizes(case))
        return {"bytes": case["steps"] * sum(p[0] for p in per) + moved,
                "flops": case["steps"] * sum(p[1] for p in per)}
    # a gradient: every step forward once and its transposed step, which
    # carries the same fields back and transforms as many
    b, f = step(case["n"], size)
    return {"bytes": 3 * case["steps"] * b + 6 * 8 * case["n"] ** 3, "flops": 3 * case["steps"] * f}


# ---------------------------------------------------------------- in 64 bits


class _Exact:
    """main.c's step in torch's float64."""

    def __init__(self, u):
        self.n = n = u.shape[1]
        self.kx, self.ky, self.kz = _wave(n, u.device)
        self.kk = self.kx ** 2 + self.ky ** 2 + self.kz ** 2
        kmax = 2.0 / 3.0 * (n // 2 + 1)
        self.mask = ((self.kx.abs() < kmax) & (self.ky.abs() < kmax) & (self.kz < kmax)).to(torch.float64)
        self.inv_kk = torch.where(self.kk > 0, 1.0 / self.kk, torch.zeros_like(self.kk))
        self.uh = torch.stack([self.forward(a) for a in u])
        self.stale = u.clone()
        self.p = torch.zeros_like(self.uh[0])

    def forward(self, a):
        return torch.fft.rfftn(a, dim=(0, 1, 2))

    def back(self, X):
        """FFTW's c2r over n^3: complex over x and y, then real along z."""
        Y = torch.fft.ifft(torch.fft.ifft(X, dim=0), dim=1)
        return torch.fft.irfft(Y, n=self.n, dim=2)

    def slope(self, us, u, nu, dt):
        kx, ky, kz = self.kx, self.ky, self.kz
        w = [self.back(1j * (ky * us[2] - kz * us[1])), self.back(1j * (kz * us[0] - kx * us[2])),
             self.back(1j * (kx * us[1] - ky * us[0]))]
        d = [self.forward(u[1] * w[2] - u[2] * w[1]), self.forward(u[2] * w[0] - u[0] * w[2]),
             self.forward(u[0] * w[1] - u[1] * w[0])]
        d = [a * (self.mask * dt) for a in d]
        p = (kx * d[0] + ky * d[1] + kz * d[2]) * self.inv_kk
        self.p = p
        return torch.stack([a - p * k - nu * dt * self.kk * b for a, k, b in zip(d, (kx, ky, kz), us)])

    def step(self, nu, dt):
        u0 = self.uh
        us, acc, u = u0, u0.clone(), self.stale
        for s in range(4):
            if s > 0:
                u = torch.stack([self.back(a) for a in us])
            d = self.slope(us, u, nu, dt)
            acc += (1 / 6, 1 / 3, 1 / 3, 1 / 6)[s] * d
            if s < 3:
                us = u0 + (0.5, 0.5, 1.0)[s] * d
        self.uh, self.stale = acc, u

    def diagnostics(self):
        e = self.uh.abs().square().sum(0)
        return float(e.sum()) / self.n ** 6, float((self.kk * e).sum()) / self.n ** 6


def _gradient(u, nu, dt, steps):
    """J and its gradient by torch's own reverse mode over _Exact's step,
    one step at a time from stored states."""
    ex = _Exact(u)
    states = [(ex.uh, ex.stale)]
    for _ in range(steps):
        ex.step(nu, dt)
        states.append((ex.uh, ex.stale))
    n = ex.n
    J, _ = ex.diagnostics()
    bar_uh, bar_stale = 2.0 * states[-1][0] / n ** 6, torch.zeros_like(u)
    gnu = 0.0
    for uh, stale in reversed(states[:-1]):
        with torch.enable_grad():
            ex.uh, ex.stale = uh.clone().requires_grad_(), stale.clone().requires_grad_()
            nu_t = torch.tensor(nu, dtype=torch.float64, device=u.device, requires_grad=True)
            inputs = (ex.uh, ex.stale, nu_t)
            ex.step(nu_t, dt)
            bar_uh, bar_stale, b = torch.autograd.grad((ex.uh, ex.stale), inputs, (bar_uh, bar_stale))
        gnu += float(b)
    with torch.enable_grad():
        v = u.clone().requires_grad_()
        (g,) = torch.autograd.grad(torch.stack([ex.forward(a) for a in v]), v, bar_uh)
    return J, g + bar_stale, gnu


@torch.no_grad()
def exact(case, seed):
    n = case["n"]
    if case["kind"] == "run":
        ex = _Exact(_field(n, seed))
        for _ in range(case["steps"]):
            ex.step(case["nu"], case["dt"])
        E, Om = ex.diagnostics()
        out = torch.stack([ex.back(a) for a in list(ex.uh) + ([ex.p] if case["pressure"] else [])])
        return {"E": E, "Om": Om, "fields": out}
    if case["kind"] == "ens":
        nu, d, spectra = _viscosities(case, seed), [], [[], []]
        for r, m in enumerate(_sizes(case)):
            ex = _Exact(_field(m, seed * 1000 + r))
            for _ in range(case["steps"]):
                ex.step(float(nu[r]), case["dt"])
            d.append(ex.diagnostics())
            spectra[0 if r < case["runs"] else 1].append(ex.uh.cpu())
        return {"diagnostics": np.array(d), "spectra": [torch.stack(s) for s in spectra]}
    J, g, gnu = _gradient(_field(n, seed), case["nu"], case["dt"], case["steps"])
    return {"J": J, "grad": list(g.cpu().numpy()), "grad_nu": gnu}
