"""Timed cases of the framework: whole calls of its public entry points as a
user's program makes them, over the sizes (powers of two, 16..2048),
precisions, integrators and options it is run with.

A case's "kind" names the program it stands for:

  steps     w_hat set from the device, a fixed-dt run (ns2d_step_n), w_hat read
            back to the device: RK4CN, explicit RK4 or AB4, 2/3 or Hou-Li
            dealiasing, unforced or Kolmogorov forced.
  adaptive  the CFL loop of SpectralSolve: get_timestep, rk4_step, repeated.
  dp5       Dormand-Prince 5(4) with the caller's step-size control.
  host      RK4Step on a host-resident state (the drop-in form): copy in, step,
            copy out, every step.
  rhs       NonlinearRHSBatch on host arrays (the drop-in form, and what the
            post-processing evaluates for every snapshot).
  measures  ComputeSystemMeasurables at a save point: totals and spectra with
            the flux terms.
  ensemble  members of uneven sizes advanced together.
  adjoint   the gradient of the final enstrophy with respect to the initial
            vorticity (checkpointed reverse sweep).

FP32 runs hand their results back as complex64: that is the precision they
carry.  The linear-operator and quirk settings are the defaults of the
reference's command line unless a case says otherwise.
"""
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "2d-navier-stokes_b200"))

from ns2d import Ensemble, Solver, abi  # noqa: E402

_INTEGRATORS = {"rk4cn": abi.RK4CN, "rk4": abi.RK4, "ab4": abi.AB4, "dp5": abi.DP5}
_SIZES = (16, 32, 64, 128, 256, 512, 1024, 2048)


def listed():
    return [
        # the drop-in's NonlinearRHS call on a small grid: launches, copies and the host path
        {"name": "rhs_64_fp64", "kind": "rhs", "n": 64, "fp32": False},
        # Taylor-Green check run: 64^2, FP64, explicit RK4, 100 steps of 1e-3
        {"name": "taylor_green_64_fp64_rk4", "kind": "steps", "n": 64, "fp32": False, "integrator": "rk4",
         "dealias": "2/3", "flow": "taylor_green", "steps": 100},
        # the stock build (RK4CN, 2/3) on a small grid, between two saves
        {"name": "decaying_128_fp64_rk4cn", "kind": "steps", "n": 128, "fp32": False, "integrator": "rk4cn",
         "dealias": "2/3", "flow": "decaying", "steps": 75},
        # decaying turbulence with the Hou-Li filter and the CFL step: 256^2, FP64
        {"name": "cfl_256_fp64_houli", "kind": "adaptive", "n": 256, "fp32": False, "dealias": "houli", "steps": 25},
        # error-controlled integration of the same flow, 2/3 rule
        {"name": "dp5_256_fp64", "kind": "dp5", "n": 256, "fp32": False, "steps": 7},
        # Kolmogorov flow with implicit hyperviscosity, the headline workload: 1024^2, FP64 and FP32
        {"name": "kolmogorov_1024_fp64_rk4cn", "kind": "steps", "n": 1024, "fp32": False, "integrator": "rk4cn",
         "dealias": "2/3", "flow": "kolmogorov", "steps": 40},
        {"name": "kolmogorov_1024_fp32_rk4cn", "kind": "steps", "n": 1024, "fp32": True, "integrator": "rk4cn",
         "dealias": "2/3", "flow": "kolmogorov", "steps": 40},
        # the largest grid, stock build
        {"name": "decaying_2048_fp64_rk4cn", "kind": "steps", "n": 2048, "fp32": False, "integrator": "rk4cn",
         "dealias": "2/3", "flow": "decaying", "steps": 15},
        # the headline workload stepped on the caller's host array
        {"name": "host_step_1024_fp64", "kind": "host", "n": 1024, "fp32": False, "steps": 3},
        # a save point of a 1024^2 run
        {"name": "measures_1024_fp64", "kind": "measures", "n": 1024, "fp32": False},
        # 64 uneven members in FP32, tuned, between two saves of all members
        {"name": "ensemble_64_fp32", "kind": "ensemble", "n128": 32, "n256": 24, "n512": 8, "n64": 0, "fp32": True,
         "steps": 250},
        # one gradient of the extreme-enstrophy search, a tenth of its horizon
        {"name": "adjoint_512_fp64", "kind": "adjoint", "n": 512, "fp32": False, "steps": 200, "every": 50},
    ]


def _cost(case):
    """Rough size of a case: grid points advanced by one step."""
    k = case["kind"]
    if k == "ensemble":
        return case["steps"] * sum(case["n%d" % n] * n * n for n in (64, 128, 256, 512))
    return case["n"] ** 2 * case.get("steps", 1) * (4 if k == "adjoint" else 2 if k == "dp5" else 1)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("steps", "steps", "steps", "adaptive", "dp5", "host", "rhs", "measures", "ensemble",
                           "adjoint"))
        fp32 = rng.random() < 0.4
        n = rng.choice(_SIZES)
        if kind == "steps":
            case = {"kind": kind, "n": n, "fp32": fp32, "integrator": rng.choice(("rk4cn", "rk4cn", "rk4", "ab4")),
                    "dealias": rng.choice(("2/3", "2/3", "houli")),
                    "flow": rng.choice(("decaying", "kolmogorov")) if n >= 64 else "decaying",
                    "steps": int(10 ** rng.uniform(0.7, 2.0))}
            if case["dealias"] == "houli":
                case["flow"] = "decaying"
        elif kind == "adaptive":
            case = {"kind": kind, "n": n, "fp32": fp32, "dealias": rng.choice(("2/3", "houli")),
                    "steps": rng.randint(5, 40)}
        elif kind == "dp5":
            case = {"kind": kind, "n": n, "fp32": False, "steps": rng.randint(3, 20)}
        elif kind == "host":
            case = {"kind": kind, "n": n, "fp32": fp32, "steps": rng.randint(1, 20)}
        elif kind in ("rhs", "measures"):
            case = {"kind": kind, "n": n, "fp32": fp32}
        elif kind == "ensemble":
            case = {"kind": kind, "fp32": rng.random() < 0.7, "steps": rng.randint(20, 250)}
            for m, top in ((64, 16), (128, 16), (256, 12), (512, 6)):
                case["n%d" % m] = rng.randint(0, top)
            if not 2 <= sum(case["n%d" % m] for m in (64, 128, 256, 512)) <= 64:
                continue
        else:
            every = rng.randint(5, 50)
            case = {"kind": kind, "n": rng.choice((64, 128, 256, 512)), "fp32": fp32,
                    "steps": rng.randint(every, 4 * every), "every": every}
        if _cost(case) <= most and (kind == "ensemble" or case["n"] >= 32 or kind in ("steps", "host", "rhs")):
            return case


# ---------------------------------------------------------------------------
# parameters and inputs


def _dt(case):
    if case["kind"] == "adjoint":
        return 5e-4
    if case.get("flow") == "kolmogorov" or case["kind"] == "host":
        return 2.5e-4
    return 1e-3 if case.get("n", 512) <= 512 else 2.5e-4


def _params(case):
    kind = case["kind"]
    n = case.get("n", 64)
    p = dict(nx=n, ny=n, precision=abi.FP32 if case["fp32"] else abi.FP64, dt=_dt(case))
    if kind == "adjoint":
        return abi.default_params(nu=1e-3, quirks=0, **p)
    if kind == "ensemble":
        return abi.default_params(nu=1e-3, **p)
    if kind == "adaptive":
        return abi.default_params(nu=5e-4, adapt_step_flag=1, cfl_cond_flag=1, cfl_const=0.9,
                                  ekmn_drag_flag=1, ekmn_alpha=0.0, ekmn_drag_pow=0.0,
                                  dealias=abi.DEALIAS_HOU_LI if case["dealias"] == "houli" else abi.DEALIAS_23, **p)
    # nu |k|^2 alone: the drag branch with no drag
    plain = dict(nu=1e-3, ekmn_drag_flag=1, ekmn_alpha=0.0, ekmn_drag_pow=0.0)
    if kind == "dp5":
        return abi.default_params(integrator=abi.DP5, **plain, **p)
    flow = case.get("flow", "kolmogorov" if kind == "host" else "decaying")
    if flow == "kolmogorov":
        # hyperviscosity |k|^16 through the drag branch, scaled with the grid
        plain = dict(nu=1e-4, ekmn_drag_flag=1, ekmn_alpha=2e-40 * (1024.0 / n) ** 16, ekmn_drag_pow=8.0,
                     forcing=abi.FORCING_KOLM, force_k=4, force_scale=1.0)
    elif flow == "taylor_green":
        plain["nu"] = 0.01
    integ = _INTEGRATORS[case.get("integrator", "rk4cn")]
    return abi.default_params(integrator=integ, dealias=abi.DEALIAS_HOU_LI if case.get("dealias") == "houli"
                              else abi.DEALIAS_23, **plain, **p)


def _waves(n):
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda").round()
    k[n // 2] = n // 2
    return k[:, None], torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda")[None, :]


def _keep(n, p):
    """Modes the dealiasing keeps (2/3 rule), as a mask; Hou-Li: its factors."""
    kx, ky = _waves(n)
    if p.dealias == abi.DEALIAS_23:
        m = int(n / 3.0)
        keep = (kx * kx + ky * ky) < m * m
        if p.forcing == abi.FORCING_KOLM:
            keep = keep & (kx != 0)
        return keep.to(torch.float64)
    fx, fy = torch.trunc(kx / (n // 2)), torch.trunc(ky / (n // 2))
    return torch.exp(-36.0 * (fx * fx + fy * fy) ** 18)


def _spectrum(n, gen, shape, dealias, vort_rms=None):
    """Random-phase vorticity [n][n/2+1] with amplitudes shape(|k|), Hermitian on ky = 0 and n/2."""
    kx, ky = _waves(n)
    k2 = kx * kx + ky * ky
    phase = 2.0 * np.pi * torch.rand(n, n // 2 + 1, dtype=torch.float64, device="cuda", generator=gen)
    w = torch.polar(shape(torch.sqrt(k2)), phase)
    for j in (0, n // 2):
        col = w[:, j].clone()
        col[n // 2 + 1:] = torch.conj(col[1:n // 2]).flip(0)
        col[0], col[n // 2] = col[0].real.clone(), col[n // 2].real.clone()
        w[:, j] = col
    w[0, 0] = 0.0
    if dealias:
        m = int(n / 3.0)
        w = w * (k2 < m * m)
    c = torch.full((1, n // 2 + 1), 2.0, dtype=torch.float64, device="cuda")
    c[0, 0] = c[0, -1] = 1.0
    if vort_rms is not None:
        return w * (vort_rms * n * n / torch.sqrt((c * w.abs() ** 2).sum()))
    k2[0, 0] = 1.0
    energy = 4.0 * np.pi ** 2 * 0.5 / float(n * n) ** 2 * (c * w.abs() ** 2 / k2).sum()
    return w * torch.sqrt(0.5 / energy)


def _decaying(n, gen, k0, dealias):
    """Energy spectrum k^4 exp(-(k/k0)^2), total energy 0.5."""
    return _spectrum(n, gen, lambda k: torch.sqrt(k ** 5 * torch.exp(-(k / k0) ** 2) / (2.0 * np.pi)), dealias)


def _w0(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    n = case["n"]
    flow = case.get("flow", "kolmogorov" if case["kind"] == "host" else "decaying")
    if flow == "taylor_green":
        # 2 sin(x) sin(y) with a seeded amplitude
        a = 1.0 + 0.1 * float(torch.rand((), dtype=torch.float64, device="cuda", generator=gen))
        w = torch.zeros(n, n // 2 + 1, dtype=torch.complex128, device="cuda")
        w[1, 1], w[n - 1, 1] = -0.5 * n * n * a, 0.5 * n * n * a
        return w
    if flow == "kolmogorov":
        # low-amplitude noise on the modes 1 <= |k| <= 8, kx = 0 removed
        w = _spectrum(n, gen, lambda k: ((k >= 1) & (k <= 8)).to(torch.float64), True, vort_rms=1e-3)
        w[0, :] = 0.0
        return w
    return _decaying(n, gen, max(2.0, min(6.0, n / 16.0)), case.get("dealias") != "houli")


def _members(case):
    return [n for n in (128, 256, 512, 64) for _ in range(case["n%d" % n])]


def _member_w0(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    sizes = _members(case)
    pick = torch.randint(0, 3, (len(sizes),), device="cuda", generator=gen).tolist()
    return [_decaying(n, gen, (4.0, 6.0, 8.0)[k], True) for n, k in zip(sizes, pick)]


# ---------------------------------------------------------------------------
# the passes


class _Pinned:
    """A page-locked host array [n][n/2+1] complex128 holding w."""

    def __init__(self, w):
        self.t = torch.view_as_real(w).cpu().pin_memory()
        self.a = self.t.numpy().view(np.complex128)[..., 0]


def prepare(case, seed):
    st = {"case": case, "dt": _dt(case)}
    kind = case["kind"]
    p = _params(case)
    if kind == "ensemble":
        st["w0"] = [w.cpu().numpy() for w in _member_w0(case, seed)]
        st["e"] = Ensemble(p, _members(case))
        st["e"].tune(st["dt"])
        return st
    w0 = _w0(case, seed)
    st["s"] = Solver(p)
    if kind in ("steps", "adaptive", "dp5"):
        st["w0"], st["out"] = w0, torch.empty_like(w0)
        torch.cuda.synchronize()
    elif kind == "host":
        st["w"] = _Pinned(w0)
    elif kind == "rhs":
        st["s"].compute_forcing(st["dt"])
        st["w"] = _Pinned(w0)
    elif kind == "measures":
        st["s"].set_w_hat(w0.cpu().numpy())
    else:
        st["w0"] = w0.cpu().numpy()
    return st


def _device_result(st):
    s = st["s"]
    s.get_w_hat_device(st["out"].data_ptr())
    s.synchronize()
    return st["out"].to(torch.complex64) if st["case"]["fp32"] else st["out"]


def run(st):
    case, dt = st["case"], st["dt"]
    kind = case["kind"]
    single = np.complex64 if case["fp32"] else np.complex128
    if kind == "ensemble":
        e = st["e"]
        for m, w in enumerate(st["w0"]):
            e.set_w_hat(m, w)
        e.step_n(case["steps"], dt)
        return [e.get_w_hat(m).astype(single, copy=False) for m in range(len(st["w0"]))]
    s = st["s"]
    if kind == "steps":
        s.set_w_hat_device(st["w0"].data_ptr())
        s.step_n(case["steps"], dt)
        return _device_result(st)
    if kind == "adaptive":
        s.set_w_hat_device(st["w0"].data_ptr())
        t = 0.0
        for _ in range(case["steps"]):
            dt = s.get_timestep(dt)
            s.rk4_step(dt)
            t += dt
        return {"w_hat": _device_result(st), "time": torch.tensor(t, dtype=torch.float32 if case["fp32"] else torch.float64)}
    if kind == "dp5":
        s.set_w_hat_device(st["w0"].data_ptr())
        t = 0.0
        for _ in range(case["steps"]):
            err = s.dp5_step(dt)
            t += dt
            dt *= min(1.5, max(0.5, 0.8 * err ** -0.2)) if err > 0.0 else 1.5
        return {"w_hat": _device_result(st), "time": torch.tensor(t, dtype=torch.float64)}
    if kind == "host":
        for _ in range(case["steps"]):
            s.rk4_step_host(st["w"].a, dt)
        return st["w"].a.astype(single, copy=False)
    if kind == "rhs":
        return s.nonlinear_rhs(st["w"].a).astype(single, copy=False)
    if kind == "measures":
        totals, spectra = s.system_measurables()
        return {"totals": totals.astype(np.float32 if case["fp32"] else np.float64, copy=False),
                "spectra": spectra.astype(np.float32 if case["fp32"] else np.float64, copy=False)}
    s.set_w_hat(st["w0"])
    value, grad = s.adjoint_gradient(case["steps"], dt, case["every"])
    return {"value": torch.tensor(value, dtype=torch.float32 if case["fp32"] else torch.float64),
            "gradient": grad.astype(single, copy=False)}


# ---------------------------------------------------------------------------
# the work of a pass: transforms of the scheme (a real 2-D transform of n^2
# points is 2.5 n^2 log2 n^2 operations, five per evaluation of the nonlinear
# term), and its inputs and results once each


def work(case):
    kind = case["kind"]
    size = 4 if case["fp32"] else 8

    def rhs(n):
        return 5 * 2.5 * n * n * 2 * (n.bit_length() - 1)

    if kind == "ensemble":
        points = sum(n * (n // 2 + 1) for n in _members(case))
        return {"bytes": 2 * 16 * points, "flops": case["steps"] * 4 * sum(rhs(n) for n in _members(case))}
    n = case["n"]
    field = n * (n // 2 + 1)
    if kind == "measures":
        return {"bytes": 2 * size * field, "flops": rhs(n) + 40.0 * field}
    if kind == "rhs":
        return {"bytes": 32 * field, "flops": rhs(n)}
    steps = case["steps"]
    if kind == "host":
        return {"bytes": 32 * field * steps, "flops": 4 * rhs(n) * steps}
    if kind == "adaptive":
        return {"bytes": 32 * field, "flops": steps * (4 + 0.4) * rhs(n)}
    if kind == "dp5":
        return {"bytes": 32 * field, "flops": steps * 7 * rhs(n)}
    if kind == "adjoint":
        # forward, and per adjoint stage one inverse and four forward transforms
        return {"bytes": 32 * field, "flops": steps * 2 * 4 * rhs(n)}
    per_step = 1 if case["integrator"] == "ab4" else 4
    return {"bytes": 32 * field, "flops": steps * per_step * rhs(n)}


# ---------------------------------------------------------------------------
# 64-bit values: the scheme with torch.fft in double precision.  Fields may
# carry a leading batch dimension.


class _Exact:
    def __init__(self, p, n):
        self.p, self.n = p, n
        self.kx, self.ky = _waves(n)
        k2 = self.kx ** 2 + self.ky ** 2
        self.k2 = k2
        self.inv = torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, 1.0), 0.0)
        self.keep = _keep(n, p)
        self.keep[0, 0] = 0.0
        self.hyper = p.hyper_visc_flag

    def force(self, r):
        if self.p.forcing == abi.FORCING_KOLM:
            k = self.p.force_k
            r = r.clone()
            r[..., k // (self.n // 2 + 1), k % (self.n // 2 + 1)] += -0.5 * self.p.force_scale * k
        return r

    def real(self, f):
        x = torch.fft.ifft(f, dim=-2, norm="forward")
        return torch.fft.irfft(x, n=self.n, dim=-1, norm="forward")

    def rhs(self, X, forced=True):
        i = 1j
        prod = self.real(i * self.ky * self.inv * X) * self.real(i * self.kx * X)
        prod = prod + self.real(-i * self.kx * self.inv * X) * self.real(i * self.ky * X)
        r = torch.fft.fft(torch.fft.rfft(prod, dim=-1), dim=-2) * (self.keep / float(self.n) ** 4)
        return self.force(r) if forced else r

    def conj(self, w, X):
        """ForceConjugacy: the state's kx < 0, ky = 0 modes from the evaluation's input."""
        w = w.clone()
        w[..., self.n // 2 + 1:, 0] = torch.conj(X[..., 1:self.n // 2, 0]).flip(-1)
        return w

    def bracket(self, latch):
        p = self.p
        k2 = torch.where(self.k2 > 0, self.k2, 1.0)
        if p.ekmn_drag_flag == 1 and self.hyper != 1:
            return p.nu * k2 + p.ekmn_alpha * k2 ** p.ekmn_drag_pow
        if p.ekmn_drag_flag == 1:
            return p.nu * k2 ** p.hyper_visc_pow + p.ekmn_alpha * k2 ** p.ekmn_drag_pow
        if latch and p.quirks & abi.QUIRK_HYPER_LATCH:
            self.hyper = 1
        return p.nu * k2 ** p.hyper_visc_pow if self.hyper == 1 else p.nu * k2

    def cn(self, dt, latch=True):
        D = dt * self.bracket(latch)
        a, b = (2.0 - D) / (2.0 + D), 2.0 * dt / (2.0 + D)
        a[0, 0] = b[0, 0] = 0.0
        return a, b

    def rk4(self, w, dt, explicit=False, first=None):
        quirk = bool(self.p.quirks & abi.QUIRK_CONJ_STATE)
        br = self.bracket(True) * (self.k2 > 0) if explicit else None
        a, b = (None, None) if explicit else self.cn(dt)
        X, acc = w, 0.0
        for s in range(4):
            r = self.rhs(X)
            if quirk:
                w = self.conj(w, X)
            if s == 0 and first is not None:
                first.append(r)
            if explicit:
                xs = w if s == 0 else X
                r = r + dt * br * xs if self.p.quirks & abi.QUIRK_RK4_LINEAR else r - br * xs
                acc = acc + (1.0, 2.0, 2.0, 1.0)[s] * r
            else:
                acc = acc + (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)[s] * r
            if s < 3:
                X = w + (0.5, 0.5, 1.0)[s] * dt * r
        if explicit:
            w = w + dt / 6.0 * acc
            w[..., 0, 0] = 0.0
            return w
        return a * w + b * acc

    def ab4(self, w, dt, hist):
        if len(hist) < 3:
            return self.rk4(w, dt, first=hist)
        r = self.rhs(w)
        w = self.conj(w, w)
        tot = 55.0 / 24.0 * r - 59.0 / 24.0 * hist[-1] + 37.0 / 24.0 * hist[-2] - 3.0 / 8.0 * hist[-3]
        a, b = self.cn(dt, latch=False)
        hist.append(r)
        hist.pop(0)
        return a * w + b * tot

    _DP_A = ((), (0.2,), (3.0 / 40.0, 9.0 / 40.0), (44.0 / 45.0, -56.0 / 15.0, 32.0 / 9.0),
             (19372.0 / 6561.0, -25360.0 / 2187.0, 64448.0 / 6561.0, -212.0 / 729.0),
             (9017.0 / 3168.0, -355.0 / 33.0, 46732.0 / 5247.0, 49.0 / 176.0, -5103.0 / 18656.0),
             (35.0 / 384.0, 0.0, 500.0 / 1113.0, 125.0 / 192.0, -2187.0 / 6784.0, 11.0 / 84.0))
    _DP_5 = (35.0 / 384.0, 0.0, 500.0 / 1113.0, 125.0 / 192.0, -2187.0 / 6784.0, 11.0 / 84.0, 0.0)
    _DP_4 = (5179.0 / 57600.0, 0.0, 7571.0 / 16695.0, 393.0 / 640.0, -92097.0 / 339200.0, 187.0 / 2100.0, 1.0 / 40.0)

    def dp5(self, w, dt):
        br = self.bracket(False) * (self.k2 > 0)
        ks = []
        for row in self._DP_A:
            X = w + dt * sum((c * k for c, k in zip(row, ks)), torch.zeros_like(w))
            ks.append(self.rhs(X) - br * X)
        y5 = w + dt * sum(c * k for c, k in zip(self._DP_5, ks))
        y4 = w + dt * sum(c * k for c, k in zip(self._DP_4, ks))
        e = (y5 - y4).abs() / (1e-7 + 1e-7 * torch.maximum(w.abs(), y5.abs()))
        e[0, 0] = 0.0
        y5[0, 0] = 0.0
        return y5, float(torch.sqrt((e * e).sum() / e.numel()))

    def cfl(self, w, keep):
        """GetTimestep with the reference's row index; keep: the velocity spectra it writes into."""
        n, p = self.n, self.p
        nyf = n // 2 + 1
        i = torch.arange(n, device="cuda")[:, None]
        j = torch.arange(nyf, device="cuda")[None, :]
        last = (j == nyf - 1) & (i < n - 1)
        at = (i * n // 2 + 1 + j)[~last]
        v = w.reshape(-1)[at]
        kx, ky, inv = (t.expand(n, nyf)[~last] for t in (self.kx, self.ky, self.inv))
        keep[0][at] = 1j * ky * inv * v
        keep[1][at] = -1j * kx * inv * v
        u, v = (self.real(f.reshape(n, nyf)) / (n * n) for f in keep)
        d = 2.0 * np.pi / n
        convect = float((np.pi * (u.abs() / d + v.abs() / d)).max())
        return p.cfl_const / (convect + np.pi ** 2 * 2.0 * p.nu / d ** 2)

    def measures(self, w):
        p, n = self.p, self.n
        r = self.rhs(w, forced=False)
        w = self.conj(w, w)
        hyper, drag = self.hyper, p.ekmn_drag_flag
        k2 = torch.where(self.k2 > 0, self.k2, 1.0)
        visc = p.nu * (k2 ** p.hyper_visc_pow if hyper == 1 else k2)
        pre = visc + p.ekmn_alpha * k2 ** p.ekmn_drag_pow if drag == 1 else visc
        c = torch.full_like(k2, 2.0)
        c[:, 0] = c[:, -1] = 1.0
        c[0, 0] = 0.0
        w2 = w.abs() ** 2
        uv2 = w2 / k2
        deriv = 2.0 * (w.real * r.real + w.imag * r.imag)
        diss = pre * w2
        zdiss = torch.where(c == 2.0, 2.0 * w2, c * diss) if p.quirks & abi.QUIRK_ENST_DISS else c * diss
        div = (1j * (self.kx * (1j * self.ky * w / k2) + self.ky * (-1j * self.kx * w / k2))).abs() ** 2
        low = (self.k2 < 4096.0) * c
        norm, const = 0.5 / float(n * n) ** 2, 4.0 * np.pi ** 2
        one = const * norm
        totals = [(c * w2 / k2).sum() * one, (c * w2).sum() * one, (c * k2 * w2).sum() * one, 0.0,
                  (c * div).sum() * one, (c * pre * uv2).sum() * 2 * one, zdiss.sum() * 2 * one,
                  (low * (deriv + diss) / k2).sum(), (low * deriv / k2).sum() * one, (low * diss / k2).sum() * 2 * one,
                  (low * (deriv + diss)).sum(), (low * deriv).sum() * one, (low * diss).sum() * 2 * one]
        ns = int(round((2 * (n / 2.0) ** 2) ** 0.5 + 1))
        b = torch.round(torch.sqrt(self.k2)).long().reshape(-1)
        ok = b < ns
        spectra = []
        for q in (w2 / k2, w2, deriv + diss, deriv, diss, (deriv + diss) / k2, deriv / k2, diss / k2):
            spectra.append(torch.zeros(ns, dtype=torch.float64, device="cuda").index_add_(
                0, b[ok], (c * q).reshape(-1)[ok]) * one)
        return torch.tensor([float(t) for t in totals], dtype=torch.float64), torch.stack(spectra)

    def enstrophy(self, w):
        c = torch.full_like(self.k2, 2.0)
        c[:, 0] = c[:, -1] = 1.0
        c[0, 0] = 0.0
        return c, 4.0 * np.pi ** 2 * 0.5 / float(self.n * self.n) ** 2


def exact(case, seed):
    kind = case["kind"]
    p, dt = _params(case), _dt(case)
    if kind == "ensemble":
        sizes, w = _members(case), _member_w0(case, seed)
        for n in sorted(set(sizes)):
            at = [m for m, k in enumerate(sizes) if k == n]
            x, batch = _Exact(p, n), torch.stack([w[m] for m in at])
            for _ in range(case["steps"]):
                batch = x.rk4(batch, dt)
            for k, m in enumerate(at):
                w[m] = batch[k]
        return w
    w = _w0(case, seed)
    x = _Exact(p, case["n"])
    if kind == "steps":
        hist = []
        for _ in range(case["steps"]):
            if case["integrator"] == "ab4":
                w = x.ab4(w, dt, hist)
            else:
                w = x.rk4(w, dt, explicit=case["integrator"] == "rk4")
        return w
    if kind == "adaptive":
        t, keep = 0.0, [torch.zeros(w.numel(), dtype=torch.complex128, device="cuda") for _ in range(2)]
        for _ in range(case["steps"]):
            dt = x.cfl(w, keep)
            w = x.rk4(w, dt)
            t += dt
        return {"w_hat": w, "time": torch.tensor(t, dtype=torch.float64)}
    if kind == "dp5":
        t = 0.0
        for _ in range(case["steps"]):
            w, err = x.dp5(w, dt)
            t += dt
            dt *= min(1.5, max(0.5, 0.8 * err ** -0.2)) if err > 0.0 else 1.5
        return {"w_hat": w, "time": torch.tensor(t, dtype=torch.float64)}
    if kind == "host":
        for _ in range(case["steps"]):
            w = x.rk4(w, dt)
        return w
    if kind == "rhs":
        return x.rhs(w)
    if kind == "measures":
        totals, spectra = x.measures(w)
        return {"totals": totals, "spectra": spectra}
    # adjoint: checkpoints every few steps, each stretch differentiated by torch
    stretch, marks = 5, [w]
    for k in range(case["steps"]):
        w = x.rk4(w, dt)
        if (k + 1) % stretch == 0 or k + 1 == case["steps"]:
            marks.append(w)
    c, cz = x.enstrophy(w)
    value = (c * w.abs() ** 2).sum() * cz
    grad = 2.0 * cz * c * w
    left = case["steps"]
    for k in range(len(marks) - 2, -1, -1):
        count = left - k * stretch
        w0 = marks[k].detach().requires_grad_(True)
        v = w0
        for _ in range(count):
            v = x.rk4(v, dt)
        (grad,) = torch.autograd.grad(v, w0, grad)
        left -= count
    c[0, 0] = 1.0
    return {"value": value, "gradient": grad / c}
