"""The measured workloads of the framework: what its users run, through its public entry points.

Five kinds of call, each over the sizes, precisions and options it is used with:

* ``run``: ``run_model_scan`` / ``run_model_scan_final``, one member or an ensemble, forward only
  (modified Euler or the semi-implicit leapfrog, with or without the per-step history);
* ``gradient``: a differentiable ``run_model_scan_final`` and its ``torch.autograd`` backward, to
  the initial fields and to taurad, taudrag, DPhieq and Phibar;
* ``retrieval``: ``simulate_scan_last`` from a prepared state, differentiated in taurad and taudrag
  (what a retrieval does per sample);
* ``emission``: terminal Phi fields to map coefficients and phase curves;
* ``phase``: the simplified phase curve of Phi fields.

``exact`` restates each of them in plain torch, FP64, on the CPU.  Gradients come from torch
autograd through that restatement.
"""
import dataclasses
import functools
import math
import random

import numpy as np
import torch

from my_swampe_gb300 import emission, run_model_scan, run_model_scan_final
from my_swampe_gb300.model import RunFlags, _init_state_from_fields, build_static, simulate_scan_last

GRID = {42: (64, 128), 63: (96, 192), 106: (160, 320)}
FIELDS = ("eta", "delta", "Phi", "U", "V")
K6, ALPHA = 1.24e33, 0.01

# Planets.  "hot": the regime of the published speed benchmark.  "strong": the forced ensemble
# (strong stratification, start from rest with Phi noise).  "wasp": WASP-43b at a time step that
# only the semi-implicit scheme takes.  g is not used by the dynamics.
PLANETS = {
    "hot": dict(omega=3.2e-5, a=8.2e7, Phibar=3.0e5),
    "strong": dict(omega=3.2e-5, a=8.2e7, Phibar=4.0e6),
    "wasp": dict(omega=8.939689388812098e-05, a=71920952.0, Phibar=4.0e6),
}


def listed():
    def run(name, M, members, steps, precision, planet, dt, scheme="euler", history=False):
        return dict(name=name, kind="run", M=M, members=members, steps=steps, precision=precision, planet=planet,
                    dt=dt, scheme=scheme, history=history)

    return [
        # the first thing a user runs: one planet, default precision, with histories and diagnostics
        run("one member fp64 history", 42, 0, 240, "fp64", "hot", 120.0, history=True),
        # the same planet with the fast precision, final state only: a long run of small steps
        run("one member fast", 42, 0, 1200, "fast", "hot", 120.0),
        # a small parameter study in the default precision
        run("ensemble 16 fp64", 42, 16, 120, "fp64", "strong", 30.0),
        # the published benchmark's ensemble
        run("ensemble 64 fast", 42, 64, 240, "fast", "strong", 30.0),
        # finer grids, with member counts that are no multiple of a tile
        run("ensemble 37 fast T63", 63, 37, 120, "fast", "strong", 20.0),
        run("ensemble 21 fast T106", 106, 21, 48, "fast", "strong", 12.0),
        # one day of WASP-43b at the semi-implicit scheme's time step
        run("ensemble 32 fast implicit", 42, 32, 72, "fast", "wasp", 1200.0, scheme="semi"),
        # calibration of one planet: a gradient in the default precision
        dict(name="gradient fp64", kind="gradient", M=42, members=1, steps=48, precision="fp64", planet="strong",
             dt=30.0),
        # the headline workload, shortened: an ensemble's gradient, fast precision
        dict(name="gradient 256 fast", kind="gradient", M=42, members=256, steps=240, precision="fast",
             planet="strong", dt=30.0),
        # one draw of a few chains of a retrieval
        dict(name="retrieval 8 fast", kind="retrieval", M=42, members=8, steps=48, precision="fast", planet="hot",
             dt=600.0),
        # the emission stage of an ensemble: 121 coefficients (degree 10), one 4.5 micron band
        dict(name="emission 256", kind="emission", M=42, members=256, coefficients=121, times=200, bands=1),
        # the smallest call: the simplified phase curve of one map
        dict(name="phase curve", kind="phase", M=42, members=1, phases=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "gradient", "retrieval", "emission", "phase"))
    if kind == "emission":
        return dict(kind=kind, M=rng.choice((42, 63)), members=_log_int(rng, 1, 200),
                    coefficients=rng.choice((36, 64, 100, 121)), times=_log_int(rng, 20, 200),
                    bands=rng.choice((0, 1, 2)))
    if kind == "phase":
        return dict(kind=kind, M=rng.choice((42, 63, 106)), members=_log_int(rng, 1, 24), phases=_log_int(rng, 10, 150))
    # M = 106 runs in the fast precision only: the reference's FP64 projection amplifies its
    # damaged basis there (finite for some 100 steps), so nobody integrates it
    precision = rng.choice(("fp64", "fast"))
    M = rng.choice((42, 42, 63) if precision == "fp64" or kind == "retrieval" else (42, 42, 63, 106))
    size = (M / 42.0) ** 3
    most = (64 if kind == "gradient" else 1920) if precision == "fp64" else (2400 if kind == "retrieval" else 24000)
    hi = {"gradient": 48, "retrieval": 16, "run": 48}[kind]
    members = _log_int(rng, 1, min(hi, 6) if precision == "fp64" and kind != "run" else hi)
    if kind == "retrieval":
        return dict(kind=kind, M=M, members=members, steps=max(4, min(_log_int(rng, 12, 60), int(most / size / members))),
                    precision="fast", planet="hot", dt=600.0 if M == 42 else 300.0)
    steps = max(4, min(_log_int(rng, 20, 400), int(most / size / members)))
    if kind == "gradient":
        return dict(kind=kind, M=M, members=members, steps=min(steps, 60), precision=precision, planet="strong",
                    dt=1260.0 / M)
    if M == 42 and rng.random() < 0.3:
        return dict(kind=kind, M=M, members=members, steps=min(steps, 72), precision=precision, planet="wasp",
                    dt=1200.0, scheme="semi", history=False)
    if members == 1 and M == 42:
        return dict(kind=kind, M=M, members=0, steps=steps, precision=precision, planet="hot", dt=120.0,
                    scheme="euler", history=steps < 300 and rng.random() < 0.5)
    return dict(kind=kind, M=M, members=members, steps=min(steps, 48 if M == 106 else 400), precision=precision,
                planet="strong", dt=1260.0 / M, scheme="euler", history=False)


# --------------------------------------------------------------------------- inputs
def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


@functools.lru_cache(maxsize=None)
def _basis(M):
    """(mu, w, P, H) of truncation M on the CPU: Gauss nodes and weights (J,), normalised associated
    Legendre functions and (1 - mu^2) dP/dmu, both (M+1, J, N+1).  At M = 106 the model's factorial
    normalisation underflows (subnormal quotients); its values carry that, and so do these."""
    J, N = GRID[M][0], M
    mu, w = np.polynomial.legendre.leggauss(J)
    s = np.sqrt(1.0 - mu * mu)
    P, H = np.zeros((M + 1, J, N + 1)), np.zeros((M + 1, J, N + 1))
    pmm = np.full(J, math.sqrt(0.5))
    for m in range(M + 1):
        if m:
            pmm = pmm * s * math.sqrt((2 * m + 1) / (2 * m))
        P[m, :, m] = pmm
        for n in range(m + 1, N + 1):
            A = math.sqrt((4 * n * n - 1) / (n * n - m * m))
            Bc = math.sqrt(((n - 1) ** 2 - m * m) / (4 * (n - 1) ** 2 - 1)) if n > m + 1 else 0.0
            P[m, :, n] = A * (mu * P[m, :, n - 1] - (Bc * P[m, :, n - 2] if n > m + 1 else 0.0))
        for n in range(m, N + 1):
            H[m, :, n] = -n * mu * P[m, :, n]
            if n > m:
                H[m, :, n] += math.sqrt((2 * n + 1) * (n * n - m * m) / (2 * n - 1)) * P[m, :, n - 1]
        for n in range(m, N + 1):
            num, den = (2 * n + 1) * math.factorial(n - m), 2 * math.factorial(n + m)
            k = max(0, den.bit_length() - num.bit_length()) // 2
            true = math.sqrt((num << (2 * k)) / den)  # times 2^-k
            got = math.sqrt(num / den)
            f = (got * 2.0 ** min(k, 1000)) / (true * 2.0 ** min(0, 1000 - k)) if got else 0.0
            if abs(f - 1.0) > 1e-15:
                P[m, :, n] *= f
                H[m, :, n] *= f
    return tuple(torch.from_numpy(x) for x in (mu, w, P, H))


@functools.lru_cache(maxsize=4)
def _noise_basis(M):
    return _basis(M)[2][:11, :, :11].to("cuda", torch.complex128)


def _noise(M, B, amplitude, gen):
    """Phi noise (B, J, I): Gaussian coefficients of degree <= 10, synthesised to the grid."""
    I = GRID[M][1]
    P = _noise_basis(M)
    c = torch.randn((B, 11, 11, 2), dtype=torch.float64, device="cuda", generator=gen)
    c[:, 0, :, 1] = 0.0
    z = torch.einsum("mjn,bmn->bjm", P, torch.view_as_complex(c * amplitude))
    spec = torch.zeros((B, z.shape[1], I // 2 + 1), dtype=torch.complex128, device="cuda")
    spec[..., :11] = z * I
    return torch.fft.irfft(spec, n=I, dim=-1)


def _inputs(case, seed):
    """Parameters and initial fields of a dynamics case: floats for a single member, else (B,)
    tensors and (B, J, I) fields on the GPU."""
    M, J, I = case["M"], *GRID[case["M"]]
    planet = PLANETS[case["planet"]]
    if not case["members"]:  # scalars and the model's own start from rest
        r = random.Random(int(seed))
        p = dict(taurad=10.0 ** r.uniform(4.3, 5.0), taudrag=10.0 ** r.uniform(4.2, 5.0), DPhieq=r.uniform(0.5e6, 1.2e6))
        return dict(params=p, fields=None)
    B, gen = case["members"], _gen(seed)
    u = torch.rand((4, B), dtype=torch.float64, device="cuda", generator=gen)
    if case["planet"] == "strong":  # from 3 hours to 12 days, DPhieq up to Phibar
        p = dict(taurad=10.0 ** (4.0 + 2.0 * u[0]), taudrag=10.0 ** (4.0 + 2.0 * u[1]), DPhieq=1e5 + 3.9e6 * u[2])
    else:
        p = dict(taurad=10.0 ** (4.3 + 0.7 * u[0]), taudrag=10.0 ** (4.2 + 0.8 * u[1]), DPhieq=0.5e6 + 0.7e6 * u[2])
    mu = _basis(M)[0].to("cuda")
    eta = (2.0 * planet["omega"] * mu)[None, :, None].expand(B, J, I).contiguous()
    zero = torch.zeros((B, J, I), dtype=torch.float64, device="cuda")
    Phi = _noise(M, B, 1e-3 * planet["Phibar"], gen)
    target = _noise(M, B, 1e-2 * planet["Phibar"], gen) if case["kind"] in ("gradient", "retrieval") else None
    p = {k: v.contiguous() for k, v in p.items()}
    return dict(params=p, fields=[eta, zero, Phi, zero.clone(), zero.clone()], target=target,
                Phibar=torch.full((B,), planet["Phibar"], dtype=torch.float64, device="cuda"))


def _emission_inputs(case, seed):
    J, I = GRID[case["M"]]
    B, gen = case["members"], _gen(seed)
    # a hot day side over the noise, some 900 to 2400 K
    mu = _basis(case["M"])[0].to("cuda")
    lam = torch.linspace(-math.pi, math.pi, I + 1, dtype=torch.float64, device="cuda")[:-1]
    day = torch.clamp(torch.cos(lam), min=0.0)[None, :] * torch.sqrt(1.0 - mu * mu)[:, None]
    amp = 1e6 + 3e6 * torch.rand((B, 1, 1), dtype=torch.float64, device="cuda", generator=gen)
    return 0.02 * amp * day * 50.0 + _noise(case["M"], B, 4.0e4, gen), gen


# The design matrices of an emission case stand for the third-party spherical-harmonic model's:
# latitude-longitude polynomials, evaluated once per retrieval, and a light curve that sees them.
@functools.lru_cache(maxsize=8)
def _projector(M, ncoef, times):
    J, I = GRID[M]
    mu, w = _basis(M)[0].to("cuda"), _basis(M)[1].to("cuda")
    deg = int(round(math.sqrt(ncoef))) - 1
    P = _basis(M)[2].to("cuda")
    lam = torch.linspace(-math.pi, math.pi, I + 1, dtype=torch.float64, device="cuda")[:-1]
    cols = []
    for n in range(deg + 1):
        for m in range(-n, n + 1):
            lon = torch.cos(m * lam) if m >= 0 else torch.sin(-m * lam)
            cols.append((P[abs(m), :, n][:, None] * lon[None, :]).reshape(-1))
    proj = emission.build_projector(torch.stack(cols, 1), w)
    k = torch.arange(ncoef, dtype=torch.float64, device="cuda")
    t = torch.linspace(0.0, 2.0 * math.pi, times, dtype=torch.float64, device="cuda")
    return proj, w, torch.cos(t[:, None] * (1.0 + k[None, :] % 7)) / (1.0 + k[None, :])


def _config(case):
    if case["bands"] == 0:
        return emission.EmissionConfig()
    if case["bands"] == 1:
        return emission.EmissionConfig(emission_model="planck")
    return emission.EmissionConfig(emission_model="planck", planck_band_wavelengths_m=(3.6e-6, 4.5e-6),
                                   planck_band_weights=(0.4, 0.6))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "phase":
        return dict(case=case, phi=_emission_inputs(case, seed)[0],
                    phases=torch.linspace(-math.pi, math.pi, case["phases"], dtype=torch.float64, device="cuda"))
    if kind == "emission":
        phi, gen = _emission_inputs(case, seed)
        proj, w, lc = _projector(case["M"], case["coefficients"], case["times"])
        amp = 1e-3 * (1.0 + torch.rand(case["members"], dtype=torch.float64, device="cuda", generator=gen))
        return dict(case=case, phi=phi, projector=proj, w=w, curve=lc, amplitude=amp, config=_config(case))
    s = _inputs(case, seed)
    s["case"] = case
    planet = PLANETS[case["planet"]]
    if kind == "gradient":
        s["params"] = {k: v.requires_grad_() for k, v in s["params"].items()}
        s["Phibar"].requires_grad_()
        s["fields"] = [f.requires_grad_() for f in s["fields"]]
    if kind == "retrieval":  # the base state is built once, the samples replace taurad and taudrag
        s["static"] = build_static(M=case["M"], dt=case["dt"], a=planet["a"], omega=planet["omega"], g=9.8,
                                   Phibar=planet["Phibar"], taurad=s["params"]["taurad"], taudrag=s["params"]["taudrag"],
                                   DPhieq=s["params"]["DPhieq"], K6=K6, K6Phi=None, test=None)
        s["flags"] = RunFlags(diagnostics=False, alpha=ALPHA)
        s["fields"] = [f.float() for f in s["fields"]]
        s["state0"] = _init_state_from_fields(static=s["static"], flags=s["flags"], test=None,
                                              **{k + "0": f for k, f in zip(FIELDS, s["fields"])})
        s["t_seq"] = torch.arange(2, 2 + case["steps"])
        s["target"] = s["target"].float()
        # a sample's parameters: near the base
        s["sample"] = {k: (0.9 * s["params"][k]).requires_grad_() for k in ("taurad", "taudrag")}
    return s


# --------------------------------------------------------------------------- the measured calls
def _last(state):
    return {k: getattr(state, k) for k in ("eta_curr", "delta_curr", "Phi_curr", "U_curr", "V_curr", "eta_prev",
                                           "delta_prev", "Phi_prev")}


def _model_args(s):
    case, planet = s["case"], PLANETS[s["case"]["planet"]]
    kw = dict(M=case["M"], dt=case["dt"], tmax=2 + case["steps"], omega=planet["omega"], a=planet["a"],
              Phibar=planet["Phibar"], K6=K6, alpha=ALPHA, precision=case["precision"], **s["params"])
    if s["fields"] is not None:
        kw.update({k + "0_init": f for k, f in zip(FIELDS, s["fields"])})
    return kw


def run(state):
    s, case = state, state["case"]
    if case["kind"] == "phase":
        return emission.simple_phase_curve(s["phi"], s["phases"])
    if case["kind"] == "emission":
        y = emission.emission_coefficients(s["phi"], PLANETS["strong"]["Phibar"], s["projector"], s["w"], s["config"])
        return dict(y=y, curve=emission.phase_curve(y, s["curve"], amplitude=s["amplitude"]))
    if case["kind"] == "run":
        kw = _model_args(s)
        if case["scheme"] == "semi":
            kw["semi_implicit"] = True
        if not case["history"]:
            return _last(run_model_scan_final(**kw)["last_state"])
        res = run_model_scan(**kw)
        return dict(_last(res["last_state"]), **res["outs"])
    if case["kind"] == "gradient":
        kw = _model_args(s)
        kw["Phibar"] = s["Phibar"]
        Phi = run_model_scan_final(**kw)["last_state"].Phi_curr
        leaves = [*s["fields"], *s["params"].values(), s["Phibar"]]
        grads = torch.autograd.grad(((Phi - s["target"].to(Phi.dtype)) ** 2).mean(), leaves)
        return dict(zip(["Phi", *FIELDS, *s["params"], "Phibar"], [Phi.detach(), *grads]))
    static = dataclasses.replace(s["static"], **s["sample"])
    U, V = s["fields"][3:]
    Phi = simulate_scan_last(static=static, flags=s["flags"], state0=s["state0"], t_seq=s["t_seq"], test=None,
                             Uic=U, Vic=V).Phi_curr
    grads = torch.autograd.grad(((Phi - s["target"]) ** 2).mean(), list(s["sample"].values()))
    return dict(zip(["Phi", *s["sample"]], [Phi.detach(), *grads]))


# --------------------------------------------------------------------------- work
def _step_flops(M):
    J, I = GRID[M]
    legendre = 4 * 16 * (J // 2) * (M + 1) * (M + 2) // 2  # 9 forward, 7 inverse, complex, equatorial symmetry
    return legendre + 12 * J * 2.5 * I * math.log2(I) + 60 * J * I


def work(case):
    J, I = GRID[case["M"]]
    B = max(1, case["members"])
    if case["kind"] == "phase":
        n = case["phases"]
        return dict(bytes=8 * B * (J * I + n), flops=B * (2 * J * I + 2 * I * n))
    if case["kind"] == "emission":
        n, t = case["coefficients"], case["times"]
        return dict(bytes=8 * (B * (J * I + n + t) + n * (J * I + t)), flops=B * (2 * n * (J * I + t) + 40 * J * I))
    size = 8 if case["precision"] == "fp64" else 4
    steps = case["steps"]
    if case["kind"] == "run":
        moved = (8 * 5 if case["members"] else 0) + 8 * size + (5 * size * steps if case["history"] else 0)
        return dict(bytes=B * J * I * moved, flops=B * steps * _step_flops(case["M"]))
    moved = 8 * 11 + size if case["kind"] == "gradient" else 7 * size
    return dict(bytes=B * J * I * moved, flops=2 * B * steps * _step_flops(case["M"]))


# --------------------------------------------------------------------------- exact values
class _Model:
    """The model in plain torch, FP64, CPU.  Fourier fields are (M+1, B, J), grid fields (B, J, I);
    a parameter is a (B,) tensor or a float."""

    def __init__(self, M, dt, a, omega, Phibar, taurad, taudrag, DPhieq):
        self.M, (self.J, self.I) = M, GRID[M]
        self.mu, w, self.P, self.H = _basis(M)
        self.PT, self.HT = self.P.transpose(1, 2).contiguous(), self.H.transpose(1, 2).contiguous()
        self.Pw, self.Hw = w[None, :, None] * self.P, w[None, :, None] * self.H
        n = torch.arange(M + 1, dtype=torch.float64)
        self.dt, self.a, self.om = dt, a, omega / math.sqrt(0.375)
        at = lambda x: torch.as_tensor(x, dtype=torch.float64).reshape(-1)  # noqa: E731
        self.Pb, self.tr, self.td, self.DP = at(Phibar), at(taurad), at(taudrag), at(DPhieq)
        self.nn1, self.tc = n * (n + 1), torch.where(n > 0, a / torch.clamp(n * (n + 1), min=1.0), 0.0)
        nc = (n ** 3 / a ** 3) * ((n + 1) ** 3 / a ** 3)
        self.sig, self.sigP = 1 / (1 + 2 * dt * K6 * (nc - 8 / a ** 6)), 1 / (1 + 2 * dt * K6 * nc)
        self.sigX = torch.exp(-2 * dt * K6 * torch.clamp(nc - 8 / a ** 6, min=0.0))
        self.sigPX = torch.exp(-2 * dt * K6 * nc)
        self.tsc = 2 * dt / (a * (1 - self.mu ** 2))
        self.im = 1j * torch.arange(M + 1, dtype=torch.float64)[:, None, None]
        lam = torch.linspace(-math.pi, math.pi, self.I + 1, dtype=torch.float64)[:-1]
        self.day = torch.where(torch.cos(lam) > 0, torch.cos(lam), 0.0)
        self.day = torch.where((lam > -math.pi / 2) & (lam < math.pi / 2), self.day, 0.0)
        self.day = self.day[None, :] * torch.sqrt(1 - self.mu[:, None] ** 2)

    def fwd(self, x):
        return (torch.fft.rfft(x, dim=-1)[..., : self.M + 1] / self.I).permute(2, 0, 1)

    def inv(self, X):
        spec = torch.nn.functional.pad(torch.view_as_real(X.permute(1, 2, 0)), (0, 0, 0, self.I // 2 - self.M))
        return torch.fft.irfft(torch.view_as_complex(spec.contiguous()) * self.I, n=self.I, dim=-1)

    @staticmethod
    def leg(X, W):
        return torch.complex(X.real @ W, X.imag @ W)

    def grid_terms(self, eta, Phi, U, V):
        """Fourier A, B, C, D, E, PhiF, F, G."""
        Pb, tr, td, DP = (x[:, None, None] for x in (self.Pb, self.tr, self.td, self.DP))
        Q = (Pb + DP * self.day - (Phi + Pb)) / tr
        r = torch.where(Q < 0, 0.0, Q) / (Phi + Pb)
        E = (U * U + V * V) / (2 * (1 - self.mu ** 2))[:, None]
        return [self.fwd(x) for x in (U * eta, V * eta, U * Phi, V * Phi, E, Q, -U * r - U / td, -V * r - V / td)]

    def euler(self, X, T):
        eta, de, ph = X
        A, B, C, D, E, PF, F, G = T
        dt, a2, Pb = self.dt, self.a ** 2, self.Pb[None, :, None]
        t1, t2 = self.tsc / 4, 2 * dt / a2 / 4
        Bf, Af, L, Hh, nn = B + F, A - G, self.Pw, self.Hw, self.nn1
        p = self.leg(ph - t1 * self.im * C - dt * Pb * de - 0.5 * Pb * t1 * self.im * Bf + dt * PF, L)
        p = p + self.leg(t1 * D - 0.5 * Pb * t1 * Af, Hh) - nn * self.leg(0.5 * Pb * (t2 * E + ph / a2), L)
        d = self.leg(de + t1 * self.im * Bf, L) + self.leg(t1 * Af, Hh)
        d = d + nn * self.leg(t2 * (ph + E) + t1 * self.im * C / (2 * a2) - Pb * de / a2 + 0.5 * dt * PF / a2, L)
        d = d + nn * self.leg(t1 * D / (2 * a2), Hh)
        e = self.leg(eta - self.tsc * self.im * Af, L) + self.leg(self.tsc * Bf, Hh)
        return self.sig * e, self.sig * d, self.sigP * p

    def semi(self, X0, ph1, T, Fx, Gx):
        """The semi-implicit solve (si_alpha = 1/2) on the filtered n-1 level X0."""
        eta0, del0, phi0 = X0
        A, B, C, D, E, PF = T[:6]
        xi = ex = self.dt
        Pb, itd, itr = self.Pb[None, :, None], 1 / self.td[None, :, None], 1 / self.tr[None, :, None]
        Aeff, Beff, tc, L, Hh = A - Gx, B + Fx, self.tsc, self.Pw, self.Hw
        lam = self.nn1 / self.a ** 2
        f = torch.zeros((self.M + 1, 1, self.M + 1), dtype=torch.float64)
        f[0, 0, 1] = self.om
        es = self.leg((1 - ex * itd) * eta0 - tc * self.im * Aeff, L) + self.leg(tc * Beff, Hh) + ex * itd * f
        ds = self.leg((1 - ex * itd) * del0 + tc * self.im * Beff, L) + self.leg(tc * Aeff, Hh)
        ds = ds + lam * self.leg(2 * self.dt * E + ex * phi0, L)
        ps = self.leg((1 - ex * itr) * phi0 - tc * self.im * C - ex * Pb * del0 + 2 * self.dt * (PF + ph1 * itr), L)
        ps = ps + self.leg(tc * D, Hh)
        kd, kr, bq, cq = xi * itd, xi * itr, xi * lam, xi * Pb
        dn = (ds + bq * ps / (1 + kr)) / ((1 + kd) + bq * cq / (1 + kr))
        return self.sigX * (es + kd * f) / (1 + kd), self.sigX * dn, self.sigPX * (ps - cq * dn) / (1 + kr)

    def winds(self, e, d):
        f = torch.zeros_like(e.real[:, :1])
        f[0, 0, 1] = self.om
        es, ds = (e - f) * self.tc, d * self.tc
        return (self.leg(es, self.HT) - self.im * self.leg(ds, self.PT),
                -self.im * self.leg(es, self.PT) - self.leg(ds, self.HT))

    def rms(self, U, V):
        phi = torch.asin(self.mu)
        area = (torch.sin(phi + math.pi / 2) ** 2) * (phi[2] - phi[1]) * (2 * math.pi / self.I) / (4 * math.pi)
        return torch.sqrt(((area / torch.cos(phi) ** 2)[:, None] * (U * U + V * V)).sum(dim=(-2, -1)))

    def integrate(self, fields, steps, scheme="euler", state0=None, keep=None):
        """The final curr (eta, delta, Phi, U, V) and prev (eta, delta, Phi) grid fields; the per-step
        rows are appended to `keep`.  state0: Fourier terms to start from (a prepared state's)."""
        curr = list(fields)
        prev = curr[:3]
        X = [self.fwd(x) for x in curr]
        T = self.grid_terms(curr[0], curr[2], curr[3], curr[4]) if state0 is None else state0
        X0, itd = X[:3], 1 / self.td[None, :, None]
        Fx, Gx = T[6] + X[3] * itd, T[7] + X[4] * itd
        for t in range(2, 2 + steps):
            if scheme == "semi":
                S = self.semi(X0, X[2], T, Fx, Gx)
                Fx, Gx = T[6] + X[3] * itd, T[7] + X[4] * itd
            else:
                S = self.euler(X[:3], T)
            N = [self.leg(c, self.PT) for c in S] + list(self.winds(S[0], S[1]))
            new = [self.inv(x) for x in N]
            al = ALPHA if t > 2 else 0.0
            mid = [c + al * (p - 2 * c + x) for p, c, x in zip(prev, curr, new)]
            X0 = [c + al * (p - 2 * c + x) for p, c, x in zip(X0, X, N)]
            if keep is not None:
                keep.append((*new, self.rms(curr[3], curr[4]), torch.sqrt(curr[3] ** 2 + curr[4] ** 2).amin((-2, -1)),
                             mid[2].amin((-2, -1)), mid[2].amax((-2, -1))))
            prev, curr, X = mid, new, N
            T = self.grid_terms(curr[0], curr[2], curr[3], curr[4])
        return curr, prev


def _exact_model(case, s, params):
    planet = PLANETS[case["planet"]]
    return _Model(case["M"], case["dt"], planet["a"], planet["omega"], **{"Phibar": planet["Phibar"], **params})


def exact(case, seed):
    if case["kind"] == "phase":
        J, I = GRID[case["M"]]
        phi = _emission_inputs(case, seed)[0].cpu()
        ph = torch.linspace(-math.pi, math.pi, case["phases"], dtype=torch.float64)
        lam = torch.linspace(-math.pi, math.pi, I + 1, dtype=torch.float64)[:-1]
        vis = torch.clamp(torch.cos(lam[None, :] - ph[:, None]), min=0.0)
        flux = torch.einsum("bji,j,ki->bk", phi, torch.sqrt(1 - _basis(case["M"])[0] ** 2), vis)
        return flux / flux.abs().mean(dim=1, keepdim=True)
    if case["kind"] == "emission":
        s = {k: v.cpu() if torch.is_tensor(v) else v for k, v in prepare(case, seed).items()}
        J, I = GRID[case["M"]]
        T = torch.clamp((PLANETS["strong"]["Phibar"] + s["phi"]) / s["config"].R_d, min=1.0)
        bands = {0: [], 1: [(4.5e-6, 1.0)], 2: [(3.6e-6, 0.4), (4.5e-6, 0.6)]}[case["bands"]]
        hck = 6.62607015e-34 * 299792458.0 / 1.380649e-23
        Imap = sum(w / (torch.expm1(torch.clamp(hck / (l * T), 0.0, 80.0)) + 1e-30) for l, w in bands) if bands else T ** 4
        w = s["w"][:, None].expand(J, I)
        rel = Imap / ((w * Imap).sum(dim=(1, 2), keepdim=True) / w.sum())
        y = (torch.sqrt(w) * rel).reshape(-1, J * I) @ s["projector"].T
        y = y / y[:, :1]
        return dict(y=y, curve=s["amplitude"][:, None] * (y @ s["curve"].T))
    B = max(1, case["members"])
    cost = B * case["steps"] * (case["M"] / 42.0) ** 3 * (1 if case["kind"] == "run" else 8)
    if cost > 24000:
        return None
    s = _inputs(case, seed)
    cpu = lambda v: v.cpu() if torch.is_tensor(v) else v  # noqa: E731
    params = {k: cpu(v) for k, v in s["params"].items()}
    if case["kind"] == "run":
        if s["fields"] is None:  # solid-body vorticity, at rest: the model's own initial fields
            planet = PLANETS[case["planet"]]
            J, I = GRID[case["M"]]
            amp = 2.0 * (2.0 * math.pi / (3600.0 * 24.0 * 12.0) + planet["omega"])
            z = torch.zeros((1, J, I), dtype=torch.float64)
            fields = [(amp * _basis(case["M"])[0])[None, :, None].expand(1, J, I), z, z, z, z]
        else:
            fields = [f.cpu() for f in s["fields"]]
        keep = [] if case["history"] else None
        with torch.no_grad():
            curr, prev = _exact_model(case, s, params).integrate(fields, case["steps"], case["scheme"], keep=keep)
        pick = (lambda v: v) if case["members"] else (lambda v: v[0])
        out = dict(zip([k + "_curr" for k in FIELDS] + [k + "_prev" for k in FIELDS[:3]], map(pick, curr + prev)))
        if keep is not None:
            rows = zip(*keep)
            for name, r in zip((*FIELDS, "rms", "spin_min", "phi_min", "phi_max"), rows):
                r = torch.stack(r, 1)
                out[name] = pick(r)
            out["dead"] = None
        return out
    if case["kind"] == "gradient":
        leaves = [f.cpu().requires_grad_() for f in s["fields"]]
        params = {k: v.requires_grad_() for k, v in params.items()}
        Pb = s["Phibar"].cpu().requires_grad_()
        curr, _ = _exact_model(case, s, dict(params, Phibar=Pb)).integrate(leaves, case["steps"])
        grads = torch.autograd.grad(((curr[2] - s["target"].cpu()) ** 2).mean(), [*leaves, *params.values(), Pb])
        return dict(zip(["Phi", *FIELDS, *params, "Phibar"], [curr[2].detach(), *grads]))
    fields = [f.float().cpu().double() for f in s["fields"]]
    with torch.no_grad():  # the prepared state's forcing is the base parameters'
        base = _exact_model(case, s, params).grid_terms(fields[0], fields[2], fields[3], fields[4])
    sample = {k: (0.9 * params[k]).requires_grad_() for k in ("taurad", "taudrag")}
    curr, _ = _exact_model(case, s, dict(params, **sample)).integrate(fields, case["steps"], state0=base)
    target = s["target"].float().cpu().double()
    grads = torch.autograd.grad(((curr[2] - target) ** 2).mean(), list(sample.values()))
    return dict(zip(["Phi", *sample], [curr[2].detach(), *grads]))
