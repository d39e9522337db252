"""Workloads of the solver through its public Python calls, with their inputs,
the work each cannot do without, and what plain 64-bit torch gives for them.

The listed cases are what a run of the framework consists of: time steps of
direct simulations (2D and 3D, both precisions, the reference's Wray stepper
and RK4), a bare right-hand side, the DNS -> LES filter, LES steps with a
classical and with a learned closure, the training gradient through a rollout,
the per-step statistics, and the plain transforms.  ``draw`` gives other sizes,
precisions, dimensions and options of the same calls.

Fields are seeded Gaussian fields with a developed spectrum (k^4 rise to the
energy-containing scale, k^(-5/3) range, exponential viscous cut-off),
divergence-free, 2/3-truncated and of unit kinetic energy, on [0, 2 pi)^D.
"""

import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "symmetrycode.jl_b200"))

import symcode as sc  # noqa: E402

# sizes 2^a 3^b 5^c the transforms take, over the range people run
SIZES_3D = (32, 36, 40, 48, 60, 64, 72, 80, 90, 96, 120, 128, 160, 180, 192, 240, 256, 270, 320, 360, 384, 512)
SIZES_2D = (64, 72, 90, 96, 120, 128, 160, 180, 192, 240, 256, 320, 360, 384, 512, 540, 640, 720, 768, 810, 1024)
SIZES_LES = (32, 36, 40, 48, 60, 64, 72, 80, 90, 96, 120, 128)
CNN_LAYERS = ((4, 32), (32, 32), (32, 32), (32, 6))
DEV = "cuda:0"


def listed():
    return [
        # 2D decaying turbulence in double precision, one RK4 step: the smallest
        # call of the solver, where launches and host work count
        {"name": "dns2d_256_f64", "kind": "rk4", "D": 2, "n": 256, "dtype": "f64", "forced": False},
        # a small 3D grid of a size that is no power of two, the reference's own
        # low-storage stepper
        {"name": "dns_96_f32", "kind": "wray3", "D": 3, "n": 96, "dtype": "f32", "forced": False},
        # forced 3D turbulence at the ordinary size, single and double precision
        {"name": "dns_256_f32", "kind": "rk4", "D": 3, "n": 256, "dtype": "f32", "forced": True},
        {"name": "dns_256_f64", "kind": "rk4", "D": 3, "n": 256, "dtype": "f64", "forced": True},
        # the production DNS: the largest grid, one forced step
        {"name": "dns_810_f32", "kind": "rk4", "D": 3, "n": 810, "dtype": "f32", "forced": True},
        # a bare right-hand side on a large double-precision grid (a user's own stepper)
        {"name": "rhs_540_f64", "kind": "rhs", "D": 3, "n": 540, "dtype": "f64"},
        # training data: a DNS snapshot filtered to LES resolution at three widths
        {"name": "sfs_810_128_f32", "kind": "sfs", "D": 3, "n": 810, "n_les": 128, "dtype": "f32", "ratios": "2,4,8"},
        # LES with the classical dynamic model
        {"name": "les_128_dynsmag", "kind": "les", "D": 3, "n": 128, "dtype": "f32", "closure": "dynsmag",
         "stepper": "rk4", "ratio": 4},
        # LES with the learned closure (BF16 tensor cores)
        {"name": "les_128_cnn", "kind": "les", "D": 3, "n": 128, "dtype": "f32", "closure": "cnn", "stepper": "rk4",
         "ratio": 4},
        # one a-posteriori training gradient (forward, loss, backward) in split precision
        {"name": "adjoint_64_split", "kind": "adjoint", "n": 64, "nsteps": 5, "ckpt": 5},
        # what a run measures between its steps: CFL step, energy, dissipation, spectrum
        {"name": "stats_256_f32", "kind": "stats", "D": 3, "n": 256, "dtype": "f32"},
        # one scalar field to spectral space and back
        {"name": "transform_360_f32", "kind": "transform", "D": 3, "n": 360, "dtype": "f32"},
    ]


def _pick(rng, sizes, lo, hi):
    """One of `sizes` in [lo, hi], spread over the logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((s for s in sizes if lo <= s <= hi), key=lambda s: abs(math.log(s / x)))


def draw(rng):
    kind = rng.choice(("rk4", "rk4", "wray3", "rhs", "sfs", "les", "les", "adjoint", "stats", "transform"))
    dtype = rng.choice(("f32", "f64"))
    if kind in ("rk4", "wray3", "rhs", "stats", "transform"):
        D = rng.choice((2, 3, 3))
        n = _pick(rng, SIZES_2D, 64, 1024) if D == 2 else _pick(rng, SIZES_3D, 32, 512 if dtype == "f32" else 384)
        case = {"kind": kind, "D": D, "n": n, "dtype": dtype}
        if kind in ("rk4", "wray3"):
            case["forced"] = kind == "rk4" and rng.random() < 0.5
        return case
    if kind == "sfs":
        n_les = _pick(rng, SIZES_LES, 32, 128)
        n = _pick(rng, SIZES_3D, 2 * n_les, 512 if dtype == "f32" else 384)
        return {"kind": "sfs", "D": 3, "n": n, "n_les": n_les, "dtype": dtype,
                "ratios": rng.choice(("2", "4", "2,4", "2,3,4", "2,4,8"))}
    if kind == "les":
        closure = rng.choice(("clark", "smagorinsky", "bardina", "dynsmag", "dynsmag", "cnn", "cnn_split"))
        cnn = closure.startswith("cnn")
        return {"kind": "les", "D": 3, "n": rng.choice((64, 128)) if cnn else _pick(rng, SIZES_LES, 32, 128),
                "dtype": "f32" if cnn else dtype, "closure": closure, "stepper": rng.choice(("rk4", "wray3")),
                "ratio": rng.choice((2, 4, 8))}
    return {"kind": "adjoint", "n": 64, "nsteps": rng.randint(1, 5), "ckpt": rng.randint(1, 5)}


# --------------------------------------------------------------------------
# parameters and inputs
# --------------------------------------------------------------------------
def _params(case):
    """dt, viscosity, filter width and forcing of a case (about k_max eta = 1, CFL 0.5)."""
    n = case["n"]
    nu = 2e-3 * (256 / n) ** (4 / 3) if case.get("D", 3) == 3 else 5e-4 * (256 / n)
    h = 2 * math.pi / n
    return {"dt": 0.1 * h, "nu": nu, "delta": case.get("ratio", 4) * h, "eps": 0.1 if case.get("forced") else None}


def _real(case):
    return torch.float64 if case.get("dtype", "f32") == "f64" else torch.float32


def _wave(n, D, dtype=torch.float64, half=True):
    """Integer wavenumbers (kx, ky[, kz]) of the half spectrum, shaped to broadcast over [z][y][x]."""
    full = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=dtype)
    kx = torch.arange(n // 2 + 1, device=DEV, dtype=dtype)
    return (kx, full[:, None]) if D == 2 else (kx, full[:, None], full[:, None, None])


def _keep(n, D):
    """The modes the 2/3 rule keeps, without the mean."""
    kc = n // 3
    m = None
    for k in _wave(n, D):
        b = k.abs() <= kc
        m = b if m is None else m & b
    m = m.clone()
    m[(0,) * D] = False
    return m


def _weight(n):
    """How often a stored mode stands for itself and its conjugate."""
    w = torch.full((n // 2 + 1,), 2.0, device=DEV, dtype=torch.float64)
    w[0] = w[-1] = 1.0
    return w


def _field(D, n, dtype, seed):
    """Seeded solenoidal turbulent velocity, D spectral fields in the full layout."""
    gen = torch.Generator(device=DEV).manual_seed(seed * 1009 + 17)
    k = _wave(n, D, dtype)
    k2 = sum(x * x for x in k)
    kp, ke = 4.0, n / 3.0
    kk = torch.sqrt(k2)
    amp = torch.sqrt(kk ** 4 / (1 + k2 / kp ** 2) ** (17 / 6) * torch.exp(-2.0 * kk / ke) / kk.clamp(min=1) ** (D - 1))
    amp *= _keep(n, D)
    u = []
    for _ in range(D):
        f = torch.fft.rfftn(torch.randn((n,) * D, generator=gen, device=DEV, dtype=dtype), norm="forward")
        u.append(f * amp)
        del f
    k2[(0,) * D] = 1
    p = sum(a * b for a, b in zip(k, u)) / k2
    for a, b in zip(k, u):
        b -= a * p
    w = _weight(n)
    e = 0.5 * sum(((c.real.double() ** 2 + c.imag.double() ** 2) * w).sum() for c in u)
    s = (1 / torch.sqrt(e)).to(dtype)
    return [(c * s).contiguous() for c in u]


def _weights(seed):
    """Kaiming weights of the closure network, its last layer small (stresses of the size of a trained one)."""
    gen = torch.Generator().manual_seed(seed * 7919 + 5)
    ws, bs = [], []
    for i, (ci, co) in enumerate(CNN_LAYERS):
        std = (2.0 / (27 * ci)) ** 0.5 * (0.05 if i == 3 else 1.0)
        ws.append((torch.randn((co, ci, 3, 3, 3), generator=gen) * std).numpy())
        bs.append((torch.randn((co,), generator=gen) * 0.01).numpy())
    return ws, bs


def _closure(case, g, seed):
    p = _params(case)
    kind = case["closure"]
    if kind == "clark":
        return sc.create_clark(p["delta"], g)
    if kind == "smagorinsky":
        return sc.create_smagorinsky(0.17, p["delta"], g)
    if kind == "bardina":
        return sc.create_bardina(2.0, p["delta"], g)
    if kind == "dynsmag":
        return sc.create_dynamic_smagorinsky(p["delta"], g)
    ws, bs = _weights(seed)
    return sc.create_cnn_closure(p["delta"], p["nu"], g, ws, bs, split=kind == "cnn_split")


def _target(case, u0):
    """The trajectory a training rollout is fitted to: `nsteps` states of a plain
    simulation at a slightly higher viscosity, the retained modes of each packed
    into (2k+1, 2k+1, k+1) arrays (k = n//3, negative wavenumbers last)."""
    p = _params(case)
    n = case["n"]
    kc = n // 3
    pick = torch.tensor([*range(kc + 1), *range(n - kc, n)], device=DEV)
    u = [c.to(torch.complex128) for c in u0]
    out = []
    for _ in range(case["nsteps"]):
        u = _rk4(u, n, 3, p["dt"], 1.2 * p["nu"], None)
        out += [c[pick][:, pick][:, :, :kc + 1].to(torch.complex64).reshape(-1) for c in u]
    return torch.cat(out)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    D = case.get("D", 3)
    g = sc.Grid(D, n, dtype=_real(case), device=DEV)
    s = {"case": case, "g": g, **_params(case)}
    if kind == "transform":
        gen = torch.Generator(device=DEV).manual_seed(seed * 1009 + 29)
        s["phys"] = torch.randn(g.phys_shape, generator=gen, device=DEV, dtype=g.dtype)
        s["spec"], s["back"] = sc.scalarfield(g), sc.spacescalarfield(g)
        return s
    s["u"] = _field(D, n, g.dtype, seed)
    if kind == "rhs":
        s["du"] = sc.vectorfield(g)
    elif kind == "sfs":
        s["gl"] = gl = sc.Grid(D, case["n_les"], dtype=g.dtype, device=DEV)
        s["deltas"] = [float(r) * gl.spacing for r in case["ratios"].split(",")]
        s["ubar"] = [sc.vectorfield(gl) for _ in s["deltas"]]
        s["tau"] = [sc.tensorfield(gl) for _ in s["deltas"]]
    elif kind == "les":
        s["closure"] = _closure(case, g, seed)
    elif kind == "adjoint":
        ws, bs = _weights(seed)
        s["closure"] = sc.create_cnn_closure(s["delta"], s["nu"], g, ws, bs, split=True)
        s["traj"] = torch.view_as_real(_target(case, s["u"])).contiguous().view(torch.uint8).reshape(-1)
    return s


def run(s):
    case, g = s["case"], s["g"]
    kind = case["kind"]
    if kind == "rk4":
        return sc.rk4_(s["u"], s["dt"], g, s["nu"], nsteps=1, eps=s["eps"])
    if kind == "wray3":
        return sc.wray3_(s["u"], s["dt"], g, s["nu"])
    if kind == "rhs":
        return sc.convectiondiffusion_(s["du"], s["u"], g, s["nu"])
    if kind == "sfs":
        ubar, tau = sc.sfs_(s["ubar"], s["tau"], s["u"], g, s["gl"], s["deltas"])
        return {"ubar": ubar, "tau": tau}
    if kind == "les":
        step = sc.les_rk4_ if case["stepper"] == "rk4" else sc.les_wray3_
        return step(s["u"], s["dt"], g, s["closure"], s["nu"])
    if kind == "adjoint":
        loss, grad = sc.rollout_adjoint(g, s["closure"], s["u"], s["traj"], s["dt"], s["nu"], case["nsteps"],
                                        case["ckpt"])
        # the network's weights are single precision, and so is their gradient
        return {"loss": loss, "grad": grad.astype(np.float32)}
    if kind == "stats":
        u, nu = s["u"], s["nu"]
        return {"dt": sc.propose_timestep(u, g, nu), "energy": sc.energy(u, g), "diss": sc.get_dissipation(u, nu, g),
                "spectrum": np.array(sc.spectrum(u, g))}
    sc.to_spec_(s["spec"], s["phys"], g)
    sc.to_phys_(s["back"], s["spec"], g)
    return {"spec": s["spec"], "phys": s["back"]}


# --------------------------------------------------------------------------
# the work of one pass
# --------------------------------------------------------------------------
def work(case):
    """Bytes: the caller's inputs read once and its outputs written once.
    Operations: the real transforms (2.5 N log2 N each) and the closure network."""
    kind, n, D = case["kind"], case["n"], case.get("D", 3)
    e = 8 if case.get("dtype", "f32") == "f32" else 16  # bytes of a complex number
    npair = 3 if D == 2 else 6
    full = (n // 2 + 1) * n ** (D - 1) * e
    fft = 2.5 * n ** D * math.log2(n ** D)
    rhs = (D + npair) * fft
    stages = {"rk4": 4, "wray3": 3}
    net = 2.0 * 27 * sum(a * b for a, b in CNN_LAYERS) * n ** 3
    if kind in ("rk4", "wray3"):
        return {"bytes": 2 * D * full, "flops": stages[kind] * rhs}
    if kind == "rhs":
        return {"bytes": 2 * D * full, "flops": rhs}
    if kind == "sfs":
        nd, m = len(case["ratios"].split(",")), case["n_les"]
        les = (m // 2 + 1) * m ** 2 * e
        return {"bytes": D * full + nd * (D + npair) * les,
                "flops": rhs + nd * (D + npair) * 2.5 * m ** 3 * math.log2(m ** 3)}
    if kind == "les":
        c = case["closure"]
        extra = {"clark": 15, "smagorinsky": 15, "bardina": 15, "dynsmag": 33}.get(c, 9) * fft
        conv = net if c == "cnn" else 3 * net if c == "cnn_split" else 0.0
        return {"bytes": 2 * D * full, "flops": stages[case["stepper"]] * (rhs + extra + conv)}
    if kind == "adjoint":
        kc = n // 3
        cube = (kc + 1) * (2 * kc + 1) ** 2 * e
        nw = sum(27 * a * b + b for a, b in CNN_LAYERS)
        # per step: four stages forward, and backward with the network's input and weight gradients
        return {"bytes": 3 * full + case["nsteps"] * 3 * cube + 4 * nw,
                "flops": case["nsteps"] * 4 * 3 * (3 * net + rhs)}
    if kind == "stats":
        return {"bytes": D * full, "flops": D * fft}
    return {"bytes": 2 * (full + n ** D * e // 2), "flops": 2 * fft}


# --------------------------------------------------------------------------
# the same results in 64 bits, with torch alone
# --------------------------------------------------------------------------
_PAIRS = {2: ((0, 0), (1, 1), (0, 1)), 3: ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))}


def _phys(f, n, D):
    return torch.fft.irfftn(f, s=(n,) * D, norm="forward")


def _spec(f):
    return torch.fft.rfftn(f, norm="forward")


def _products(u, n, D, keep):
    """The spectra of u_i u_j, one pair after another."""
    v = [_phys(c * keep, n, D) for c in u]
    for i, j in _PAIRS[D]:
        yield (i, j), _spec(v[i] * v[j])


def _rhs(u, n, D, nu, stress=None):
    """-div(u u - 2 nu S + stress) on the retained modes."""
    k = _wave(n, D)
    keep = _keep(n, D)
    du = [torch.zeros_like(c) for c in u]
    for q, ((i, j), sig) in enumerate(_products(u, n, D, keep)):
        if stress is not None:
            sig += stress[q]
        sig -= 1j * nu * (k[j] * u[i] + k[i] * u[j])
        du[i] -= 1j * k[j] * sig
        if i != j:
            du[j] -= 1j * k[i] * sig
        del sig
    return [c * keep for c in du]


def _project(u, n, D):
    k = _wave(n, D)
    k2 = sum(x * x for x in k)
    k2[(0,) * D] = 1
    p = sum(a * b for a, b in zip(k, u)) / k2
    return [c - a * p for a, c in zip(k, u)]


def _force(du, u, n, D, eps):
    k2 = sum(x * x for x in _wave(n, D))
    band = (k2 >= 1) & (k2 < 9)
    w = _weight(n) * band
    e = 0.5 * sum(((c.real ** 2 + c.imag ** 2) * w).sum() for c in u)
    a = eps / (2 * e) * band
    return [d + a * c for d, c in zip(du, u)]


def _rk4(u, n, D, dt, nu, eps, tau=None):
    def f(x):
        du = _project(_rhs(x, n, D, nu, tau(x) if tau else None), n, D)
        return _force(du, x, n, D, eps) if eps is not None else du

    acc, x = list(u), list(u)
    for w, c in ((1 / 6, 0.5), (1 / 3, 0.5), (1 / 3, 1.0), (1 / 6, None)):
        k = f(x)
        acc = [a + w * dt * b for a, b in zip(acc, k)]
        if c is not None:
            x = [a + c * dt * b for a, b in zip(u, k)]
    return acc


def _wray3(u, n, D, dt, nu, tau=None):
    base = list(u)
    for a, b in ((8 / 15, 1 / 4), (5 / 12, 0.0), (3 / 4, None)):
        k = _rhs(u, n, D, nu, tau(u) if tau else None)
        u = _project([x + a * dt * y for x, y in zip(base, k)], n, D)
        if b:
            base = [x + b * dt * y for x, y in zip(base, k)]
    return u


def _gauss(n, D, delta):
    """The Gaussian filter's transfer function; modes below |k| = 3 are spared."""
    k2 = sum(x * x for x in _wave(n, D))
    return torch.where(k2 < 9, torch.ones_like(k2), torch.exp(-delta * delta * k2 / 24))


def _classical(kind, u, n, D, delta):
    """Stress spectra of the classical closures."""
    keep, k = _keep(n, D), _wave(n, D)
    pairs = _PAIRS[D]
    if kind in ("clark", "smagorinsky"):
        G = torch.stack([torch.stack([_phys(1j * k[b] * u[a] * keep, n, D) for b in range(D)], -1) for a in range(D)], -2)
        if kind == "clark":
            t = delta ** 2 / 12 * (G @ G.mT)
        else:
            S = (G + G.mT) / 2
            t = -2 * (0.17 * delta) ** 2 * torch.sqrt(2 * (S * S).sum((-1, -2), keepdim=True)) * S
        return [_spec(t[..., i, j].contiguous()) for i, j in pairs]

    def trace_free(t):
        m = sum(t[:D]) / D
        return [x - m for x in t[:D]] + list(t[D:])

    if kind == "bardina":
        f = _gauss(n, D, 2 * delta) * keep
        v = [_phys(c * f, n, D) for c in u]
        # the smooth field's own products are dealiased like the solver's, then compared in physical space
        t = [_phys(s * f, n, D) - v[i] * v[j] for (i, j), s in _products(u, n, D, keep)]
        return [_spec(x) for x in trace_free(t)]
    f = _gauss(n, D, 2 * delta) * keep

    def smag(S, width):
        s2 = sum(x * x for x in S[:D]) + 2 * sum(x * x for x in S[D:])
        return [-2 * width ** 2 * torch.sqrt(2 * s2) * x for x in S]

    strain = [0.5j * (k[j] * u[i] + k[i] * u[j]) for i, j in pairs]
    m1 = [_spec(x) for x in smag([_phys(x * keep, n, D) for x in strain], delta)]
    m2 = smag([_phys(x * f, n, D) for x in strain], math.sqrt(5.0) * delta)
    M = [_phys(a * f, n, D) - b for a, b in zip(m1, m2)]
    v = [_phys(c * f, n, D) for c in u]
    L = trace_free([_phys(s * f, n, D) - v[i] * v[j] for (i, j), s in _products(u, n, D, keep)])
    dot = lambda a, b: sum((x * y).sum() * (1 if q < D else 2) for q, (x, y) in enumerate(zip(a, b)))  # noqa: E731
    c = torch.clamp(-dot(M, L) / dot(M, M), min=0)
    return [c * x for x in m1]


def _network(u, n, ws, bs, delta, nu):
    """Stress spectra of the closure network: (u, log Re_Delta) -> four periodic convolutions."""
    F = torch.nn.functional
    keep = _keep(n, 3)
    k2 = sum(x * x for x in _wave(n, 3))
    a2 = sum(((c.real ** 2 + c.imag ** 2) * k2 * keep * _weight(n)).sum() for c in u)
    z = torch.log(delta ** 2 * torch.sqrt(a2) / nu)
    x = torch.stack([_phys(c * keep, n, 3) for c in u] + [z * torch.ones((n,) * 3, device=DEV, dtype=torch.float64)])[None]
    for i, (w, b) in enumerate(zip(ws, bs)):
        x = F.conv3d(F.pad(x, (1,) * 6, mode="circular"), w, b)
        if i < 3:
            x = F.gelu(x, approximate="tanh")
    return [_spec(c) for c in x[0]]


def exact(case, seed):
    kind, n, D = case["kind"], case["n"], case.get("D", 3)
    p = _params(case)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, p)
    with torch.no_grad():
        if kind == "transform":
            gen = torch.Generator(device=DEV).manual_seed(seed * 1009 + 29)
            x = torch.randn((n,) * D, generator=gen, device=DEV, dtype=_real(case)).double()
            return {"spec": _spec(x), "phys": x}
        u = [c.to(torch.complex128) for c in _field(D, n, _real(case), seed)]
        if kind == "rk4":
            return _rk4(u, n, D, p["dt"], p["nu"], p["eps"])
        if kind == "wray3":
            return _wray3(u, n, D, p["dt"], p["nu"])
        if kind == "rhs":
            return _rhs(u, n, D, p["nu"])
        if kind == "les":
            if case["closure"].startswith("cnn"):
                ws, bs = ([torch.from_numpy(x).to(DEV).double() for x in y] for y in _weights(seed))
                tau = lambda x: _network(x, n, ws, bs, p["delta"], p["nu"])  # noqa: E731
            else:
                tau = lambda x: _classical(case["closure"], x, n, D, p["delta"])  # noqa: E731
            if case["stepper"] == "rk4":
                return _rk4(u, n, D, p["dt"], p["nu"], None, tau)
            return _wray3(u, n, D, p["dt"], p["nu"], tau)
        if kind == "stats":
            return _exact_stats(u, n, D, p["nu"])
        return _exact_sfs(case, u, n, D)


def _exact_stats(u, n, D, nu):
    k2 = sum(x * x for x in _wave(n, D))
    keep, w = _keep(n, D), _weight(n)
    e = sum(c.real ** 2 + c.imag ** 2 for c in u)
    shell = torch.floor(torch.sqrt(k2)).long()
    spec = torch.zeros(n // 3 + 1, device=DEV, dtype=torch.float64)
    use = keep & (shell <= n // 3)
    spec.index_add_(0, shell[use], (0.5 * e * w)[use])
    vmax = torch.sqrt(sum(_phys(c * keep, n, D) ** 2 for c in u).max()).item()
    h = 2 * math.pi / n
    return {"dt": min(h / vmax, h * h / D / 2 / nu), "energy": 0.5 * (e * w).sum().item(),
            "diss": nu * (e * w * k2).sum().item(), "spectrum": spec[1:].cpu().numpy()}


def _exact_sfs(case, u, n, D):
    m = case["n_les"]
    at = torch.tensor([*range(m // 2), *range(n - m // 2, n)], device=DEV)

    def cut(f):
        f = f[at][..., : m // 2 + 1] if D == 2 else f[at][:, at][..., : m // 2 + 1]
        return f.clone()

    keep_l = _keep(m, D)
    ul = [cut(c) for c in u]
    sig = [cut(s) for _, s in _products(u, n, D, _keep(n, D))]
    ubar, tau = [], []
    for r in case["ratios"].split(","):
        f = _gauss(m, D, float(r) * 2 * math.pi / m) * keep_l
        ub = [c * f for c in ul]
        t = [(a * f - b * keep_l) for a, (_, b) in zip(sig, _products(ub, m, D, keep_l))]
        tr = sum(t[:D]) / D
        ubar.append(ub)
        tau.append([x - tr for x in t[:D]] + t[D:])
    return {"ubar": ubar, "tau": tau}


def _exact_adjoint(case, seed, p):
    n = case["n"]
    kc = n // 3
    u0 = _field(3, n, torch.float32, seed)
    with torch.no_grad():
        target = _target(case, u0).to(torch.complex128).reshape(case["nsteps"], 3, 2 * kc + 1, 2 * kc + 1, kc + 1)
    pick = torch.tensor([*range(kc + 1), *range(n - kc, n)], device=DEV)
    ws, bs = ([torch.from_numpy(x).to(DEV).double().requires_grad_() for x in y] for y in _weights(seed))
    w = _weight(n)[: kc + 1]

    def stage(x, y, z):
        u = [x, y, z]
        return tuple(_project(_rhs(u, n, 3, p["nu"], _network(u, n, ws, bs, p["delta"], p["nu"])), n, 3))

    def f(x):  # one stage at a time keeps its activations
        return torch.utils.checkpoint.checkpoint(stage, *x, use_reentrant=False)

    u = [c.to(torch.complex128) for c in u0]
    loss = 0.0
    for s in range(case["nsteps"]):
        acc, x = list(u), list(u)
        for a, c in ((1 / 6, 0.5), (1 / 3, 0.5), (1 / 3, 1.0), (1 / 6, None)):
            k = f(x)
            acc = [q + a * p["dt"] * r for q, r in zip(acc, k)]
            if c is not None:
                x = [q + c * p["dt"] * r for q, r in zip(u, k)]
        u = acc
        for c in range(3):
            d = u[c][pick][:, pick][:, :, : kc + 1] - target[s, c]
            loss = loss + ((d.real ** 2 + d.imag ** 2) * w).sum()
    loss = loss / case["nsteps"]
    loss.backward()
    grad = torch.cat([q.grad.reshape(-1) for pair in zip(ws, bs) for q in pair])
    return {"loss": loss.item(), "grad": grad.cpu().numpy()}
