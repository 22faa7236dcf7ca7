"""Cases for timing the CDD time step: what is run, on which inputs, and what the results should be.

``listed()`` gives the fixed cases and ``draw(rng)`` further ones of the same ranges; ``prepare``
builds the plan and the seeded inputs of a case on the GPU, ``run`` is one pass through the public
entry points, ``work`` the bytes and operations a pass cannot do without and ``exact`` the result of
the first pass in plain FP64 torch, written independently of the library.

Fields are seeded Gaussian random fields (rms 0.05, sigma given in units of the box), mu = 1,
nu = 0.3, CFL 0.25 and, where a case is loaded, the traceless strain rate r (-1/2, -1/2, 1).
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-plasticity_b200"))

import cdd  # noqa: E402
from cdd.adjoint import Rollout  # noqa: E402

MU, NU, RMS = 1.0, 0.3, 0.05
VACANCY = (0.4, 0.7, 0.02)          # alpha, beta, gamma of the vacancy coupling
EPS = 2.220446049250313080847263336181640625e-16
# the 2-D and 3-D grids of the ensemble, most cells last
ENSEMBLE = ((256, 256), (512, 512), (48, 48, 48), (64, 64, 64), (96, 96, 96), (128, 128, 128))
FIELDS = ("beta_elastic", "rotation", "rodrigues", "rho")


def listed():
    return [
        # a 2-D run at the size of the 2-D example: a few microseconds of work per kernel, so launches count
        dict(name="run 2d 128 f64", op="run", shape="128x128", prec="f64", steps=10, sigma=0.05, rate=0.0),
        # one flux evaluation of a small 3-D grid, called eagerly: the smallest call
        dict(name="flux 24 f32", op="flux", shape="24x24x24", prec="f32", sigma=0.08, rate=0.05),
        # a short run of a small 3-D grid with uneven axes (2^a 3^b and 2^a 5^c)
        dict(name="run 36x40x54 f64", op="run", shape="36x40x54", prec="f64", steps=5, sigma=0.08, rate=0.05),
        # the drop-in: FP64 128^3 under load
        dict(name="run 128 f64", op="run", shape="128x128x128", prec="f64", steps=1, sigma=0.04, rate=0.05),
        # the FP32 form at 256^3, and the plain FP64 form of the same grid (the largest)
        dict(name="run 256 f32", op="run", shape="256x256x256", prec="f32", steps=1, sigma=0.03, rate=0.05),
        dict(name="run 256 f64", op="run", shape="256x256x256", prec="f64", steps=1, sigma=0.03, rate=0.05),
        # an uneven ensemble in one plan: per-instance time steps, six shapes
        dict(name="ensemble 24 f32", op="ensemble", each=4, prec="f32", steps=1),
        # gradients of a rollout's loss (forward, segment re-runs and reverse sweep), FP32 and FP64
        dict(name="gradient 64 f32", op="gradient", shape="64x64x64", prec="f32", steps=10, keep=5, sigma=0.05,
             rate=0.05),
        dict(name="gradient 32 f64", op="gradient", shape="32x32x32", prec="f64", steps=4, keep=2, sigma=0.08,
             rate=0.05),
        # the glide-only dynamics on a 2^a 3 grid
        dict(name="glide 96 f32", op="glide", shape="96x96x96", prec="f32", steps=1, sigma=0.05, rate=0.05),
        # vacancy coupling with its diffusion, a wide 3-D grid
        dict(name="vacancy 32x100x128 f64", op="vacancy", shape="32x100x128", prec="f64", steps=2, sigma=0.05,
             rate=0.0),
        # an output time: energy and mean strain, the k-space field observables, and the field in file order
        dict(name="output 128 f64", op="output", shape="128x128x128", prec="f64", sigma=0.04),
    ]


def _sizes(low, high):
    """Even lengths 2^a 3^b or 2^a 5^c."""
    got = set()
    for q in (3, 5):
        a = 2
        while a <= high:
            v = a
            while v <= high:
                if v >= low:
                    got.add(v)
                v *= q
            a *= 2
    return sorted(got)


def _shape(rng, nd, low, high, most):
    """A grid of `nd` axes whose cells are spread over the logarithm of [low^nd, most]."""
    want = math.exp(rng.uniform(math.log(low ** nd), math.log(most)))
    sizes, got = _sizes(low, high), []
    for left in range(nd, 0, -1):
        mean = want ** (1.0 / left) * (rng.uniform(0.6, 1.6) if left > 1 else 1.0)
        n = min(sizes, key=lambda s: abs(math.log(s / max(mean, 1.0))))
        got.append(n)
        want /= n
    while math.prod(got) > most:
        got[got.index(max(got))] = max(s for s in sizes if s < max(got))
    rng.shuffle(got)
    return "x".join(str(n) for n in got)


def draw(rng):
    op = rng.choice(("run", "run", "run", "flux", "ensemble", "gradient", "glide", "vacancy", "output"))
    prec = rng.choice(("f32", "f64"))
    c = dict(op=op, prec=prec)
    if op == "ensemble":
        c.update(each=rng.randint(1, 6), steps=1, prec="f32")
        return c
    nd = rng.choice((2, 3, 3))
    most = {"gradient": 64 ** 3 if prec == "f32" else 48 ** 3, "run": 256 ** 3, "flux": 256 ** 3}.get(op, 128 ** 3)
    if nd == 2:
        most = min(most, 1024 ** 2)
    c["shape"] = _shape(rng, nd, 64 if nd == 2 else 24, 1024 if nd == 2 else 256, most)
    c["sigma"] = round(rng.uniform(0.04, 0.08), 4)
    if op != "output":
        c["rate"] = 0.0 if op == "vacancy" else rng.choice((0.0, round(rng.uniform(0.01, 0.1), 4)))
    if op == "gradient":
        c["steps"], c["keep"] = rng.randint(2, 6), rng.randint(1, 4)
    elif op not in ("flux", "output"):
        c["steps"] = rng.randint(1, 4) if most <= 128 ** 3 else 1
    return c


# ------------------------------------------------------------------ inputs
def _grid(case):
    return tuple(int(n) for n in case["shape"].split("x"))


def _members(case):
    """(shape, sigma, rate) of each instance of an ensemble: spread evenly over [0.02, 0.08] and [0, 0.1]."""
    n = case["each"]
    return [(s, 0.02 + 0.06 * (k + 0.5) / n, 0.1 * (k + 0.5) / n) for s in ENSEMBLE for k in range(n)]


def _ksq(shape, device):
    total = 0.0
    for d, n in enumerate(shape):
        m = torch.arange(n // 2 + 1, device=device, dtype=torch.float64) if d == len(shape) - 1 else \
            torch.fft.fftfreq(n, d=1.0 / n, device=device, dtype=torch.float64)
        view = [1] * len(shape)
        view[d] = -1
        total = total + ((2.0 * math.pi * m) ** 2).view(view)
    return total


def _random(shape, sigma, seed, comps=9):
    """White noise per component, filtered by exp(-|k|^2 sigma^2 / 2) and scaled to rms 0.05 (FP64)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    out = torch.empty((comps,) + shape, dtype=torch.float64, device="cuda")
    filt = torch.exp(-0.5 * sigma * sigma * _ksq(shape, "cuda"))
    dims = tuple(range(len(shape)))
    for c in range(comps):
        white = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
        out[c] = torch.fft.irfftn(torch.fft.rfftn(white, dim=dims) * filt, s=shape, dim=dims)
    return out.mul_(RMS / out.square().mean().sqrt())


def _dtype(case):
    return torch.float64 if case["prec"] == "f64" else torch.float32


def _inputs(case, seed):
    """The case's fields, rounded to its precision (FP64 or FP32 values)."""
    if case["op"] == "ensemble":
        return [_random(s, sig, 1000 * seed + k).to(_dtype(case)) for k, (s, sig, _) in enumerate(_members(case))]
    return [_random(_grid(case), case["sigma"], 1000 * seed).to(_dtype(case))]


def _vacancies(case, seed):
    return (_random(_grid(case), case["sigma"], 1000 * seed + 7, comps=1)[0] + 0.1).to(_dtype(case))


def _load(rate):
    return None if not rate else (-0.5 * rate, -0.5 * rate, rate)


def _fixed_dt(case):
    return 0.1 / max(_grid(case))


# ------------------------------------------------------------------ the passes
def prepare(case, seed):
    op, s = case["op"], {"op": case["op"], "steps": case.get("steps", 1)}
    fields = _inputs(case, seed)
    if op == "gradient":
        s["rollout"] = Rollout(_grid(case), MU, NU, case["rate"] or None, _fixed_dt(case), case["steps"],
                               precision=case["prec"], checkpoint_every=case["keep"])
        s["beta"] = s["rollout"].plan.pack(fields)
        return s
    if op == "ensemble":
        insts = [cdd.Instance(sh, mu=MU, nu=NU, cfl=0.25, load_rate=_load(r)) for sh, _, r in _members(case)]
    else:
        insts = [cdd.Instance(_grid(case), mu=MU, nu=NU, cfl=0.25, load_rate=_load(case.get("rate")),
                              glide_only=op == "glide", vacancy=VACANCY if op == "vacancy" else None,
                              dt_max=0.01 if op == "vacancy" else 0.0)]
    plan = s["plan"] = cdd.Plan(insts, case["prec"])
    s["beta"] = plan.pack(fields)
    if op == "vacancy":
        s["c"] = plan.empty_vacancy()
        plan.vacancy_view(s["c"], 0).copy_(_vacancies(case, seed))
        plan.set_vacancy(s["c"])
    plan.set_time(0.0)
    return s


def run(state):
    op, beta = state["op"], state["beta"]
    if op == "gradient":
        # the whole of a gradient evaluation: the loss at the end of the rollout, then its gradients
        uN, loss = state["rollout"].forward(beta)
        g, params = state["rollout"].backward()
        return {"uN": uN, "loss": loss, "beta": g, "params": [params[k] for k in ("mu", "nu", "rate_zz")]}
    plan = state["plan"]
    if op == "flux":
        rhs, speed = plan.flux(beta, 0.5)
        return {"rhs": rhs, "speed": speed}
    if op == "output":
        energy, mean = plan.observables(beta)
        out = {"energy": energy, "mean": mean, "file": plan.export_field(beta)}
        for kind in FIELDS:
            out[kind] = plan.observe(kind, beta)
        return out
    # adaptive steps of the plan's own clock; the field is advanced in place
    plan.run(beta, state["steps"])
    if op == "vacancy":
        return {"beta": beta, "c": state["c"]}
    return {"beta": beta}


def work(case):
    """Bytes: inputs read once and outputs written once. Operations: per cell and flux evaluation 1300
    (3-D; the limited derivatives, corner velocities and sums) or 620 (2-D), and 2.5 log2(cells) per
    cell and real transform."""
    op, el = case["op"], 8 if case["prec"] == "f64" else 4

    def cost(shape):
        n, nd = math.prod(shape), len(shape)
        flux, fft = n * (1300.0 if nd == 3 else 620.0), 2.5 * n * math.log2(n)
        solve = 12 * fft + 100.0 * n
        if op == "flux":
            return 19 * el * n, flux + solve
        if op == "output":
            return el * n * (9 + 9 + 9 + 3 + 3 + 9), solve + fft * (15 + 9 + 9 + 18) + 200.0 * n
        if op == "gradient":
            # forward, one re-run of every step but the last segment's, reverse at about twice a flux
            again = max(0, case["steps"] - case["keep"]) / case["steps"]
            return 27 * el * n, case["steps"] * 3 * (flux + solve) * (3 + again)
        extra = 2 * el * n if op == "vacancy" else 0
        return 18 * el * n + extra, case["steps"] * (3 * (flux + solve) + (2 * fft if op == "vacancy" else 0.0))

    parts = [cost(s) for s in (ENSEMBLE * case["each"] if op == "ensemble" else (_grid(case),))]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


# ------------------------------------------------------------------ the same in plain FP64 torch
SYM = ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))


class _Box:
    """The k tables of a grid: n 2 pi m / n with the Nyquist value positive, n the grid's scale."""

    def __init__(self, shape):
        self.shape, self.nd = shape, len(shape)
        self.dims = tuple(range(-self.nd, 0))
        k = []
        for d, n in enumerate(shape):
            i = torch.arange(n // 2 + 1 if d == self.nd - 1 else n, dtype=torch.float64, device="cuda")
            a = 2.0 * math.pi * i / n
            a = torch.where(a > math.pi, a - 2.0 * math.pi, a)
            view = [1] * self.nd
            view[d] = -1
            k.append((shape[d] if self.nd == 3 else shape[-1]) * a.view(view))
        self.k = k + [torch.zeros((), dtype=torch.float64, device="cuda")] * (3 - self.nd)
        self.q2 = sum(v * v for v in self.k)
        self.mask = torch.ones(self.q2.shape, dtype=torch.float64, device="cuda")
        self.mask[(0,) * self.nd] = 0.0
        self.i2, self.i4 = 1.0 / (self.q2 + EPS), 1.0 / (self.q2 * self.q2 + EPS)

    def f(self, x):
        return torch.fft.rfftn(x, dim=self.dims)

    def b(self, x):
        return torch.fft.irfftn(x, s=self.shape, dim=self.dims)

    def elastic(self, beta):
        """k_i g_j per component, the transform of beta^E + beta^P."""
        k, w = self.k, [self.f(beta[c]) for c in range(9)]
        lam = 2.0 * MU * NU / (1.0 - 2.0 * NU)
        A, B = lam / (lam + 2.0 * MU), 2.0 * (lam + MU) / (lam + 2.0 * MU)
        tr = w[0] + w[4] + w[8]
        v = [sum(k[m] * (w[3 * m + j] + w[3 * j + m]) for m in range(3)) for j in range(3)]
        r = 0.5 * sum(k[m] * v[m] for m in range(3))
        g = [self.mask * (k[j] * (A * tr * self.i2 - B * r * self.i4) + v[j] * self.i2) for j in range(3)]
        return lambda i, j: k[i] * g[j]

    def beta_e(self, beta):
        kg = self.elastic(beta)
        return torch.stack([self.b(kg(c // 3, c % 3)) - beta[c] for c in range(9)])

    def stress(self, beta):
        lam = 2.0 * MU * NU / (1.0 - 2.0 * NU)
        e = self.beta_e(beta)
        tr = e[0] + e[4] + e[8]
        return torch.stack([MU * (e[3 * i + j] + e[3 * j + i]) + (lam * tr if i == j else 0.0) for i, j in SYM])


def _energy(s):
    sq = s[0] ** 2 + s[3] ** 2 + s[5] ** 2 + 2.0 * (s[1] ** 2 + s[2] ** 2 + s[4] ** 2)
    return ((sq - NU / (1.0 + NU) * (s[0] + s[3] + s[5]) ** 2) / (4.0 * MU)).sum()


def _one_sided(u, d):
    """Minmod-limited forward and backward derivatives along grid axis d (spacing 1 / last length)."""
    n = u.shape[-1]
    dim = d - (u.dim() - 1)
    diff = torch.roll(u, -1, dim) - u
    e = torch.roll(diff, -1, dim) - diff
    p = torch.roll(e, 1, dim)
    dd = torch.where(e * p > 0, torch.where(e.abs() <= p.abs(), e, p), torch.zeros_like(e))
    return (diff - 0.5 * dd) * n, torch.roll(diff + 0.5 * dd, 1, dim) * n


def _flux(u, s6, glide):
    """rhs and CFL speed of the central-upwind scheme for the total stress s6."""
    nd = u.dim() - 1
    S = [[s6[SYM.index((min(i, j), max(i, j)))] for j in range(3)] for i in range(3)]
    D = [_one_sided(u, d) for d in range(nd)]          # D[d][0]: forward, D[d][1]: backward

    def corner(c):
        return [D[d][(c >> d) & 1] for d in range(nd)]

    def velocity(us):
        v = []
        for l in range(3):
            a = sum(us[d][3 * l + n] * S[d][n] for d in range(nd) for n in range(3))
            if l < nd:
                a = a - sum(us[l][3 * m + n] * S[m][n] for m in range(3) for n in range(3))
            v.append(a)
        if glide:
            g = []
            for d in range(3):
                a = -sum(us[e][3 * d + e] for e in range(nd))
                if d < nd:
                    a = a + us[d][0] + us[d][4] + us[d][8]
                g.append(a)
            f = (EPS + sum(a * b for a, b in zip(v, g))) / (EPS + sum(a * a for a in g))
            v = [a + b * f for a, b in zip(v, g)]
        rho = EPS
        for d in range(nd):
            rho = rho + sum(us[d][3 * l + j] ** 2 for l in range(3) if l != d for j in range(3))
            for e in range(d + 1, nd):
                rho = rho - 2.0 * sum(us[d][3 * e + j] * us[e][3 * d + j] for j in range(3))
        rho = rho ** 0.5
        return [a / rho for a in v]

    corners = range(1 << nd)
    V = [velocity(corner(c)) for c in corners]
    zero = torch.zeros_like(V[0][0])
    up = [torch.stack([V[c][d] for c in corners] + [zero]).amax(0) for d in range(nd)]
    dn = [-torch.stack([V[c][d] for c in corners] + [zero]).amin(0) for d in range(nd)]
    tot = [a + b + EPS for a, b in zip(up, dn)]
    rhs = sum((D[d][0] - D[d][1]) * (dn[d] * up[d] / tot[d]) for d in range(nd))
    norm = math.prod(tot[1:], start=tot[0])
    for c in corners:
        us = corner(c)
        w = math.prod([(up if (c >> d) & 1 else dn)[d] for d in range(1, nd)], start=(up if c & 1 else dn)[0]) / norm
        H = [sum(us[d][q] * V[c][d] for d in range(nd))
             - (sum(V[c][l] * us[q // 3][3 * l + q % 3] for l in range(3)) if q // 3 < nd else 0.0) for q in range(9)]
        rhs = rhs - torch.stack(H) * w
    return rhs, sum(tot)


def _total(box, u, t, rate):
    s = box.stress(u)
    if not rate:
        return s
    shift = torch.zeros(6, dtype=torch.float64, device="cuda")
    shift[0] = shift[3] = -MU * rate * t
    shift[5] = 2.0 * MU * rate * t
    return s + shift.view((6,) + (1,) * box.nd)


def _rk3(box, u, t, rate, dt=None, glide=False, vac=None, bound=0.0):
    def load(v):
        s = _total(box, v, t, rate)
        if vac is not None:
            s = s.clone()
            s[[0, 3, 5]] -= VACANCY[0] * vac
        return s

    L, speed = _flux(u, load(u), glide)
    if dt is None:
        dt = 0.25 / (max(box.shape) * float(speed.max()))
        dt = min(dt, bound) if bound else dt
    f = u + dt * L
    f = 0.75 * u + 0.25 * f + 0.25 * dt * _flux(f, load(f), glide)[0]
    return u / 3.0 + 2.0 / 3.0 * f + 2.0 / 3.0 * dt * _flux(f, load(f), glide)[0], dt


def _trace(u):
    return u[0] + u[4] + u[8]


def _run64(case, box, u, rate, seed):
    t, glide = 0.0, case["op"] == "glide"
    c = _vacancies(case, seed).double() if case["op"] == "vacancy" else None
    for _ in range(case["steps"]):
        new, dt = _rk3(box, u, t, rate, glide=glide, vac=c, bound=0.01 if c is not None else 0.0)
        if c is not None:
            c = c + VACANCY[1] * (_trace(new) - _trace(u))
            c = box.b(box.f(c) * torch.exp(-VACANCY[2] * dt * box.q2))
        u, t = new, t + dt
    return (u, c)


def _gradient64(case, box, u0):
    rate = case["rate"]
    dt = _fixed_dt(case)
    with torch.no_grad():
        us = [u0]
        for n in range(case["steps"]):
            us.append(_rk3(box, us[-1], n * dt, rate, dt)[0])
    # the parameter gradients come out of the code alone
    uN = us[-1].clone().requires_grad_(True)
    loss = _energy(box.stress(uN)) + 10.0 * uN[8].mean()
    g, = torch.autograd.grad(loss, uN)
    for n in reversed(range(case["steps"])):
        v = us[n].clone().requires_grad_(True)
        g, = torch.autograd.grad(_rk3(box, v, n * dt, rate, dt)[0], v, g)
    return {"uN": us[-1].reshape(-1), "loss": float(loss), "beta": g.reshape(-1), "params": [None, None, None]}


def _output64(box, u):
    kg, k = box.elastic(u), box.k
    out = {"energy": _energy(box.stress(u)).view(1), "mean": u[8].mean().view(1),
           "file": u.permute((0,) + tuple(range(box.nd, 0, -1))).contiguous()}
    e = box.beta_e(u)
    out["beta_elastic"] = e
    out["rotation"] = torch.stack([(e[3 * i + j] - e[3 * j + i]) / 2 for i, j in ((0, 1), (0, 2), (1, 2))])
    del e, kg
    w = [box.f(u[c]) for c in range(9)]
    q = [0.5 * sum(k[n] * (w[3 * j + n] + w[3 * n + j]) for n in range(3)) for j in range(3)]
    rod = [box.b(box.mask * box.i2 * (k[(a + 1) % 3] * q[(a + 2) % 3] - k[(a + 2) % 3] * q[(a + 1) % 3]))
           for a in range(3)]
    out["rodrigues"] = torch.stack([rod[a] - 0.5 * (u[3 * ((a + 1) % 3) + (a + 2) % 3]
                                                    - u[3 * ((a + 2) % 3) + (a + 1) % 3]) for a in range(3)])
    rho = []
    for a in range(3):
        p, r = (a + 1) % 3, (a + 2) % 3
        rho += [box.b(1j * (k[r] * w[3 * p + i] - k[p] * w[3 * r + i])) for i in range(3)]
    out["rho"] = torch.stack(rho)
    return {n: out[n].reshape(-1) if n in FIELDS else out[n] for n in out}


def exact(case, seed):
    if math.prod(_grid(case) if "shape" in case else (case["each"],)) * (3 if case["op"] == "gradient" else 1) > 2 ** 25:
        return None
    fields = [f.double() for f in _inputs(case, seed)]
    if case["op"] == "ensemble":
        outs = []
        for u, (shape, _, rate) in zip(fields, _members(case)):
            outs.append(_run64(case, _Box(shape), u, rate, seed)[0].reshape(-1))
        return {"beta": torch.cat(outs)}
    box, u = _Box(_grid(case)), fields[0]
    if case["op"] == "gradient":
        return _gradient64(case, box, u)
    if case["op"] == "flux":
        rhs, speed = _flux(u, _total(box, u, 0.5, case["rate"]), False)
        return {"rhs": rhs.reshape(-1), "speed": speed.reshape(-1)}
    if case["op"] == "output":
        return _output64(box, u)
    u, c = _run64(case, box, u, case["rate"], seed)
    if c is not None:
        return {"beta": u.reshape(-1), "c": c.reshape(-1)}
    return {"beta": u.reshape(-1)}
