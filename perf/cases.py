"""The work this framework is measured on: its public entry points over the sizes they are used at.

A case is one call (or one short sequence of calls) that a program makes once it holds an object:
chi^2 of one model, of a few hundred, of a hundred thousand; a simplex fit; a batch of fits of
uneven objects; the model curve of the plot mode, its periodogram, the animation's frames.
Objects are synthetic, in the shapes of the benchmark configurations (c0: 300 points in 5 nights,
c1: 480 points over 8 days in 2 filters, c2: 2000 points over 60 days in 3 filters with observed
minima, c3: objects of three variants, 50-2000 points, 1-4 filters): a tumbling body that a fit
would end on, its light curve at nightly times with 0.1 mag of noise.

Vectors come in two kinds: "near", the points that the simplexes of a re-optimisation visit around
a model, and "wide", one independent body per vector, as a screening of unrelated models.

A model without ACC computes in CHI_FLOAT = float: its chi^2 and delta_V are floats in the API's
double arrays, and are kept as float32 here, which changes no value.
"""
import ctypes
import math

import numpy as np
import torch

from asteroid_gb300 import api, capi

PREC = {"fp64": api.PREC_FP64, "mixed": api.PREC_MIXED, "rhs32": api.PREC_MIXED_RHS32}


def listed():
    return [
        # chi^2 of one model: what the plot mode and a check of one result call; latency alone.
        dict(name="eval_1_fp64", kind="eval", flags="TORQUE,P_PSI,ACC", prec="fp64", n=1, vectors="near",
             points=300, filters=1, days=5, step=1e-2, minima=0),
        # A screening of a few hundred models, black-and-white-ball variant, odd count.
        dict(name="eval_337_fp64_ball", kind="eval", flags="BW_BALL,ACC", prec="fp64", n=337, vectors="wide",
             points=611, filters=3, days=17, step=1e-2, minima=0),
        # The same in mixed precision for a photometric shape of its own (free rotation).
        dict(name="eval_1001_mixed_bc", kind="eval", flags="BC,INTERP", prec="mixed", n=1001, vectors="near",
             points=480, filters=2, days=8, step=1e-2, minima=0),
        # The plain path at a size that fills the GPU (the default precision of every entry point).
        dict(name="eval_20k_fp64", kind="eval", flags="TORQUE,INTERP,ACC", prec="fp64", n=20011, vectors="wide",
             points=480, filters=2, days=8, step=1e-2, minima=0),
        # The mixed path's ordinary batch: the reference's default build (float), c1's shape.
        dict(name="eval_120k_mixed", kind="eval", flags="TORQUE,INTERP", prec="mixed", n=120000, vectors="near",
             points=480, filters=2, days=8, step=1e-2, minima=0),
        # The long light curve with observed minima, c2's shape: 12 500 RK4 steps an evaluation.
        dict(name="eval_60k_mixed_long", kind="eval", flags="TORQUE,P_PSI,INTERP,NUDGE", prec="mixed", n=58368,
             vectors="near", points=2000, filters=3, days=60, step=5e-3, minima=5),
        # A random-start search in the default precision, c0: every chain from the prior.
        dict(name="fit_2048_fp64", kind="fit", flags="TORQUE,P_PSI,ACC", prec="fp64", chains=2048, group=256, evals=20,
             reopt=False, points=300, filters=1, days=5, step=1e-2),
        # A re-optimisation of a found model with the default number of chains, mixed search.
        dict(name="fit_14336_mixed", kind="fit", flags="TORQUE,P_PSI,ACC", prec="mixed", chains=14336, group=256,
             evals=40, reopt=True, points=300, filters=1, days=5, step=1e-2),
        # Uneven objects of the three variants in one persistent launch, FP64 results.
        dict(name="batch_24_objects", kind="batch", objects=24, chains=256, evals=30, step=1e-2),
        # The plot mode's model curve on its 20 000-point grid.
        dict(name="curve_20000", kind="curve", flags="TORQUE,P_PSI,ACC", points=20000, days=5, step=1e-2),
        # The plot mode's periodogram of a long curve.
        dict(name="periodogram_20000", kind="periodogram", points=20000, days=60),
        # Frames of the animation at its own size.
        dict(name="frames_24", kind="frames", frames=24, pixels=1080),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval"] * 6 + ["fit"] * 2 + ["batch", "curve", "periodogram", "frames"])
    if kind == "eval":
        prec = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed", "rhs32"])
        variant = rng.choice(["TORQUE", "BC", "BW_BALL", "TORQUE,P_PSI"])
        interp = rng.choice(["", ",INTERP"])
        acc = ",ACC" if prec == "fp64" else ""
        points, days = _logint(rng, 50, 2000), rng.randint(3, 60)
        # RK4 steps and observations of one evaluation bound the count.
        cost = points + days * 100
        n = _logint(rng, 1, max(2, min(120000, (3e7 if prec == "fp64" else 1.2e8) / cost)))
        return dict(kind="eval", flags=variant + interp + acc, prec=prec, n=n,
                    vectors="near" if prec != "fp64" else rng.choice(["near", "wide"]), points=points,
                    filters=rng.randint(1, 4), days=days, step=1e-2, minima=0)
    if kind == "fit":
        prec = rng.choice(["fp64", "mixed"])
        return dict(kind="fit", flags=rng.choice(["TORQUE,P_PSI,ACC", "TORQUE,ACC", "BC,ACC"]), prec=prec,
                    chains=64 * _logint(rng, 1, 24 if prec == "fp64" else 224), group=64, evals=rng.randint(14, 40),
                    reopt=prec == "mixed", points=_logint(rng, 50, 300), filters=rng.randint(1, 3),
                    days=rng.randint(3, 6), step=1e-2)
    if kind == "batch":
        return dict(kind="batch", objects=rng.randint(2, 24), chains=64 * rng.randint(1, 4), evals=rng.randint(14, 30),
                    step=1e-2)
    if kind == "curve":
        return dict(kind="curve", flags=rng.choice(["TORQUE,P_PSI,ACC", "BC,INTERP,ACC", "BW_BALL,ACC"]),
                    points=_logint(rng, 300, 20000), days=rng.randint(3, 20), step=1e-2)
    if kind == "periodogram":
        return dict(kind="periodogram", points=_logint(rng, 1000, 20000), days=rng.randint(3, 60))
    return dict(kind="frames", frames=rng.randint(1, 24), pixels=2 * _logint(rng, 60, 540))


# ---------------------------------------------------------------- objects

class Body:
    """A synthetic object: its variant, its observation times and vectors, one regular tumbler."""

    def __init__(self, rng, flags, points, filters, days, step, minima=0):
        self.flags = api.flags_from_names(flags)
        self.model = api.make_model(self.flags, step, (20.0, 4800.0))
        self.names = api.param_names(self.model)
        self.step = step
        t = rng.uniform(0.0, 0.25, points) + rng.integers(0, days, points)
        t = np.unique(t)
        t = t - t[0]
        self.t = t
        n = len(t)
        self.filt = rng.integers(0, filters, n).astype(np.int32)
        self.filt[:filters] = np.arange(filters)
        self.filters = filters
        self.eph_t = np.array([-1.0, 0.5 * t[-1], t[-1] + 1.0])
        e, s = self._tracks(self.eph_t)
        self.eph_e, self.eph_s = e.T.copy(), s.T.copy()
        e, s = self._tracks(t)
        self.e = e / np.linalg.norm(e, axis=1, keepdims=True)
        self.s = s / np.linalg.norm(s, axis=1, keepdims=True)
        self.truth = self.wide(rng, 1)[0]
        self.minima = minima

    def _tracks(self, t):
        """Asteroid -> Earth and asteroid -> Sun (au): linear tracks near 1 and 1.2 au."""
        d = np.asarray(t) - 0.5 * self.t[-1]
        a = np.stack([1.2 * math.cos(0.52) - 0.010 * d, 1.2 * math.sin(0.52) + 0.015 * d, 0.05 + 0.002 * d], -1)
        e = np.stack([1.0 + 0 * d, 0.0172 * d, 0 * d], -1)
        return e - a, -a

    def wide(self, rng, n):
        """n independent bodies: a spin that the fixed step resolves, clear of the separatrix and
        of principal-axis rotation, a torque that changes it by a few percent over the span."""
        v = {k: np.zeros(n) for k in self.names}
        u = lambda lo, hi: rng.uniform(lo, hi, n)
        v["theta_M"], v["phi_M"], v["phi_0"] = np.arccos(u(-0.95, 0.95)), u(0, 2 * np.pi), u(0, 2 * np.pi)
        c = np.exp(u(math.log(0.2), math.log(0.65)))
        b = c ** u(0.25, 0.75)
        isv, iiv = (b * b + c * c) / (1 + b * b), (b * b + c * c) / (1 + c * c)
        lam = rng.random(n) < 0.5
        x = u(0.1, 0.35)
        es_l = 2 * x * (1 - iiv) + iiv
        es_s = 2 * x * (iiv - isv) + isv
        ii, is_ = 1 / iiv, 1 / isv
        psi_m = np.arctan(np.sqrt(np.maximum(ii * (is_ - 1 / es_s) / is_ / (1 / es_s - ii), 0)))
        v["c_tumb"], v["b_tumb"] = c, b
        v["Es"] = np.where(lam, es_l, es_s)
        v["psi_0"] = np.where(lam, u(0, 2 * np.pi), u(-0.8, 0.8) * psi_m)
        v["L"] = np.exp(u(math.log(16.0), math.log(min(60.0, 0.3 / self.step))))
        for k in ("Ti", "Ts", "Tl"):
            if k in v:
                v[k] = u(-0.02, 0.02) * v["L"] / max(self.t[-1], 1.0)
        if "c" in v:
            v["c"] = c * u(0.9, 1.1)
            v["b"] = b * u(0.9, 1.1)
        if "kappa" in v:
            v["theta_R"], v["phi_R"], v["kappa"] = u(0.3, 2.8), u(0, 2 * np.pi), np.exp(u(math.log(0.015), math.log(0.09)))
        return np.stack([v[k] for k in self.names], 1)

    def near(self, rng, n):
        """n points within a re-optimisation's reach of the truth."""
        p = np.repeat(self.truth[None], n, 0)
        width = {"L": 0.3, "theta_M": 5e-3, "phi_M": 5e-3, "phi_0": 5e-3, "psi_0": 5e-3, "theta_R": 5e-3, "phi_R": 5e-3}
        for i, k in enumerate(self.names):
            w = width.get(k, 1e-3 * abs(self.truth[i]))
            p[:, i] += rng.uniform(-w, w, n)
        return p

    def light_curve(self, rng):
        """api.Obs with the truth's magnitudes, offsets of the filters and 0.1 mag of noise."""
        if not hasattr(self, "v"):
            mag = self.base_curve()
            off = 22.0 + rng.uniform(-0.5, 0.5, self.filters)
            self.v = (mag + off[self.filt] + rng.normal(0, 0.1, len(self.t))).astype(np.float32)
            self.t_min = self.v_min = np.zeros(0, np.float32)
            if self.minima:
                i = np.arange(1, len(mag) - 1)
                i = i[(mag[i] > mag[i - 1]) & (mag[i] >= mag[i + 1])]
                i = i[np.unique(np.linspace(0, len(i) - 1, self.minima).round().astype(int))]
                self.t_min, self.v_min = self.t[i].astype(np.float32), (mag[i] + off[0]).astype(np.float32)
        return api.Obs(self.t, self.v, np.full(len(self.t), 100.0, np.float32), self.filt, self.e, self.s, self.eph_e,
                       self.eph_s, self.eph_t, self.t_min, self.v_min)

    def base_curve(self):
        return _magnitudes(self, self.truth[None], self.t, self.e, self.s, "cpu")[:, 0].numpy()


# ---------------------------------------------------------------- the model in plain FP64

def _angles_one(body, p, t):
    """Euler angles [len(t), 3] of one body: RK4 with plain floats."""
    q = dict(zip(body.names, (float(x) for x in p)))
    y, mu, torque = _start(body, {k: torch.tensor(x, dtype=torch.float64) for k, x in q.items()})
    y, mu = [float(x) for x in y], [float(x) for x in mu]
    sin, cos = math.sin, math.cos
    out = np.empty((len(t), 3))
    if torque:
        a, b, c, ta, tb, tc = mu

        def f(w0, w1, w2, ph, th, ps):
            s5, c5, s4 = sin(ps), cos(ps), sin(th)
            k3 = (w0 * s5 + w1 * c5) / s4
            return a * w1 * w2 + ta, b * w2 * w0 + tb, c * w0 * w1 + tc, k3, w0 * c5 - w1 * s5, w2 - k3 * cos(th)
    else:
        big, ip, im = mu

        def f(ph, th, ps):
            k0 = big * (ip - im * cos(2 * ps))
            return k0, big * im * sin(th) * sin(2 * ps), cos(th) * (big - k0)
    y = tuple(y)
    for i in range(len(t)):
        if i:
            n = int((t[i] - t[i - 1]) / body.step + 1)
            h = (t[i] - t[i - 1]) / n
            for _ in range(n):
                k1 = f(*y)
                k2 = f(*[u + 0.5 * h * v for u, v in zip(y, k1)])
                k3 = f(*[u + 0.5 * h * v for u, v in zip(y, k2)])
                k4 = f(*[u + h * v for u, v in zip(y, k3)])
                y = tuple(u + h / 6.0 * (p + 2 * q + 2 * r + s) for u, p, q, r, s in zip(y, k1, k2, k3, k4))
        out[i] = y[-3:]
    return out


def _start(body, q):
    """Initial state and the constants of the rotation from the parameters (tensors by name)."""
    b, c, psi = q["b_tumb"], q["c_tumb"], q["psi_0"]
    is_, ii = (1 + b * b) / (b * b + c * c), (1 + c * c) / (b * b + c * c)
    theta = torch.asin(torch.sqrt((q["Es"] - 1) / (torch.sin(psi) ** 2 * (1 / ii - 1 / is_) + 1 / is_ - 1)))
    big = q["L"]
    if body.flags & api.TORQUE:
        w = [big / ii * torch.sin(theta) * torch.sin(psi), big / is_ * torch.sin(theta) * torch.cos(psi), big * torch.cos(theta)]
        return w + [q["phi_0"], theta, psi], [(is_ - 1) / ii, (1 - ii) / is_, ii - is_, q["Ti"], q["Ts"], q["Tl"]], True
    return [q["phi_0"], theta, psi], [big, 0.5 * (1 / ii + 1 / is_), 0.5 * (1 / ii - 1 / is_)], False


def _angles_many(body, P, t):
    """Euler angles [len(t), 3, n] of n bodies at once, on P's device."""
    y, mu, torque = _start(body, {k: P[:, i] for i, k in enumerate(body.names)})
    y = torch.stack([v.expand(P.shape[0]) for v in y])

    def f(y):
        if torque:
            w0, w1, w2, _, th, ps = y
            s5, c5 = torch.sin(ps), torch.cos(ps)
            k3 = (w0 * s5 + w1 * c5) / torch.sin(th)
            return torch.stack([mu[0] * w1 * w2 + mu[3], mu[1] * w2 * w0 + mu[4], mu[2] * w0 * w1 + mu[5], k3,
                                w0 * c5 - w1 * s5, w2 - k3 * torch.cos(th)])
        _, th, ps = y
        k0 = mu[0] * (mu[1] - mu[2] * torch.cos(2 * ps))
        return torch.stack([k0, mu[0] * mu[2] * torch.sin(th) * torch.sin(2 * ps), torch.cos(th) * (mu[0] - k0)])

    out = torch.empty((len(t), 3, P.shape[0]), dtype=torch.float64, device=P.device)
    for i in range(len(t)):
        if i:
            n = int((t[i] - t[i - 1]) / body.step + 1)
            h = (t[i] - t[i - 1]) / n
            for _ in range(n):
                k1 = f(y)
                k2 = f(y + 0.5 * h * k1)
                k3 = f(y + 0.5 * h * k2)
                k4 = f(y + h * k3)
                y = y + h / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)
        out[i] = y[-3:]
    return out


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _frame(body, q, ang):
    """Body axes a, b, c in inertial coordinates for Euler angles ang [.., 3, n]."""
    th, ph = q["theta_M"], q["phi_M"]
    m = [torch.sin(th) * torch.cos(ph), torch.sin(th) * torch.sin(ph), torch.cos(th)]
    r = torch.sqrt(m[2] ** 2 + m[0] ** 2)
    x = [m[2] / r, torch.zeros_like(r), -m[0] / r]
    y = _cross(m, x)
    phi, theta, psi = ang[..., 0, :], ang[..., 1, :], ang[..., 2, :]
    node = [xx * torch.cos(phi) + yy * torch.sin(phi) for xx, yy in zip(x, y)]
    p = _cross(node, m)
    a = [mm * torch.cos(theta) + pp * torch.sin(theta) for mm, pp in zip(m, p)]
    w = _cross(a, node)
    b = [nn * torch.cos(psi) + ww * torch.sin(psi) for nn, ww in zip(node, w)]
    return a, b, _cross(a, b)


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _magnitudes(body, P, t, e, s, device):
    """Model magnitudes [len(t), n] in FP64 (Lommel-Seeliger ellipsoid or the two-tone ball)."""
    P = torch.as_tensor(P, dtype=torch.float64, device=device)
    if P.shape[0] == 1:
        ang = torch.as_tensor(_angles_one(body, P[0].cpu().numpy(), t), device=device)[:, :, None]
    else:
        ang = _angles_many(body, P, t)
    q = {k: P[:, i] for i, k in enumerate(body.names)}
    if body.flags & api.INTERP:
        m = body.eph_t
        r = np.stack([(t - m[1]) * (t - m[2]) / (m[0] - m[1]) / (m[0] - m[2]),
                      (t - m[0]) * (t - m[2]) / (m[1] - m[0]) / (m[1] - m[2]),
                      (t - m[0]) * (t - m[1]) / (m[2] - m[0]) / (m[2] - m[1])], 1)
        e, s = r @ body.eph_e.T, r @ body.eph_s.T
        e, s = e / np.linalg.norm(e, axis=1, keepdims=True), s / np.linalg.norm(s, axis=1, keepdims=True)
    out = torch.empty((len(t), P.shape[0]), dtype=torch.float64, device=device)
    for i0 in range(0, len(t), 64):  # a slice of observations at a time bounds the memory
        sl = slice(i0, min(len(t), i0 + 64))
        a, b, c = _frame(body, q, ang[sl])
        ev = [torch.as_tensor(e[sl, k], device=device)[:, None] for k in range(3)]
        sv = [torch.as_tensor(s[sl, k], device=device)[:, None] for k in range(3)]
        if body.flags & api.BW_BALL:
            n = [bb * torch.cos(q["phi_R"]) + cc * torch.sin(q["phi_R"]) for bb, cc in zip(b, c)]
            p = _cross(n, a)
            a = [aa * torch.cos(q["theta_R"]) + pp * torch.sin(q["theta_R"]) for aa, pp in zip(a, p)]
            z = _dot(a, ev)
            out[sl] = -2.5 * torch.log10(0.5 * (q["kappa"] * (1 + z) + 0.5 * (1 - z)))
            continue
        bb, cc = (q["b"], q["c"]) if body.flags & api.BC else (q["b_tumb"], q["c_tumb"])
        S, E = [_dot(b, sv) / bb, _dot(c, sv) / cc, _dot(a, sv)], [_dot(b, ev) / bb, _dot(c, ev) / cc, _dot(a, ev)]
        ns, ne = torch.sqrt(_dot(S, S)), torch.sqrt(_dot(E, E))
        ca = _dot(S, E) / (ns * ne)
        sa = torch.sqrt(1 - ca * ca)
        al = torch.atan2(sa, ca)
        sc = torch.sqrt(ns * ns + ne * ne + 2 * ns * ne * ca)
        cl, sl_ = (ns + ne * ca) / sc, ne * sa / sc
        la = torch.atan2(sl_, cl)
        out[sl] = -2.5 * torch.log10(bb * cc * ns * ne / sc * (torch.cos(la - al) + cl + sl_ * torch.sin(la - al) * torch.log(
            1 / torch.tan(0.5 * la) / torch.tan(0.5 * (al - la)))))
    return out


# ---------------------------------------------------------------- preparation

def _vectors(case, body, rng):
    return body.wide(rng, case["n"]) if case["vectors"] == "wide" else body.near(rng, case["n"])


def _body(case, rng):
    return Body(rng, case["flags"], case["points"], case["filters"], case["days"], case["step"], case.get("minima", 0))


def _batch_bodies(case, rng):
    """The three variants in turn, 50 to 500 points, 1 to 4 filters, 3 to 8 days."""
    return [Body(rng, ("TORQUE,ACC", "BC,ACC", "BW_BALL,ACC")[i % 3], round(50 * 10 ** (i * 7 % 24 / 23)), 1 + i * 5 % 4,
                 3 + i * 11 % 6, case["step"]) for i in range(case["objects"])]


def _grid(body, case):
    t = np.linspace(0.0, body.t[-1], case["points"])
    e, s = body._tracks(t)
    return t, e / np.linalg.norm(e, axis=1, keepdims=True), s / np.linalg.norm(s, axis=1, keepdims=True)


def _curve(case, rng):
    """A light curve of two frequencies and a slow beat, as a tumbler's, on an even grid."""
    t = np.linspace(0.0, float(case["days"]), case["points"])
    f1, f2 = rng.uniform(2.5, 4.0), rng.uniform(7.0, 11.0)
    return t, (0.6 * np.sin(2 * np.pi * 2 * f1 * t + rng.uniform(0, 6)) + 0.35 * np.sin(2 * np.pi * f2 * t + rng.uniform(0, 6))
               + 0.2 * np.sin(2 * np.pi * (2 * f1 + f2) * t) + 0.1 * np.sin(2 * np.pi * 0.13 * t))


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    if kind == "eval":
        body = _body(case, rng)
        obs = body.light_curve(rng)
        n, n_f = case["n"], case["filters"]
        return dict(case=case, engine=api.Engine(body.model, obs), params=_vectors(case, body, rng),
                    chi2=np.zeros(n), dv=np.zeros((n, n_f)))
    if kind == "fit":
        body = _body(case, rng)
        return dict(case=case, engine=api.Engine(body.model, body.light_curve(rng)), start=body.truth,
                    seed=int(rng.integers(1, 1 << 31)))
    if kind == "batch":
        bodies = _batch_bodies(case, rng)
        return dict(case=case, objects=[(b.model, b.light_curve(rng), b.truth) for b in bodies],
                    seed=int(rng.integers(1, 1 << 31)))
    if kind == "curve":
        body = Body(rng, case["flags"], 300, 1, case["days"], case["step"])
        return dict(case=case, engine=api.Engine(body.model, body.light_curve(rng)), params=body.truth, grid=_grid(body, case))
    if kind == "periodogram":
        return dict(case=case, curve=_curve(case, rng))
    return dict(case=case, geo=_geometry(case, rng),
                rgb=np.zeros((case["frames"], case["pixels"], case["pixels"], 3), np.uint8))


def _geometry(case, rng):
    """The frames' geometry (ast_model_geometry's rows) of consecutive snapshots of one body."""
    body = Body(rng, "TORQUE,ACC", 60, 1, 4, 1e-2)
    t = np.linspace(0.0, 0.01 * case["frames"], max(2, case["frames"]))
    e, s = body._tracks(t)
    e, s = e / np.linalg.norm(e, axis=1, keepdims=True), s / np.linalg.norm(s, axis=1, keepdims=True)
    P = torch.as_tensor(body.truth[None])
    q = {k: P[:, i] for i, k in enumerate(body.names)}
    ang = torch.as_tensor(_angles_one(body, body.truth, t))[:, :, None]
    a, b, c = ([x[:, 0].numpy() for x in v] for v in _frame(body, q, ang))
    geo = np.zeros((len(t), capi.AST_GEO))
    geo[:, 0], geo[:, 1] = float(q["b_tumb"]), float(q["c_tumb"])
    geo[:, 2:5] = e
    for k, (axis) in enumerate((b, c, a)):
        axis = np.stack(axis, 1)
        geo[:, 5 + k], geo[:, 8 + k] = (axis * e).sum(1), (axis * s).sum(1)
        geo[:, 11 + 3 * k:14 + 3 * k] = axis
    return np.ascontiguousarray(geo[: case["frames"]])


# ---------------------------------------------------------------- one pass

def _own(case, x):
    """The value in its own type: CHI_FLOAT is float without ACC (no value changes)."""
    return x if "ACC" in case["flags"] else x.astype(np.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "eval":
        chi2, dv = state["engine"].eval(state["params"], PREC[case["prec"]], state["chi2"], state["dv"])
        return {"chi2": _own(case, chi2), "dv": _own(case, dv)}
    if kind == "fit":
        kw = dict(reopt=True, params0=state["start"], fp64_result=True) if case["reopt"] else {}
        r = state["engine"].fit(n_chains=case["chains"], group_size=case["group"], seed=state["seed"],
                                precision=PREC[case["prec"]], evals_cap=case["evals"], **kw)
        return {"best_f": r.best_f, "best_params": r.best_params, "best_dv": r.best_dv, "n_evals": r.n_evals}
    if kind == "batch":
        out = []
        with api.Batch(precision=api.PREC_MIXED, acc=True) as b:
            for model, obs, truth in state["objects"]:
                b.add(model, obs, n_chains=case["chains"], group_size=64, seed=state["seed"], evals_cap=case["evals"],
                      reopt=True, params0=truth, fp64_result=True)
            b.run()
            for i in range(len(state["objects"])):
                r = b.result(i)
                out.append(np.concatenate([r.best_f[:, None], r.best_params, r.best_dv], 1))
        return out
    if kind == "curve":
        return state["engine"].model_curve_at(state["params"], *state["grid"])
    if kind == "periodogram":
        r = api.minima(*state["curve"])
        return {"counts": r.counts, "cl_fr": r.cl_fr, "cl_H": r.cl_H, "n_minima": r.n_minima, "n_clusters": r.n_clusters}
    rgb, pixels = state["rgb"], case["pixels"]
    lib = capi.load()
    capi.check(lib.ast_render_frames(-1, capi.dptr(state["geo"]), case["frames"], pixels,
                                     rgb.ctypes.data_as(ctypes.POINTER(ctypes.c_uint8)), None), "ast_render_frames")
    return rgb


# ---------------------------------------------------------------- what a pass cannot do without

def _eval_work(points, days, step, filters):
    """(flops, bytes read) of one chi^2: the reference's operation count, the light curve."""
    steps = points + (days - 1) * 0.75 / step + max(0.0, days * 0.25 / step - points)
    return 152 * steps + 156 * points + 6 * filters + 50, 72 * points


def work(case):
    kind = case["kind"]
    if kind in ("eval", "fit"):
        f, by = _eval_work(case["points"], case["days"], case["step"], case["filters"])
        n = case["n"] if kind == "eval" else case["chains"] * case["evals"]
        io = 8 * (11 + 1 + case["filters"]) * (case["n"] if kind == "eval" else case["chains"] // case["group"])
        return {"bytes": by + io, "flops": f * n}
    if kind == "batch":
        f, by = _eval_work(160, 6, case["step"], 2)
        return {"bytes": by * case["objects"], "flops": f * case["objects"] * case["chains"] * case["evals"]}
    if kind == "curve":
        return {"bytes": 64 * case["points"], "flops": 308 * case["points"]}
    if kind == "periodogram":
        # At least one interval value per grid distance, tested at 10 000 frequencies.
        return {"bytes": 16 * case["points"] + 4e4, "flops": 4e4 * case["points"]}
    return {"bytes": 3 * case["frames"] * case["pixels"] ** 2 + 160 * case["frames"], "flops": 60 * case["frames"] * case["pixels"] ** 2}


# ---------------------------------------------------------------- the same in plain FP64

def exact(case, seed):
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "eval":
        body = _body(case, rng)
        obs = body.light_curve(rng)
        P = _vectors(case, body, rng)
        mag = _magnitudes(body, P, body.t, body.e, body.s, device)
        r = torch.as_tensor(obs.v, device=device).double()[:, None] - mag
        w = torch.as_tensor(obs.w, device=device).double()[:, None]
        chi2, dv = 0, []
        for m in range(case["filters"]):
            k = torch.as_tensor(obs.filt == m, device=device)
            sy, sy2, sw = (w[k] * r[k]).sum(0), (w[k] * r[k] ** 2).sum(0), w[k].sum()
            chi2 = chi2 + sy2 - sy * sy / sw
            dv.append(sy / sw)
        chi2 = chi2 / (obs.n_data - body.model.n_params - case["filters"])
        # The reward for observed minima is single-precision arithmetic by definition.
        return {"chi2": None if body.flags & api.NUDGE else chi2.cpu().numpy(), "dv": torch.stack(dv, 1).cpu().numpy()}
    if kind == "curve":
        body = Body(rng, case["flags"], 300, 1, case["days"], case["step"])
        return _magnitudes(body, body.truth[None], *_grid(body, case), "cpu")[:, 0].numpy()
    if kind == "periodogram":
        return _periodogram(*_curve(case, rng))
    return None


def _periodogram(t, v):
    i = np.arange(1, len(t) - 1)
    tm = t[i[(v[i] > v[i - 1]) & (v[i] >= v[i + 1])]]
    d = (tm[None] - tm[:, None])[np.triu_indices(len(tm), 1)]
    d, mult = np.unique(d, return_counts=True)
    fr = 24 / 80 + np.arange(10000) / 9999.0 * (24 - 24 / 80)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    d, mult = torch.as_tensor(d, device=device), torch.as_tensor(mult, device=device)
    one = torch.as_tensor(1 / fr, device=device)
    count = torch.zeros(10000, dtype=torch.int64, device=device)
    for f0 in range(0, 10000, 200):
        x = d[None] / one[f0:f0 + 200, None]
        count[f0:f0 + 200] = (((x - torch.floor(x + 0.5)).abs() < 0.1) * mult[None]).sum(1)
    h = count.cpu().numpy().astype(np.float64)
    h = (h - h.mean()) / math.sqrt(((h - h.mean()) ** 2).sum() / 9999)
    cl_fr, cl_h, marked = np.full(5, -1.0), np.zeros(5), np.zeros(10000, bool)
    for k in range(5):
        free = np.where(~marked)[0]
        if not len(free) or h[free].max() < 3:
            break
        top = int(free[np.argmax(h[free])])
        cl_fr[k], cl_h[k] = fr[top], h[top]
        for step in (1, -1):
            j = top if step == 1 else top - 1
            while 0 <= j < 10000 and h[j] > 3:
                marked[j] = True
                j += step
    return {"counts": None, "cl_fr": cl_fr, "cl_H": cl_h, "n_minima": None, "n_clusters": None}
