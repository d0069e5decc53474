"""The work that users of this framework have it do, as cases that can be timed and compared.

Every case starts each pass from the same state (positions, velocities, accelerations, frame position and
increment are set through the setters), so a pass is the same work however often it is repeated.  Disorder
is the library's usual one: yield distances Weibull(2, 1) + 1e-5 from pcg32, m = 1, eta = 0.1 (0.2 on the
grid), mu = 1, k_interactions = 1, k_frame = 1 / N, dt = 0.1.

`exact` follows the same protocols with plain torch operations in 64 bits: the pcg32 stream, the yield
positions, the velocity-Verlet step with its three velocity updates, the residual stop test, the
event-driven step and, for the adjoint, torch's own autograd through the unrolled steps.
"""

import math

import numpy as np
import torch

from frictionqpotspringblock_gb300 import Line1d, Line2d, Particles
from frictionqpotspringblock_gb300 import _capi as capi
from frictionqpotspringblock_gb300 import autograd as fqad
from frictionqpotspringblock_gb300 import batch as fqbatch

DISORDER = dict(distribution="weibull", parameters=[2.0, 1.0, 1e-5])
DT = 0.1
EPS = 1e-5
#: from this many particles on, a program keeps the state on the GPU and hands it over there
ON_DEVICE = 1 << 16


def listed():
    return [
        # a small chain advanced one time step per call, as scripts that look at every step do
        {"name": "steps_n100", "kind": "single", "n": 100, "calls": 20, "potential": "cuspy", "ring": True},
        # the quasistatic protocol of the examples on a small chain: event, kick, minimise
        {"name": "quasistatic_n1024", "kind": "quasistatic", "n": 1024, "cycles": 2, "activity": False},
        # the same near the largest chain that one cluster holds, an odd size, with plastic activity counted
        {"name": "quasistatic_n10007", "kind": "quasistatic", "n": 10007, "cycles": 1, "activity": True},
        # an ordinary chain under a steadily moving frame
        {"name": "flow_n65536", "kind": "flow", "n": 65536, "steps": 1000, "potential": "cuspy", "ring": True},
        # the throughput size, state resident on the GPU
        {"name": "flow_n4194304", "kind": "flow", "n": 4194304, "steps": 100, "potential": "cuspy", "ring": True},
        # a large odd chain relaxed after a jump of the frame
        {"name": "minimise_n1048583", "kind": "jump", "n": 1048583, "jump": 0.5},
        # the large grid under a steadily moving frame
        {"name": "grid_flow_2048x2048", "kind": "grid_flow", "rows": 2048, "cols": 2048, "steps": 60},
        # an ordinary ragged grid through one quasistatic cycle
        {"name": "grid_quasistatic_301x257", "kind": "grid_quasistatic", "rows": 301, "cols": 257, "cycles": 1},
        # an ensemble of uneven realisations: built, then one quasistatic cycle of all of them
        {"name": "ensemble_96", "kind": "ensemble", "count": 96, "lo": 256, "hi": 32768, "cycles": 1},
        # gradients of a trajectory loss (smooth potential): forward and backward
        {"name": "adjoint_n65536", "kind": "adjoint", "n": 65536, "steps": 200, "every": 50, "potential": "smooth"},
        # thermal forcing at the size of the reference's example
        {"name": "thermal_n1000", "kind": "thermal", "n": 1000, "steps": 1000, "period": 100},
        # a new sample: construction of its disorder, then a drive far beyond the first yield positions
        {"name": "disorder_n16384", "kind": "disorder", "n": 16384, "nchunk": 1000, "reach": 2000.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "quasistatic", "flow", "flow", "jump", "grid_flow", "grid_quasistatic", "ensemble",
                       "adjoint", "thermal", "disorder"])
    if kind == "single":
        return {"kind": kind, "n": _log_int(rng, 50, 20000), "calls": rng.randint(5, 20),
                "potential": rng.choice(["cuspy", "semismooth", "smooth"]), "ring": rng.random() < 0.7}
    if kind == "quasistatic":
        return {"kind": kind, "n": _log_int(rng, 64, 100000), "cycles": 1, "activity": rng.random() < 0.5}
    if kind == "flow":
        n = _log_int(rng, 1000, 4194304)
        return {"kind": kind, "n": n, "steps": rng.randint(60, 100) if n > 300000 else rng.randint(200, 1000),
                "potential": rng.choice(["cuspy", "cuspy", "semismooth"]), "ring": rng.random() < 0.8}
    if kind == "jump":
        return {"kind": kind, "n": _log_int(rng, 20000, 1048583), "jump": round(rng.uniform(0.2, 0.5), 3)}
    if kind == "grid_flow":
        return {"kind": kind, "rows": _log_int(rng, 40, 2048), "cols": _log_int(rng, 40, 2048),
                "steps": rng.randint(30, 60)}
    if kind == "grid_quasistatic":
        return {"kind": kind, "rows": _log_int(rng, 20, 400), "cols": _log_int(rng, 20, 400), "cycles": 1}
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(10, 96), "lo": 256, "hi": _log_int(rng, 1000, 32768), "cycles": 1}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_int(rng, 500, 65536), "steps": rng.randint(60, 200),
                "every": rng.randint(20, 60), "potential": rng.choice(["smooth", "semismooth"])}
    if kind == "thermal":
        return {"kind": kind, "n": _log_int(rng, 100, 200000), "steps": rng.randint(200, 600),
                "period": rng.randint(20, 200)}
    return {"kind": kind, "n": _log_int(rng, 200, 16384), "nchunk": rng.randint(100, 1000),
            "reach": round(rng.uniform(200.0, 2000.0), 1)}


# ------------------------------------------------------------------------------------------ systems


def _shape(case):
    return [case["rows"], case["cols"]] if "rows" in case else [case["n"]]


def _size(case):
    return math.prod(_shape(case))


def _nchunk(case):
    """Yield positions kept per particle: the examples' thousands for small systems, fewer for large ones."""
    if case["kind"] == "disorder":
        return case["nchunk"]
    return 1000 if _size(case) <= 20000 else 200


def _par(case, seed):
    n = _size(case)
    grid = "rows" in case
    return dict(eta=0.2 if grid else 0.1, mu=1.0, k_frame=1.0 / n, dt=DT, shape=_shape(case), seed=seed * 10_000_019 % (1 << 40),
                offset=-100.0, nchunk=_nchunk(case), **DISORDER)


def _system(case, seed):
    p = _par(case, seed)
    kind = case["kind"]
    if kind in ("grid_flow", "grid_quasistatic"):
        return Line2d.System_Cuspy_Laplace(m=1.0, k_interactions=1.0, **p)
    if kind == "thermal":
        init = np.random.default_rng(seed).integers(0, case["period"], case["n"])
        return Line1d.System_Cuspy_Laplace_RandomForcing(
            m=1.0, k_interactions=1.0, mean=0.0, stddev=0.05, seed_forcing=seed, dinc_init=init,
            dinc=np.full(case["n"], case["period"]), **p)
    potential = case.get("potential", "cuspy")
    if potential == "semismooth":
        p["kappa"] = 1.0
    if case.get("ring", True):
        cls = {"cuspy": Line1d.System_Cuspy_Laplace, "semismooth": Line1d.System_SemiSmooth_Laplace,
               "smooth": Line1d.System_Smooth_Laplace}[potential]
        return cls(m=1.0, k_interactions=1.0, **p)
    cls = {"cuspy": Particles.System_Cuspy, "semismooth": Particles.System_SemiSmooth,
           "smooth": Particles.System_Smooth}[potential]
    return cls(m=1.0, **p)


def _initial(case, seed):
    """Initial positions: N(0, 0.1^2), as the throughput workload starts; a pass then moves particles across wells."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return 0.1 * torch.randn(_size(case), dtype=torch.float64, device="cuda", generator=g)


def _sched(case):
    t = np.arange(case["steps"])
    return 1e-3 * t + 0.05 * np.sin(2 * np.pi * t / 500)


def prepare(case, seed):
    st = {"case": case}
    if case["kind"] == "ensemble":
        st["sizes"] = fqbatch.log_uniform_sizes(case["count"], case["lo"], case["hi"], seed=3)
        st["seeds"] = 1000 * (seed % 1_000_003) + np.arange(case["count"])
        return st
    u0 = _initial(case, seed)
    if case["kind"] == "disorder":
        st["u"] = u0.cpu().numpy()
        st["par"] = dict(_par(case, seed), m=1.0, k_interactions=1.0)
        return st
    s = st["system"] = _system(case, seed)
    if case["kind"] == "adjoint":
        st["u"], st["v"] = u0, torch.zeros_like(u0)
        st["schedule"] = torch.from_numpy(_sched(case))
        st["params"] = torch.tensor([1.0, 1.0, 0.1], dtype=torch.float64)
        return st
    if s.size >= ON_DEVICE:
        st["u"] = u0
        st["zero"] = torch.zeros_like(u0)
    else:
        st["u"] = u0.cpu().numpy().reshape(s.shape)
        st["zero"] = np.zeros(s.shape)
    if case["kind"] == "thermal":
        st["forcing"] = (s.external.state, s.external.f_thermal, s.external.next)
    return st


def _reset(st):
    s = st["system"]
    s.inc = 0
    s.u_frame = 0.0
    if s.size >= ON_DEVICE:
        s.set_field_device(capi.FIELD_U, st["u"].data_ptr())
        s.set_field_device(capi.FIELD_V, st["zero"].data_ptr())
        s.set_field_device(capi.FIELD_A, st["zero"].data_ptr())
    else:
        s.u, s.v, s.a = st["u"], st["zero"], st["zero"]
    if "forcing" in st:
        s.external.state, s.external.f_thermal, s.external.next = st["forcing"]
    return s


def _state(st):
    s = st["system"]
    if s.size < ON_DEVICE:
        return {"u": s.u, "v": s.v, "a": s.a, "u_frame": s.u_frame, "i": s.chunk.index_at_align}
    out = {}
    for name, field in (("u", capi.FIELD_U), ("v", capi.FIELD_V), ("a", capi.FIELD_A)):
        out[name] = torch.empty(s.shape, dtype=torch.float64, device="cuda")
        s.get_field_device(field, out[name].data_ptr())
    out["u_frame"] = s.u_frame
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ensemble":
        n = st["sizes"]
        b = fqbatch.Line1d_System_Cuspy_Laplace(n, st["seeds"], 1.0 / n, m=1.0, eta=0.1, mu=1.0, k_interactions=1.0,
                                                dt=DT, offset=-100.0, nchunk=1000, window=64, **DISORDER)
        out = b.quasistatic(case["cycles"], EPS)
        out["u"] = np.concatenate([b.field(j) for j in range(len(n))])
        out["i"] = np.concatenate([b.index_at_align(j) for j in range(len(n))])
        return out
    if kind == "disorder":
        s = Line1d.System_Cuspy_Laplace(**st["par"])
        s.u = st["u"]
        near = s.chunk.index_at_align
        s.u = st["u"] + case["reach"]
        return {"near": near, "i": s.chunk.index_at_align, "left": s.chunk.left_of_align,
                "right": s.chunk.right_of_align, "residual": s.residual}
    if kind == "adjoint":
        u, v = st["u"].requires_grad_(), st["v"].requires_grad_()
        sched, params = st["schedule"].requires_grad_(), st["params"].requires_grad_()
        loss = fqad.trajectory_loss(st["system"], u, v, sched, params, K=case["every"], last=case["steps"] // 4)
        return [loss.detach(), *torch.autograd.grad(loss, (u, v, sched, params))]
    s = _reset(st)
    if kind == "single":
        for _ in range(case["calls"]):
            s.timeStep()
    elif kind in ("flow", "grid_flow", "thermal"):
        s.flowSteps(case["steps"], 1e-3)
    elif kind == "jump":
        s.u_frame = case["jump"]
        s.minimise()
    else:
        for _ in range(case["cycles"]):
            s.eventDrivenStep(EPS, False)
            s.eventDrivenStep(EPS, True)
            s.minimise(time_activity=bool(case.get("activity", kind == "grid_quasistatic")))
    return _state(st)


def work(case):
    """State and current wells read once and the state written once; 24 additions and multiplications per
    particle and time step (some hundreds per drawn yield distance).  Relaxations: their usual number of steps."""
    kind = case["kind"]
    if kind == "ensemble":
        n = case["count"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": 64.0 * n, "flops": 24.0 * n * 3900 * case["cycles"]}
    n = float(_size(case))
    if kind == "disorder":
        draws = n * max(case["nchunk"], (case["reach"] + 100.0) / 0.886)
        return {"bytes": 8.0 * n * case["nchunk"] + 40.0 * n, "flops": 50.0 * draws}
    if kind == "adjoint":
        return {"bytes": 64.0 * n, "flops": n * case["steps"] * (44.0 + 44.0 + 60.0)}
    steps = {"single": case.get("calls"), "flow": case.get("steps"), "grid_flow": case.get("steps"),
             "thermal": case.get("steps"), "jump": 1900}.get(kind)
    if steps is None:
        steps = 3000 * case["cycles"]
    return {"bytes": 64.0 * n, "flops": (26.0 if "rows" in case else 24.0) * n * steps}


# ------------------------------------------------------------------------------------------ exact values

MULT = 0x5851F42D4C957F2D


def _lsr(x, k):
    """Logical right shift of 64-bit patterns held as int64."""
    return (x >> k) & ((1 << (64 - k)) - 1)


def _pcg_out(old):
    xs = _lsr(_lsr(old, 18) ^ old, 27) & 0xFFFFFFFF
    rot = _lsr(old, 59)
    return ((xs >> rot) | (xs << ((32 - rot) & 31))) & 0xFFFFFFFF


def _yields(n, seed, count, offset=-100.0):
    """The first `count` yield positions of each of n particles, [n, count]."""
    st = (torch.arange(n, dtype=torch.int64, device="cuda") + seed + 1) * MULT + 1
    y = torch.empty(n, count, dtype=torch.float64, device="cuda")
    c = None
    for k in range(count):
        r = _pcg_out(st).to(torch.float64) * 2.0 ** -32
        d = torch.sqrt(-torch.log(1.0 - r)) + 1e-5
        c = d if c is None else c + d
        y[:, k] = c + offset
        st = st * MULT + 1
    return y


class _Plain:
    """The model in plain torch operations."""

    def __init__(self, case, seed, count):
        p = _par(case, seed)
        self.case, self.shape, self.n = case, _shape(case), _size(case)
        self.y = _yields(self.n, p["seed"], count)
        self.potential, self.ring = case.get("potential", "cuspy"), case.get("ring", True)
        self.mu, self.k, self.eta, self.kf, self.kappa = 1.0, 1.0, p["eta"], p["k_frame"], 1.0
        self.u = _initial(case, seed)
        self.v = torch.zeros_like(self.u)
        self.a = torch.zeros_like(self.u)
        self.uf = 0.0
        self.f = self.ff = None
        self.thermal = None

    def wells(self, u):
        i = torch.searchsorted(self.y, u.detach().unsqueeze(1), right=True) - 1
        if bool((i < 0).any()) or bool((i > self.y.shape[1] - 2).any()):
            raise ValueError("more yield positions are needed")
        return i.squeeze(1), self.y.gather(1, i).squeeze(1), self.y.gather(1, i + 1).squeeze(1)

    def f_potential(self, u):
        _, lo, hi = self.wells(u)
        if self.potential == "cuspy":
            return self.mu * (0.5 * (lo + hi) - u)
        if self.potential == "smooth":
            c, w = 0.5 * (lo + hi), 0.5 * (hi - lo)
            return (-self.mu * w / math.pi) * torch.sin(math.pi * (u - c) / w)
        c = 0.5 * (lo + hi)
        ul = (self.mu * c + self.kappa * lo) / (self.mu + self.kappa)
        ur = (self.mu * c + self.kappa * hi) / (self.mu + self.kappa)
        return torch.where(u < ul, self.kappa * (u - lo), torch.where(u <= ur, self.mu * (c - u), self.kappa * (u - hi)))

    def f_interactions(self, u):
        if len(self.shape) == 2:
            g = u.reshape(self.shape)
            f = g.roll(1, 0) + g.roll(-1, 0) + g.roll(1, 1) + g.roll(-1, 1) - 4.0 * g
            return self.k * f.reshape(-1)
        if not self.ring:
            return torch.zeros_like(u)
        return self.k * (u.roll(1) - 2.0 * u + u.roll(-1))

    def step(self):
        dt = DT
        self.u = self.u + dt * self.v + (0.5 * dt * dt) * self.a
        self.ff = self.kf * (self.uf - self.u)
        s = self.ff + self.f_potential(self.u) + self.f_interactions(self.u)

        def force(v):
            f = s - self.eta * v
            return f if self.thermal is None else f + self.thermal

        v = self.v + dt * self.a
        f = force(v)
        for _ in range(2):
            v = self.v + (0.5 * dt) * (self.a + f)
            f = force(v)
        self.v, self.a, self.f = v, f, f

    def minimise(self, tol=1e-5, window=10):
        last = [math.inf] * window
        for _ in range(200000):
            self.step()
            norms = torch.stack([self.f.square().sum(), self.ff.square().sum()]).sqrt().tolist()
            last = last[1:] + [norms[0] / norms[1] if norms[1] != 0.0 else norms[0]]
            down = all(b <= a for a, b in zip(last, last[1:]))
            if (down and max(last) < tol) or max(last) < tol * tol:
                break
        self.v, self.a = torch.zeros_like(self.u), torch.zeros_like(self.u)

    def advance(self, du):
        self.u = self.u + du
        self.uf += du * (self.kf + self.mu) / self.kf

    def event(self):
        _, _, hi = self.wells(self.u)
        du = float((hi - self.u).min())
        if du >= 0.5 * EPS:
            self.advance(du - 0.5 * EPS)
        self.advance(EPS)

    def state(self):
        out = {"u": self.u.reshape(self.shape), "v": self.v.reshape(self.shape), "a": self.a.reshape(self.shape),
               "u_frame": self.uf}
        if self.n < ON_DEVICE:
            out["i"] = self.wells(self.u)[0].reshape(self.shape)
        return out


def _pcg_scalar(seed):
    mask, inc = (1 << 64) - 1, (0xDA3E39CB94B95BDB << 1 | 1) & ((1 << 64) - 1)
    s = ((inc + seed) * MULT + inc) & mask
    while True:
        xs, rot = ((s >> 18 ^ s) >> 27) & 0xFFFFFFFF, s >> 59
        yield ((xs >> rot) | (xs << (-rot & 31))) & 0xFFFFFFFF
        s = (s * MULT + inc) & mask


def _erfinv(y):
    """torch's erfinv with one Newton step on the smaller of erf and erfc."""
    x = torch.erfinv(y)
    a, z = y.abs(), x.abs()
    r = torch.where(a > 0.5, (1.0 - a) - torch.erfc(z), torch.erf(z) - a)
    z = z - r * (0.5 * math.sqrt(math.pi)) * torch.exp(z * z)
    return torch.where(y < 0, -z, z)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return None  # thousands of steps of every realisation, one after another: minutes
    if kind == "disorder":
        p = _par(case, seed)
        u0 = _initial(case, seed)
        y = _yields(case["n"], p["seed"], int((case["reach"] + 101.0) / 0.886 * 1.1) + 200)
        u = u0 + case["reach"]
        near = torch.searchsorted(y, u0.unsqueeze(1), right=True).squeeze(1) - 1
        i = torch.searchsorted(y, u.unsqueeze(1), right=True) - 1
        lo, hi = y.gather(1, i).squeeze(1), y.gather(1, i + 1).squeeze(1)
        ff = p["k_frame"] * (0.0 - u)
        f = ff + (0.5 * (lo + hi) - u) + (u.roll(1) - 2.0 * u + u.roll(-1))
        return {"near": near, "i": i.squeeze(1), "left": lo, "right": hi, "residual": float(f.norm() / ff.norm())}
    m = _Plain(case, seed, 200)
    if kind == "adjoint":
        u, v = m.u.requires_grad_(), m.v.requires_grad_()
        sched = torch.from_numpy(_sched(case)).cuda().requires_grad_()
        params = torch.tensor([1.0, 1.0, 0.1], dtype=torch.float64, device="cuda", requires_grad=True)
        m.mu, m.k, m.eta = params[0], params[1], params[2]
        m.u, m.v = u, v
        last, loss = case["steps"] // 4, 0.0
        for t in range(case["steps"]):
            m.uf = sched[t]
            m.step()
            if t >= case["steps"] - last:
                loss = loss + m.ff.mean() / last
        loss = loss + 0.5 * m.u.square().mean()
        g = torch.autograd.grad(loss, (u, v, sched, params))
        return [loss.detach(), g[0], g[1], g[2].cpu(), g[3].cpu()]
    with torch.no_grad():
        if kind == "single":
            for _ in range(case["calls"]):
                m.step()
        elif kind in ("flow", "grid_flow"):
            for _ in range(case["steps"]):
                m.uf += 1e-3 * DT
                m.step()
        elif kind == "thermal":
            nxt = np.random.default_rng(seed).integers(0, case["period"], case["n"])
            stream, th = _pcg_scalar(seed), np.zeros(case["n"])
            for inc in range(case["steps"] + 1):
                due = np.flatnonzero(inc >= nxt)
                if len(due):
                    r = torch.tensor([next(stream) for _ in due], dtype=torch.float64) * 2.0 ** -32
                    th[due] = (0.05 * math.sqrt(2.0)) * _erfinv(2.0 * r - 1.0).numpy()
                    nxt[due] += case["period"]
                m.thermal = torch.from_numpy(th).cuda()
                if inc:
                    m.uf += 1e-3 * DT
                    m.step()
        elif kind == "jump":
            m.uf = case["jump"]
            m.minimise()
        else:
            for _ in range(case["cycles"]):
                m.event()
                m.minimise()
    return m.state()
