"""The work that a user of this framework has it do, as cases that can be timed and compared.

Kinds of case (the ``kind`` of a case):

* ``step``: a running simulation advances by ``steps`` time steps and its state is read back on the
  device (every field and the neighbour counts), with the step's energies and time step on the host, as
  a driver loop does that prints them and keeps a snapshot.  Precision, equation of state, softening,
  neighbour number, equal or unequal masses, gravity (direct or tree) and graph replay are the options
  of a run.
* ``host``: the same step for a program that owns its state on the host (the reference driver's
  manner): fields in from pinned buffers, one step, fields out.
* ``forces``: the first force evaluation on a particle set that a program has just loaded or made
  (ranges only estimated): sort, tree, smoothing lengths, density, pressure, hydro, gravity.
* ``adjoint``: one step of a reverse sweep: the pre-step state set, the step replayed, the adjoints of
  the post-step state mapped to those of the pre-step state.
* ``rollout``: gradients of a loss through K steps by the torch binding (forward, checkpoints, reverse).
* ``gravity``: the stand-alone direct-sum operator on a caller's own buffers.

Particle sets: ``star`` is one n-polytrope with rotation and pulsation, ``pair`` two of them head on,
``sphere`` a cold uniform sphere.  Field values of the mixed form that carry its FP32 pair terms are
kept in float32, those that it computes in FP64 in float64.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from cudasph_b200 import ics
from cudasph_b200._capi import ADJ_FIELDS, ADJ_ID, FIELD_ID, FIELDS, STATS, check, lib
from cudasph_b200.simulation import Simulation, make_params

GAMMA = 5.0 / 3.0
MU = 0.62
OUT = tuple(f for f in FIELDS if f not in ("m", "mu"))
OUT64 = ("x", "y", "z", "range", "rho", "omega", "psi")  # FP64 in the mixed form, whatever gravity rounds
IN = ("x", "y", "z", "range", "vx", "vy", "vz", "m", "u", "mu")
TOLD = ("W", "T", "U", "E", "ngb_mean", "ngb_min", "ngb_max", "dt", "time")


def _case(name, kind, n, **kw):
    c = dict(name=name, kind=kind, n=n, model="star", poly=1.5, precision="fp64", eos="ideal", soft="plummer",
             eps=0.01, n_ngb=50.0, grav="direct", theta=0.5, masses="equal", steps=1, graph=False)
    c.update(kw)
    return c


def listed():
    return [
        # a small set, as in parameter studies and unit checks: ten steps between two looks at the state
        _case("step_2k_x10", "step", 2049, steps=10),
        # the same with the steps replayed from a graph, unequal masses, mixed precision
        _case("step_6k_graph_x10", "step", 6007, steps=10, graph=True, masses="unequal", precision="mixed",
              eos="gas_radiation", n_ngb=64.0),
        # the plain FP64 star of 16,384 particles
        _case("step_16k_fp64", "step", 16384),
        # the reference's own parameters and the size of its input: spline softening, 24 neighbours
        _case("step_60k_reference", "step", 60000, eos="gas_radiation", soft="spline", n_ngb=24.0),
        # FP64 star with gas and radiation, 262,144 particles
        _case("step_262k_fp64", "step", 262144, eos="gas_radiation", eps=0.005, n_ngb=64.0),
        # two stars head on, 1,048,576 particles, mixed precision: the headline run
        _case("step_1m_mixed", "step", 1048576, model="pair", precision="mixed", eos="gas_radiation", eps=0.002,
              n_ngb=64.0),
        # a large gravity-dominated collapse with the tree
        _case("step_2m_tree", "step", 2000003, model="sphere", precision="mixed", eps=0.001, grav="tree"),
        # a host-side driver's step, odd size
        _case("host_100k_mixed", "host", 100003, model="pair", precision="mixed", eos="gas_radiation", eps=0.002,
              n_ngb=64.0),
        # the first evaluation on a new particle set
        _case("forces_130k_new", "forces", 130001, eos="gas_radiation", eps=0.005, n_ngb=64.0),
        # one reverse step of an n = 3 star, 65,536 particles, mixed precision
        _case("adjoint_65k_mixed", "adjoint", 65536, poly=3.0, precision="mixed", eos="gas_radiation", n_ngb=64.0),
        # gradients through four steps by the torch binding, FP64
        _case("rollout_12k_fp64", "rollout", 12001, poly=3.0, eos="gas_radiation", n_ngb=64.0, steps=4),
        # direct sum over a caller's own sources of unequal mass
        _case("gravity_30k_mixed", "gravity", 30011, precision="mixed", masses="unequal"),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n | 1 if rng.random() < 0.5 else n

    kind = rng.choice(("step", "step", "step", "step", "step", "tree", "host", "forces", "adjoint", "rollout",
                       "gravity"))
    o = dict(precision=rng.choice(("fp64", "mixed")), eos=rng.choice(("ideal", "gas_radiation")),
             n_ngb=rng.choice((24.0, 50.0, 64.0)), eps=rng.choice((0.01, 0.005, 0.002)),
             masses=rng.choice(("equal", "equal", "unequal")), model=rng.choice(("star", "pair")),
             poly=rng.choice((1.5, 3.0)))
    top = 900000 if o["precision"] == "mixed" else 400000
    if kind == "step":
        if rng.random() < 0.25:
            o.update(soft="spline")
            top = 150000
        n = size(1500, top)
        o.update(steps=10 if n < 10000 else 1, graph=rng.random() < 0.25)
    elif kind == "tree":
        kind, n = "step", size(20000, 2000000)
        o.update(model=rng.choice(("pair", "sphere")), precision="mixed", grav="tree",
                 theta=rng.choice((0.3, 0.5, 0.7)))
    elif kind == "host":
        n = size(5000, top // 2)
    elif kind == "forces":
        n = size(5000, 300000)
    elif kind == "adjoint":
        n = size(3000, 150000)
    elif kind == "rollout":
        n = size(2000, 30000)
        o.update(steps=rng.choice((3, 4, 5)))
    else:
        n = size(1000, top)
        if rng.random() < 0.25:
            o.update(soft="spline")
            n = min(n, 150001)
    c = _case("", kind, n, **o)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------
# particle sets, made on the device from the seed
# ------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _polytrope_profile(poly):
    xi, th, dth = ics.lane_emden(poly, dxi=1e-3)
    mf = -(xi * xi * dth)
    w1 = mf[-1]
    mf = mf / mf[-1]
    mf[0] = 0.0
    a = 1.0 / xi[-1]
    rho_c = 1.0 / (4.0 * math.pi * a ** 3 * w1)
    k = 4.0 * math.pi * a * a * rho_c ** (1.0 - 1.0 / poly) / (poly + 1.0)
    return tuple(torch.tensor(t, device="cuda") for t in (xi * a, th, mf)) + (rho_c, k)


def _interp(x, xp, fp):
    i = torch.searchsorted(xp, x).clamp(1, xp.numel() - 1)
    x0, x1 = xp[i - 1], xp[i]
    t = ((x - x0) / (x1 - x0)).clamp(0.0, 1.0)
    return fp[i - 1] + t * (fp[i] - fp[i - 1])


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _star(n, poly, n_ngb, g):
    """An n-polytrope of mass and radius 1 (G = 1): a rotated cubic lattice stretched radially."""
    r, th, mf, rho_c, kk = _polytrope_profile(poly)
    k = int(math.ceil((n * 6.0 / math.pi) ** (1.0 / 3.0) / 2.0)) + 2
    ax = torch.arange(-k, k + 1, device="cuda", dtype=torch.float64)
    p = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    p = p + (_uniform(g, 3) - 0.5)
    a = _uniform(g, 3) * (2.0 * math.pi)
    c, s = torch.cos(a).tolist(), torch.sin(a).tolist()
    rot = torch.eye(3, dtype=torch.float64)
    for d in range(3):
        m = torch.eye(3, dtype=torch.float64)
        i, j = (d + 1) % 3, (d + 2) % 3
        m[i, i], m[i, j], m[j, i], m[j, j] = c[d], -s[d], s[d], c[d]
        rot = rot @ m
    p = p @ rot.to("cuda")
    rad = (p * p).sum(1).sqrt()
    order = torch.argsort(rad, stable=True)[:n]
    p, rad = p[order], rad[order]
    rn = _interp((torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n, mf, r)
    rn = (rn + (_uniform(g, n) - 0.5) * (0.02 * n ** (-1.0 / 3.0))).clamp(0.0, 1.0)
    rho = (rho_c * _interp(rn, r, th).clamp(min=0.0) ** poly).clamp(min=1e-4 * rho_c)
    q = {}
    q["pos"] = p / rad.clamp(min=1e-300)[:, None] * rn[:, None]
    q["vel"] = torch.stack((-0.2 * q["pos"][:, 1], 0.2 * q["pos"][:, 0], torch.zeros_like(rn)), 1) + 0.05 * q["pos"]
    q["u"] = kk * rho ** (1.0 / poly) / (GAMMA - 1.0)
    q["rho"] = rho
    return q


def _sphere(n, g):
    rad = _uniform(g, n) ** (1.0 / 3.0)
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    d = d / (d * d).sum(1).sqrt()[:, None]
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64) * math.sqrt(0.02)
    return {"pos": d * rad[:, None], "vel": v, "u": torch.full_like(rad, 1e-6),
            "rho": torch.full_like(rad, 3.0 / (4.0 * math.pi))}


def _particles(case, seed):
    """Fields of a particle set (device float64 tensors), and the time step to begin with."""
    n = case["n"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["model"] == "sphere":
        q = _sphere(n, g)
    elif case["model"] == "pair":
        n1 = n // 2
        a, b = _star(n1, case["poly"], case["n_ngb"], g), _star(n - n1, case["poly"], case["n_ngb"], g)
        off = torch.tensor([2.0, 0.0, 0.0], device="cuda", dtype=torch.float64)
        a["pos"], b["pos"] = a["pos"] - off, b["pos"] + off
        a["vel"], b["vel"] = a["vel"] + 0.25 * off, b["vel"] - 0.25 * off
        q = {k: torch.cat((a[k], b[k])) for k in a}
    else:
        q = _star(n, case["poly"], case["n_ngb"], g)
    # no particular order: files and samplers give none
    order = torch.randperm(n, generator=g, device="cuda")
    q = {k: v[order] for k, v in q.items()}
    m = torch.full((n,), (2.0 if case["model"] == "pair" else 1.0) / n, device="cuda", dtype=torch.float64)
    if case["masses"] == "unequal":
        m = m * (0.8 + 0.4 * _uniform(g, n))
    f = {"x": q["pos"][:, 0], "y": q["pos"][:, 1], "z": q["pos"][:, 2],
         "range": (3.0 * case["n_ngb"] * m / (4.0 * math.pi * q["rho"])) ** (1.0 / 3.0),
         "vx": q["vel"][:, 0], "vy": q["vel"][:, 1], "vz": q["vel"][:, 2], "m": m,
         "u": q["u"] * (1.0 + 0.1 * (_uniform(g, n) - 0.5)), "mu": torch.full_like(m, MU)}
    return {k: v.contiguous() for k, v in f.items()}, 0.02 * n ** (-1.0 / 3.0)


# ------------------------------------------------------------------------------------------------
# the program's side of the C ABI
# ------------------------------------------------------------------------------------------------
def _params(case):
    return make_params(n_target=case["n_ngb"], eos=case["eos"], soft=case["soft"], eps=case["eps"],
                       precision=case["precision"], grav_mode=1 if case["grav"] == "tree" else 0, theta=case["theta"])


def _ptrs(fields):
    p = (C.c_void_p * len(FIELDS))()
    for k, t in fields.items():
        p[FIELD_ID[k]] = t.data_ptr()
    return p


class _Context:
    """A context with its state on the device, and the buffers that the program reads it into."""

    def __init__(self, case, fields, dt):
        self.h = C.c_void_p()
        p = _params(case)
        n = case["n"]
        check(lib().cudasph_create(C.byref(p), n, 0, C.byref(self.h)), "create")
        s = C.c_void_p()
        check(lib().cudasph_get_stream(self.h, C.byref(s)), "get_stream")
        self.stream = torch.cuda.ExternalStream(s.value or 0)
        self.n, self.mixed = n, case["precision"] == "mixed"
        self.fields, self.ptrs = fields, _ptrs(fields)
        torch.cuda.synchronize()
        self.call("set_state", self.ptrs, 1)
        self.call("set_time", 0.0, dt)
        self.out = torch.empty(len(OUT), n, device="cuda", dtype=torch.float64)
        self.out_ptrs = _ptrs({k: self.out[i] for i, k in enumerate(OUT)})
        self.count = torch.empty(n, device="cuda", dtype=torch.int32)
        self.low = [k for k in OUT if k not in OUT64] if self.mixed else []
        self.rows = torch.tensor([OUT.index(k) for k in self.low], device="cuda", dtype=torch.int64)
        self.stats = np.empty(len(STATS), np.float64)

    def call(self, name, *a):
        check(getattr(lib(), "cudasph_" + name)(self.h, *a), name)

    def read(self):
        self.call("get_state", self.out_ptrs, 1)
        self.call("get_n_ngb", self.count.data_ptr(), 1)
        res = {k: self.out[i] for i, k in enumerate(OUT)}
        res["n_ngb"] = self.count
        if self.mixed:
            with torch.cuda.stream(self.stream):
                res.update(zip(self.low, self.out[self.rows].float()))
        return res

    def told(self):
        self.call("statistics", self.stats.ctypes.data)
        v = np.array([self.stats[STATS.index(k)] for k in TOLD])
        return v.astype(np.float32) if self.mixed else v

    def __del__(self):
        try:
            if self.h.value:
                lib().cudasph_destroy(self.h)
        except Exception:
            pass


def _pinned(t):
    return t.cpu().pin_memory().numpy()


def _tilt(case, seed):
    """Adjoints of a post-step state: those of a kinetic energy, with a smooth weight."""
    f, _ = _particles(case, seed)
    w = 1.0 + 0.5 * torch.sin(3.0 * f["x"] + 2.0 * f["y"])
    return {"vx": f["m"] * f["vx"] * w, "vy": f["m"] * f["vy"] * w, "vz": f["m"] * f["vz"] * w,
            "u": f["m"] * w, "rho": f["m"] * (0.1 * w)}


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    f, dt = _particles(case, seed)
    if kind == "gravity":
        out = torch.empty(n, 4, device="cuda", dtype=torch.float64)
        return dict(case=case, out=out, pos=torch.stack((f["x"], f["y"], f["z"], f["m"]), 1).contiguous(),
                    range=f["range"])
    if kind == "rollout":
        from cudasph_b200.autograd import RolloutContext

        host = {k: v.cpu().numpy() for k, v in f.items()}
        host["dt"] = dt
        rc = RolloutContext(host, _params(case), case["steps"], every=2)
        leaf = [torch.stack((f["x"], f["y"], f["z"]), 1), torch.stack((f["vx"], f["vy"], f["vz"]), 1), f["u"].clone()]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + 1)
        probe = torch.randint(0, n, (256,), generator=g, device="cuda")
        return dict(case=case, rc=rc, leaf=[t.requires_grad_(True) for t in leaf], m=f["m"], probe=probe)
    if kind == "host":
        host = {k: _pinned(v) for k, v in f.items()}
        host["dt"] = dt
        sim = Simulation(host, _params(case))
        host = {k: host[k] for k in IN}
        for k in ("ax", "ay", "az", "du"):
            host[k] = _pinned(torch.zeros(n, dtype=torch.float64))
        out = {k: _pinned(torch.zeros(n, dtype=torch.float64)) for k in OUT}
        sim.CUDA_solve_range()  # a running program's ranges
        sim.synchronize()
        host["range"][:] = sim.get("range")
        return dict(case=case, sim=sim, fin=host, out=out)
    ctx = _Context(case, f, dt)
    if kind == "step":
        if case["graph"]:
            ctx.call("set_graph", 1)
        ctx.call("solve_range")  # a running program's ranges
        ctx.call("synchronize")
        return dict(case=case, ctx=ctx)
    if kind == "forces":
        return dict(case=case, ctx=ctx)
    assert kind == "adjoint"
    ctx.call("set_keep", 1)
    ctx.call("solve_range")
    state = {k: torch.zeros(n, device="cuda", dtype=torch.float64) for k in IN + ("ax", "ay", "az", "du")}
    torch.cuda.synchronize()
    pre = _ptrs(state)
    ctx.call("get_state", pre, 1)
    ctx.call("synchronize")
    bar = _tilt(case, seed)
    full = {k: bar.get(k, torch.zeros(n, device="cuda", dtype=torch.float64)).contiguous() for k in ADJ_FIELDS}
    grad = torch.empty(11, n, device="cuda", dtype=torch.float64)
    return dict(case=case, ctx=ctx, dt=dt, state=state, pre=pre, bar=full, grad=grad)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gravity":
        p = state["pos"]
        check(lib().cudasph_gravity_direct(case["n"], p.data_ptr(), state["range"].data_ptr(), state["out"].data_ptr(),
                                           1 if case["soft"] == "plummer" else 0, case["eps"], 1.0,
                                           1 if case["precision"] == "mixed" else 0,
                                           torch.cuda.current_stream().cuda_stream), "gravity_direct")
        return state["out"].float() if case["precision"] == "mixed" else state["out"]
    if kind == "rollout":
        from cudasph_b200.autograd import rollout

        x, v, u = state["leaf"]
        vk, rho = rollout(x, v, u, state["rc"])
        loss = 0.5 * (state["m"][:, None] * vk * vk).sum() + rho[state["probe"]].mean()
        grads = torch.autograd.grad(loss, (x, v, u))
        res = (loss.detach(), vk.detach(), rho.detach()) + grads
        return tuple(t.float() for t in res) if case["precision"] == "mixed" else res
    if kind == "host":
        sim, out = state["sim"], state["out"]
        sim.step_host(state["fin"], out)
        if case["precision"] == "mixed":
            return {k: (out[k] if k in OUT64 else out[k].astype(np.float32)) for k in OUT}
        return out
    ctx = state["ctx"]
    if kind == "step":
        ctx.call("steps", case["steps"])
        res = ctx.read()
        res["told"] = ctx.told()
        return res
    if kind == "forces":
        ctx.call("set_state", ctx.ptrs, 1)
        ctx.call("sph_accelerations")
        ctx.call("gravity")
        return ctx.read()
    ctx.call("set_state", state["pre"], 1)
    ctx.call("set_time", 0.0, state["dt"])
    ctx.call("step")
    for k, t in state["bar"].items():
        ctx.call("adjoint_set_field", ADJ_ID[k], t.data_ptr(), 1)
    ctx.call("adjoint_set_dt", 0.01)
    ctx.call("adjoint")
    grad = state["grad"]
    for i, k in enumerate(ADJ_FIELDS[:11]):
        ctx.call("adjoint_get_field", ADJ_ID[k], grad[i].data_ptr(), 1)
    dtb = C.c_double()
    ctx.call("adjoint_get_dt", C.byref(dtb))
    if ctx.mixed:
        with torch.cuda.stream(ctx.stream):
            grad = grad.float()
    return {"grad": grad, "dtbar": np.float32(dtb.value) if ctx.mixed else dtb.value}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def work(case):
    """Bytes: each input field read and each output field written once.  Operations: a direct sum's N^2
    interactions at 20 (each pair's both directions), 42 for its reverse; per neighbour pair (the mean
    count is 1.4 n_ngb) 45 for the solve's one evaluation, 75 for the density and 70 for the hydro loop,
    twice that again in reverse; a tree walk of about 600 accepted nodes and near particles per target."""
    n, kind = float(case["n"]), case["kind"]
    direct = 20.0 * n * n if case["grav"] == "direct" else 600.0 * 30.0 * n
    pairs = 1.4 * case["n_ngb"] * n
    sph = 190.0 * pairs
    step = direct + sph
    if kind == "gravity":
        return {"bytes": 64.0 * n, "flops": direct}
    if kind == "adjoint":
        return {"bytes": 8.0 * n * (14 + 12 + 11), "flops": step + 2.1 * direct + 2.0 * sph}
    if kind == "rollout":
        k, every = case["steps"], 2
        replay = sum(min(every, k - s) * 2 - 1 for s in range(0, k, every))
        return {"bytes": 8.0 * n * (7 + 4 + 7), "flops": (k + replay) * step + k * (2.1 * direct + 2.0 * sph)}
    k = case["steps"] if kind == "step" else 1
    return {"bytes": 8.0 * n * (len(IN) + 4 + len(OUT)) * k, "flops": k * step}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch, over all pairs
# ------------------------------------------------------------------------------------------------
IPI, PI = 0.318309886183791, 3.141592653589793


def _w(u):
    t = (2.0 - u).clamp(min=0.0)
    return torch.where(u < 1, IPI * (1 - 1.5 * u * u + 0.75 * u ** 3), 0.25 * IPI * t ** 3)


def _dw(u):  # (1 / u) dW / du
    t = (2.0 - u).clamp(min=0.0)
    return torch.where(u < 1, IPI * (2.25 * u - 3), -0.75 * IPI * t * t / u.clamp(min=1.0))


def _dwdh(u):
    v = IPI * (-6 + 12 * u - 7.5 * u * u + 1.5 * u ** 3)
    return torch.where(u < 1, IPI * (-3 + 7.5 * u * u - 4.5 * u ** 3), torch.where(u < 2, v, 0.0))


def _dphidh(u):
    u2 = u * u
    v = 1.6 - 4 * u2 + 4 * u2 * u - 1.5 * u2 * u2 + 0.2 * u2 * u2 * u
    return torch.where(u < 1, 1.4 - 2 * u2 + 1.5 * u2 * u2 - 0.6 * u2 * u2 * u, torch.where(u < 2, v, 0.0))


def _ig(u):
    x = 4.0 * (1.0 - (u - 1.0).abs())
    x3 = x ** 3
    a = 4 * (x3 / 3.0 - 0.3 * x3 * x * x + 0.125 * x3 * x3)
    b = 4 * (-1.0 / 60 + 2.0 / 3 * x3 - 0.75 * x3 * x + 0.3 * x3 * x * x - x3 * x3 / 24.0)
    return torch.where(x <= 0, 0.0, torch.where(x < 1, a, torch.where(x < 2, b, 1.0)))


def _dig_du(u):
    s = torch.where(u < 1, 1.0, -1.0)
    x = 4.0 * torch.where(u < 1, u, 2.0 - u)
    return torch.where((u > 0) & (u < 2), 16.0 * PI * s * x * x * _w(x), 0.0)


def _row_chunks(n):
    r = max(1, min(n, (1 << 26) // n))
    return [(a, min(n, a + r)) for a in range(0, n, r)]


def _exact_gravity(pos, m, rng, soft, eps):
    n = pos.shape[0]
    out = torch.empty(n, 4, device=pos.device, dtype=torch.float64)
    for a, b in _row_chunks(n):
        d = [pos[None, :, k] - pos[a:b, None, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        if soft == "plummer":
            inv = (r2 + eps * eps).rsqrt()
            f = inv * inv * inv
            pot = -inv
        else:
            inv = torch.where(r2 > 0, r2, 1.0).rsqrt() * (r2 > 0)
            far = inv ** 3

            def soft_of(h):
                u2 = r2 / (h * h)
                u = u2.sqrt()
                us = u.clamp(min=0.5)
                lo = 10.666666666667 + u2 * (32.0 * u - 38.4)
                hi = (21.333333333333 - 48.0 * u + 38.4 * u2 - 10.666666666667 * u2 * u - 0.066666666667 / us ** 3)
                plo = -2.8 + u2 * (5.333333333333 + u2 * (6.4 * u - 9.6))
                phi = (-3.2 + 0.066666666667 / us +
                       u2 * (10.666666666667 + u * (-16.0 + u * (9.6 - 2.133333333333 * u))))
                near = r2 < h * h
                return (torch.where(near, torch.where(u < 0.5, lo, hi) / h ** 3, far),
                        torch.where(near, torch.where(u < 0.5, plo, phi) / h, -inv))

            gi, pot = soft_of(rng[a:b, None])
            f = 0.5 * (gi + soft_of(rng[None, :])[0])
        mf = m[None, :] * f
        for k in range(3):
            out[a:b, k] = (mf * d[k]).sum(1)
        out[a:b, 3] = (m[None, :] * pot).sum(1)
    return out


def _count_sums(pos, w, at):
    """Smooth neighbour number and its derivative's sum at ranges w of the particles `at`."""
    f, s = torch.empty_like(w), torch.empty_like(w)
    c = max(1, (1 << 26) // pos.shape[0])
    for a in range(0, at.numel(), c):
        i = at[a:a + c]
        d = pos[i][:, None, :] - pos[None, :, :]
        r2 = (d * d).sum(-1)
        ww = w[a:a + c, None]
        u = 2.0 * r2.sqrt() / ww
        inside = r2 < ww * ww
        f[a:a + c] = (_ig(u) * inside).sum(1)
        s[a:a + c] = -(u * _dig_du(u) * inside).sum(1)
    return f, s


def _solve_ranges(pos, w, target, rel=1e-3, fs=0.1, max_iter=20):
    """Bracket by clamped Newton steps, then safeguarded Newton, on every particle by itself."""
    n = w.numel()
    z = lambda: torch.zeros_like(w)  # noqa: E731
    w, dx, xl, ft, rx, ry = w.clone(), z(), z(), z(), z(), z()
    phase = torch.zeros(n, device=w.device, dtype=torch.int64)  # 0, 1 bracket; 2 solve; 3 done
    it = torch.zeros_like(phase)
    while True:
        at = torch.nonzero(phase < 3).flatten()
        if not at.numel():
            return w
        c, s = _count_sums(pos, w[at], at)
        W, P, I = w[at], phase[at], it[at]
        RX, RY, XL, FT = rx[at], ry[at], xl[at], ft[at]
        F = c - target
        S = s / W
        D = torch.where(S != 0, F / S, torch.where(F < 0, -W, W))
        br = P < 2
        hit = br & (D.abs() < rel * W)
        RX, RY = torch.where(hit, W - 0.5 * D.abs(), RX), torch.where(hit, W + 0.5 * D.abs(), RY)
        go = br & ~hit
        D = torch.where(go, D.clamp(-fs * W, fs * W), D)
        new = go & (P == 0)
        XL, FT, I = torch.where(new, W, XL), torch.where(new, F, FT), torch.where(new, 0, I)
        same = go & (FT * F >= 0)
        more = same & (I < max_iter)
        I = torch.where(same, I + 1, I)
        end = go & ~more
        lo, hi = torch.minimum(XL, W), torch.maximum(XL, W)
        RX, RY = torch.where(end, lo, RX), torch.where(end, hi, RY)
        XL, FT = torch.where(more, W, XL), torch.where(more, F, FT)
        init = hit | end
        sol = ~br
        RX, RY = torch.where(sol & (F < 0), W, RX), torch.where(sol & ~(F < 0), W, RY)
        keep = torch.where(sol, D.abs() > rel * W, torch.ones_like(sol))
        W = torch.where(more, W - D, W)
        P = torch.where(more, 1, P)
        W = torch.where(init, 0.5 * (RX + RY), W)
        D = torch.where(init, 0.0, D)
        wide = init & ((RX - RY).abs() > rel * W)
        I = torch.where(wide, 0, I)
        P = torch.where(init & ~wide, 3, P)
        chk = sol | wide
        on = chk & keep & (I < max_iter)
        I = torch.where(chk & keep, I + 1, I)
        W2 = W - D
        out = (W2 - RY) * (W2 - RX) >= 0
        W2 = torch.where(out, 0.5 * (RX + RY), W2)
        W = torch.where(on, W2, W)
        P = torch.where(on, 2, torch.where(chk, 3, P))
        w[at], phase[at], it[at], rx[at], ry[at], xl[at], ft[at] = W, P, I, RX, RY, XL, FT


def _exact_pressure(rho, u, eos):
    if eos == "ideal":
        return (GAMMA - 1.0) * rho * u
    d, e = rho * 5.89994031541978, u * 1.90698842928778e+15
    mu, kb, ar = MU * 1.66054e-24, 1.380658e-16, 7.56591414984829e-15
    t = (GAMMA - 1.0) * e * mu / kb  # energy of the gas alone: above the root
    t = torch.minimum(t, (d * e / ar) ** 0.25)
    for _ in range(60):  # e d = kb d T / (mu (gamma - 1)) + a T^4
        f = kb * d * t / (mu * (GAMMA - 1.0)) + ar * t ** 4 - d * e
        t = t - f / (kb * d / (mu * (GAMMA - 1.0)) + 4.0 * ar * t ** 3)
    return (d * kb * t / mu + ar / 3.0 * t ** 4) / 1.1251117914994e+16


def _exact_sph(pos, vel, m, u_th, w, eos, psi_on):
    n = m.numel()
    e = lambda: torch.empty_like(m)  # noqa: E731
    rho, div, curl, om, ps, du, vs = e(), e(), e(), e(), e(), e(), e()
    cnt = torch.empty(n, device=m.device, dtype=torch.int32)
    h = 0.5 * w

    def pairs(a, b):
        d = pos[a:b, None, :] - pos[None, :, :]
        dv = vel[a:b, None, :] - vel[None, :, :]
        r2 = (d * d).sum(-1)
        return d, dv, r2, (r2 < (w * w)[a:b, None]).to(torch.float64)

    chunks = [(a, min(n, a + max(1, (1 << 24) // n))) for a in range(0, n, max(1, (1 << 24) // n))]
    for a, b in chunks:
        d, dv, r2, k = pairs(a, b)
        u = r2.sqrt() / h[a:b, None]
        mj = m[None, :] * k
        cnt[a:b] = k.sum(1).to(torch.int32)
        s = -(u * _dig_du(u) * k).sum(1)
        hh = h[a:b]
        rho[a:b] = (mj * _w(u)).sum(1) / hh ** 3
        om[a:b] = (mj * _dwdh(u)).sum(1) / hh ** 3 / s
        ps[a:b] = (mj * _dphidh(u)).sum(1) / hh / s
        wt = mj * _dw(u)
        c = (wt[..., None] * torch.linalg.cross(d, dv)).sum(1)
        div[a:b] = (wt * (d * dv).sum(-1)).sum(1) / rho[a:b] / hh ** 5
        curl[a:b] = (c * c).sum(1).sqrt() / rho[a:b] / hh ** 5
    P = _exact_pressure(rho, u_th, eos)
    cs, pr = (GAMMA * P / rho).sqrt(), P / rho ** 2
    bal = div.abs() / (div.abs() + curl + 1e-4 * cs / h)
    acc = torch.zeros_like(pos)
    for a, b in chunks:
        d, dv, r2, k = pairs(a, b)
        r = r2.sqrt()
        ir = torch.where(r > 0, 1.0 / r.clamp(min=1e-300), 0.0)
        u = r / h[a:b, None]
        drdv = (d * dv).sum(-1)
        mu = torch.where(drdv < 0, drdv * ir, 0.0)
        cc = cs[a:b, None] + cs[None, :]
        q = mu / cc * (bal[a:b, None] + bal[None, :])
        visc = (pr[a:b, None] + pr[None, :]) * (2.0 * q * q - q)
        vs[a:b] = torch.where(k > 0, cc - 2.0 * mu, 0.0).max(1).values
        hi = h[a:b, None]
        ta = (pr[a:b, None] + 0.5 * visc) * _dw(u) / hi ** 5
        dig = _dig_du(u) * torch.where(r > 0, hi * ir, 0.0) / hi ** 2
        f = k * (ta - (pr * om + 0.5 * ps * psi_on)[a:b, None] / m[None, :] * dig)
        du[a:b] = (k * (m[None, :] * ta - (pr * om)[a:b, None] * dig) * drdv).sum(1)
        acc[a:b] -= ((m[None, :] * f)[..., None] * d).sum(1)
        acc += ((m[a:b, None] * f)[..., None] * d).sum(0)
    return dict(rho=rho, P=P, divv=div, curlv=curl, omega=om, psi=ps, du=du, vsig=vs, n_ngb=cnt, acc=acc)


DENSE = 20000  # largest set whose SPH sums are taken over all pairs


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind in ("adjoint", "rollout"):
        return None  # a reverse sweep has no plain dense form at these sizes
    f, dt = _particles(case, seed)
    pos = torch.stack((f["x"], f["y"], f["z"]), 1)
    if kind == "gravity":
        return _exact_gravity(pos, f["m"], f["range"], case["soft"], case["eps"]) if n <= 300000 else None
    if case["grav"] == "tree" or n > 300000 or (kind == "forces" and n > DENSE):
        return None
    vel = torch.stack((f["vx"], f["vy"], f["vz"]), 1)
    u, m = f["u"], f["m"]
    acc, du, t = torch.zeros_like(pos), torch.zeros_like(u), 0.0
    if n > DENSE:  # the positions and the direct sum; spline softening takes the solved ranges
        x = pos + vel * dt
        got = {"x": x[:, 0], "y": x[:, 1], "z": x[:, 2]}
        if case["soft"] == "plummer":
            g = _exact_gravity(x, m, None, "plummer", case["eps"])
            got.update(gx=g[:, 0], gy=g[:, 1], gz=g[:, 2], phi=g[:, 3])
        return {k: got.get(k) for k in OUT}
    w = f["range"]
    if kind != "forces":
        w = _solve_ranges(pos, w, case["n_ngb"])
    psi_on = 1.0 if case["soft"] == "spline" else 0.0
    for _ in range(case["steps"] if kind == "step" else 1):
        if kind != "forces":
            pos = pos + vel * dt
            vp, up = vel + acc * (0.5 * dt), u + du * (0.5 * dt)
        else:
            vp, up = vel, u
        w = _solve_ranges(pos, w, case["n_ngb"])
        s = _exact_sph(pos, vp, m, up, w, case["eos"], psi_on)
        g = _exact_gravity(pos, m, w, case["soft"], case["eps"])
        acc, du = s["acc"], s["du"]
        if kind == "forces":
            break
        acc = acc + g[:, :3]
        t += dt
        nn = s["n_ngb"].double()
        told = [0.5 * (m * g[:, 3]).sum(), 0.5 * (m[:, None] * vp * vp).sum(), (m * up).sum(), 0.0, nn.mean(), nn.min(),
                nn.max()]
        told[3] = told[0] + told[1] + told[2]
        dtv, dte = 0.3 * (w / s["vsig"]).abs(), 0.2 * (up / du).abs()
        new = float((1.0 / (1.0 / dtv + 1.0 / dte)).min())
        vel, u = vel + acc * (0.5 * (dt + new)), u + du * (0.5 * (dt + new))
        dt = new
    got = dict(s)
    del got["acc"]
    got.update(x=pos[:, 0], y=pos[:, 1], z=pos[:, 2], range=w, vx=vel[:, 0], vy=vel[:, 1], vz=vel[:, 2], u=u,
               ax=acc[:, 0], ay=acc[:, 1], az=acc[:, 2], gx=g[:, 0], gy=g[:, 1], gz=g[:, 2], phi=g[:, 3])
    if kind == "step":
        got["told"] = np.array([float(v) for v in told] + [dt, t])
    return got
