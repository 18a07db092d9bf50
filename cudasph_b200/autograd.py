"""torch.autograd.Function over K steps of the device-resident step.

Forward runs K whole steps through the C ABI and keeps a checkpoint of the
particle state every `every` steps.  Backward walks the segments from the
last to the first: it re-runs the segment from its checkpoint to recover the
pre-step state of every step in it, then for each step (last first) replays
that one step with keep on and calls the hand-written adjoint kernels
(cudasph_adjoint), chaining the state adjoints from step to step.

Inputs:  x0 (N,3), v0 (N,3), u0 (N) -- float64 tensors (any device)
Outputs: v_K (N,3), rho_K (N) -- the velocities after K steps and the density
         computed in the last step; a loss such as kinetic energy plus the mean
         density at probe particles is formed from them in torch.
Gradients flow to x0, v0, u0.  This is a test / harness binding: the step and
its adjoint run in libcudasph_b200.so.

Checkpoints, replayed states and the state adjoints stay on the device, in
tensors of the context's own stream (exchanged through host arrays, 12 fields
at a time, the transfers and their synchronisations were about 40 % of a
rollout of 12,001 particles: 16.4 -> 9.9 ms).  A state is 96 bytes per
particle; a context holds as many on the device as fit in a quarter of the
memory that was free when it was created, and the others on the host, so that
the length of a rollout is not limited by the device's memory.
"""
from __future__ import annotations

import ctypes as C
import threading
from collections import deque

import numpy as np
import torch

from ._capi import ADJ_ID, FIELD_ID, FIELDS, check, lib
from .simulation import Simulation

STATE = ("x", "y", "z", "range", "vx", "vy", "vz", "u", "ax", "ay", "az", "du")
ADJ = ("x", "y", "z", "vx", "vy", "vz", "u", "ax", "ay", "az", "du")
ROW = {k: i for i, k in enumerate(STATE)}


class _Budget:
    """Bytes of device memory that the states of a context may still take."""

    def __init__(self, size: int):
        self._left = size
        self._given = deque()
        self._lock = threading.Lock()

    def _gather(self):
        while self._given:
            self._left += self._given.popleft()

    def take(self, size: int) -> bool:
        with self._lock:
            self._gather()
            fits = size <= self._left
            if fits:
                self._left -= size
            return fits

    def give(self, size: int):
        # without the lock: the garbage collector may free a state inside take()
        self._given.append(size)

    @property
    def left(self) -> int:
        with self._lock:
            self._gather()
            return self._left


class _State:
    """A particle state: a (12, N) tensor of the rows STATE, on the device while
    the budget lasts and else on the host, with time and dt."""

    def __init__(self, rows, time: float, dt: float, budget: _Budget):
        size = rows.numel() * rows.element_size()
        self.held = size if budget.take(size) else 0
        self.rows = rows if self.held else rows.cpu()
        self.time, self.dt, self.budget = time, dt, budget

    def __del__(self):
        if getattr(self, "held", 0):
            self.budget.give(self.held)


class RolloutContext:
    """The simulation and the fixed part of the initial conditions.
    device_bytes: device memory for the states (default: a quarter of what is
    free)."""

    def __init__(self, ic: dict, params, steps: int, every: int = 5, device: int = 0, device_bytes: int | None = None):
        self.ic = ic
        self.params = params
        self.steps = int(steps)
        self.every = max(1, int(every))
        self.sim = Simulation(ic, params, device=device)
        self.sim.set_keep(True)
        if device_bytes is None:
            device_bytes = torch.cuda.mem_get_info(device)[0] // 4
        self.budget = _Budget(device_bytes)

    def close(self):
        self.sim.close()
        # torch keeps freed memory for the stream it was used on, which is gone
        torch.cuda.empty_cache()

    # The library works on the context's stream; the callers below make that
    # the current one, so every tensor here is allocated, written and freed on it.
    def _set(self, rows, time: float, dt: float):
        rows = rows.to(f"cuda:{self.sim.device}")
        check(lib().cudasph_set_state(self.sim._h, _pointers(rows, STATE), 1), "set_state")
        self.sim.set_time(time, dt)

    def _read(self, names):
        rows = torch.empty(len(names), self.sim.n, dtype=torch.float64, device=f"cuda:{self.sim.device}")
        check(lib().cudasph_get_state(self.sim._h, _pointers(rows, names), 1), "get_state")
        return rows

    def _get(self):
        t, d = C.c_double(), C.c_double()
        rows = self._read(STATE)
        check(lib().cudasph_get_time(self.sim._h, C.byref(t), C.byref(d)), "get_time")
        return _State(rows, t.value, d.value, self.budget)


def _pointers(rows, names):
    p = (C.c_void_p * len(FIELDS))()
    for i, k in enumerate(names):
        p[FIELD_ID[k]] = rows[i].data_ptr()
    return p


class _OnStream:
    """Runs the body on the context's stream, ordered after the work that the
    caller's stream holds and before what it gets later.  So a caller's tensor
    may be read, and one that was allocated on the caller's stream before may
    be written, in the body; what the body allocates belongs to the context's
    stream and stays inside (states) or is copied out."""

    def __init__(self, sim):
        check(lib().cudasph_get_stream(sim._h, C.byref(C.c_void_p())), "rollout")  # a closed context has no stream
        self.stream = sim.torch_stream()
        self.device = torch.device("cuda", sim.device)

    def __enter__(self):
        self.caller = torch.cuda.current_stream(self.device)
        self.stream.wait_stream(self.caller)
        self.guard = torch.cuda.stream(self.stream)
        self.guard.__enter__()
        return self

    def __exit__(self, *a):
        self.guard.__exit__(*a)
        self.caller.wait_stream(self.stream)

    def take(self, t):
        """A caller's tensor in float64 on the context's device."""
        return t.detach().to(self.device, torch.float64)


def _results(sim, *shapes):
    """Float64 tensors of the caller's stream on the context's device."""
    return [torch.empty(s, dtype=torch.float64, device=f"cuda:{sim.device}") for s in shapes]


def _checked(n, x0, v0, u0, ic):
    """The first three columns of x0 and v0, u0 as a vector, and the fields
    taken from the initial conditions, each for the context's n particles (a
    state of another size would be read past its end, or spread over all)."""
    for name, t in (("x0", x0), ("v0", v0)):
        if t.dim() < 2 or t.shape[1] < 3 or t[:, 0].numel() != n:
            raise ValueError(f"rollout: {name} has shape {tuple(t.shape)}, ({n}, 3) is required")
    if u0.numel() != n:
        raise ValueError(f"rollout: u0 has {u0.numel()} values, {n} are required")
    if "range" not in ic:
        raise KeyError("range")
    fields = {k: np.array(ic[k], np.float64).reshape(-1) for k in ("range", "ax", "ay", "az", "du") if k in ic}
    for k, a in fields.items():
        if a.size != n:
            raise ValueError(f"rollout: {k} of the initial conditions has {a.size} values, {n} are required")
    return x0[:, :3], v0[:, :3], u0.reshape(-1), fields


class Rollout(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x0, v0, u0, rc: RolloutContext):
        n = rc.sim.n
        x0, v0, u0, fields = _checked(n, x0, v0, u0, rc.ic)
        vK, rhoK = _results(rc.sim, (n, 3), (n,))
        with _OnStream(rc.sim) as on:
            rows = torch.zeros(len(STATE), n, dtype=torch.float64, device=on.device)
            for k, a in fields.items():
                rows[ROW[k]].copy_(torch.from_numpy(a))
            rows[ROW["x"]:ROW["z"] + 1] = on.take(x0).transpose(0, 1).reshape(3, n)
            rows[ROW["vx"]:ROW["vz"] + 1] = on.take(v0).transpose(0, 1).reshape(3, n)
            rows[ROW["u"]] = on.take(u0)
            rc._set(rows, float(rc.ic.get("time", 0.0)), float(rc.ic.get("dt", 0.0)))
            ckpt = {0: rc._get()}
            for s in range(rc.steps):
                rc.sim.step()
                if (s + 1) % rc.every == 0 and s + 1 < rc.steps:
                    ckpt[s + 1] = rc._get()
            last = rc._read(("vx", "vy", "vz", "rho"))
            vK.copy_(last[:3].t())
            rhoK.copy_(last[3])
        ctx.rc = rc
        ctx.ckpt = ckpt
        ctx.dev = x0.device
        return vK.to(x0.device), rhoK.to(x0.device)

    @staticmethod
    def backward(ctx, gv, grho):
        rc, ckpt = ctx.rc, ctx.ckpt
        sim = rc.sim
        n = sim.n
        h = sim._h
        gx, gvv, gu = _results(sim, (n, 3), (n, 3), (n,))
        with _OnStream(sim) as on:
            adj = torch.zeros(len(ADJ), n, dtype=torch.float64, device=on.device)
            if gv is not None:
                adj[3:6] = on.take(gv).t()
            rho_bar = on.take(grho).contiguous() if grho is not None else None
            dtbar = 0.0
            starts = sorted(ckpt)
            for si in range(len(starts) - 1, -1, -1):
                s0 = starts[si]
                s1 = starts[si + 1] if si + 1 < len(starts) else rc.steps
                # pre-step states of the segment
                pre = [ckpt[s0]]
                rc._set(pre[0].rows, pre[0].time, pre[0].dt)
                for s in range(s0, s1 - 1):
                    sim.step()
                    pre.append(rc._get())
                for s in range(s1 - 1, s0 - 1, -1):
                    st = pre[s - s0]
                    rc._set(st.rows, st.time, st.dt)
                    sim.step()  # replays step s with keep on
                    for i, k in enumerate(ADJ):
                        check(lib().cudasph_adjoint_set_field(h, ADJ_ID[k], adj[i].data_ptr(), 1), "adjoint_set")
                    if s == rc.steps - 1 and rho_bar is not None:
                        check(lib().cudasph_adjoint_set_field(h, ADJ_ID["rho"], rho_bar.data_ptr(), 1), "adjoint_set")
                    sim.adjoint_set_dt(dtbar)
                    sim.adjoint()
                    for i, k in enumerate(ADJ):
                        check(lib().cudasph_adjoint_get_field(h, ADJ_ID[k], adj[i].data_ptr(), 1), "adjoint_get")
                    dtbar = sim.adjoint_get_dt()
            gx.copy_(adj[0:3].t())
            gvv.copy_(adj[3:6].t())
            gu.copy_(adj[6])
        return gx.to(ctx.dev), gvv.to(ctx.dev), gu.to(ctx.dev), None


def rollout(x0, v0, u0, rc: RolloutContext):
    return Rollout.apply(x0, v0, u0, rc)
