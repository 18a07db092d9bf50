"""The reverse sweep at the sizes where its launches change: 16 and 4 lanes per
particle, gravity with one tile, a ragged last tile and source slices.

Reference: the sweep is linear, so it is checked by the identity
<adjoint(y), dx> = <y, d step(dx)> with d step a central difference of the
forward step over a random smooth direction (FP64, h solve at 1e-12).  The
difference error is O(delta^2) and rounding O(1e-13 / delta): at delta = 1e-5
both are below 1e-7 of the value; neighbours entering or leaving a ball are
smooth in the kernels to second order.  Bound 1e-5."""
import numpy as np
import pytest

from cudasph_b200 import ics

pytestmark = pytest.mark.gpu

POST = ("vx", "vy", "vz", "u")
PRE = ("x", "y", "z", "vx", "vy", "vz", "u")


@pytest.mark.parametrize("n,equal", [(600, True), (1024, False), (1500, True), (2049, False), (8191, True), (8200, False)])
def test_adjoint_is_the_transpose_of_the_step(n, equal):
    from cudasph_b200.simulation import Simulation, make_params
    ic = ics.polytrope(n, n_ngb=40, seed=n)
    rs = np.random.default_rng(n)
    if not equal:
        ic["m"] = ic["m"] * rs.uniform(0.8, 1.2, n)
    ic["vx"], ic["vy"] = -0.2 * ic["y"], 0.2 * ic["x"] + 0.1 * ic["z"]
    ic["vz"] = -0.1 * ic["x"]
    ic["dt"] = 2e-3
    sim = Simulation(ic, make_params(n_target=40.0, rel_err=1e-12, max_iter=80, eos_mode=1, soft_mode=1, eps=0.02))
    sim.CUDA_solve_range()
    base = {k: sim.get(k) for k in ("x", "y", "z", "range", "vx", "vy", "vz", "u", "ax", "ay", "az", "du")}
    d = {k: np.sin(2.0 * base["x"] + i) * (1.0 if k == "u" else 0.5) * (base["u"] if k == "u" else 1.0)
         for i, k in enumerate(PRE)}
    y = {k: rs.normal(size=n) * ic["m"] for k in POST}

    def step(delta):
        for k, v in base.items():
            sim.set(k, v + delta * d[k] if k in d else v)
        sim.set_time(0.0, 2e-3)
        sim.step()
        return sum(float((y[k] * sim.get(k)).sum()) for k in POST)

    h = 1e-5
    want = (step(h) - step(-h)) / (2 * h)
    sim.set_keep(True)
    step(0.0)
    for k in ("x", "y", "z", "vx", "vy", "vz", "u", "ax", "ay", "az", "du"):
        sim.adjoint_set(k, y.get(k, np.zeros(n)))
    sim.adjoint_set_dt(0.0)
    sim.adjoint()
    got = sum(float((sim.adjoint_get(k) * d[k]).sum()) for k in PRE)
    scale = sum(float(np.abs(sim.adjoint_get(k) * d[k]).sum()) for k in PRE)
    assert abs(got - want) < 1e-5 * scale, (got, want, scale)
    sim.close()
