"""The equal-mass form of the direct sum follows the masses a caller sets, also
between steps replayed from a graph: a context whose masses were equal, then
unequal, then equal again equals one made with those masses.  Same kernels on
the same state: bound 1e-12 (order of FP64 atomics)."""
import numpy as np
import pytest

from cudasph_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
def test_masses_set_between_steps(graph, precision):
    from cudasph_b200.simulation import Simulation, make_params
    n = 3000
    ic = ics.polytrope(n, n_ngb=40, seed=8)
    ic["dt"] = 1e-3
    kw = dict(n_target=40.0, eos_mode=0, soft_mode=1, eps=0.02, precision=precision)
    sim = Simulation(ic, make_params(**kw))
    sim.set_graph(graph)
    sim.step(4)
    rs = np.random.default_rng(1)
    for m in (ic["m"] * rs.uniform(0.5, 1.5, n), ic["m"] * 2.0):
        sim.set("m", m)
        state = {k: sim.get(k) for k in ("x", "y", "z", "range", "vx", "vy", "vz", "m", "u", "mu", "ax", "ay", "az", "du")}
        state.update(time=sim.time, dt=sim.dt)
        ref = Simulation(state, make_params(**kw))
        sim.step()
        ref.step()
        for k in ("gx", "gy", "gz", "phi", "ax", "rho"):
            a, b = sim.get(k), ref.get(k)
            assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b)), k
        ref.close()
        sim.step(2)
    sim.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_masses_set_between_a_kept_step_and_its_reverse_sweep(precision):
    """The reverse sweep of gravity belongs to the sources the step packed:
    unequal masses, although equal ones were set since.  Cold gas, so that the
    hydro part (1e-6 of the whole) does not count."""
    from cudasph_b200.simulation import Simulation, make_params
    n = 3000
    ic = ics.polytrope(n, n_ngb=40, seed=8)
    rs = np.random.default_rng(2)
    ic["m"] = ic["m"] * rs.uniform(0.1, 2.0, n)
    ic["u"] = ic["u"] * 1e-9
    ic["dt"] = 1e-3
    y = {k: rs.normal(size=n) for k in ("vx", "vy", "vz")}
    res = []
    for later in (False, True):
        sim = Simulation(ic, make_params(n_target=40.0, eos_mode=0, soft_mode=1, eps=0.02, precision=precision))
        sim.set_keep(True)
        sim.step()
        for k in ("x", "y", "z", "vx", "vy", "vz", "u", "ax", "ay", "az", "du"):
            sim.adjoint_set(k, y.get(k, np.zeros(n)))
        sim.adjoint_set_dt(0.0)
        if later:
            sim.set("m", np.full(n, 1.0 / n))
        sim.adjoint()
        res.append(np.stack([sim.adjoint_get(k) for k in "xyz"]))
        sim.close()
    assert np.max(np.abs(res[1] - res[0])) <= 1e-3 * np.max(np.abs(res[0]))
