"""The neighbour lists as the caller gets them, over several of the host
buffers that the rows come through (4 MB) and with truncated lists: equal to a
search in the caller's own order, each list ascending by tree slot."""
import numpy as np
import pytest

from cudasph_b200 import ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap", [(33, 0), (4500, 0), (4520, 0), (30000, 0), (9000, 60), (5, 600000)])
def test_lists_in_the_callers_order(n, cap):
    from cudasph_b200.simulation import Simulation, make_params
    ic = ics.polytrope(n, n_ngb=50, seed=n) if n > 50 else {
        **{k: np.random.default_rng(n).uniform(-1, 1, n) for k in "xyz"}, "range": np.full(n, 1.2), "m": np.ones(n),
        "u": np.ones(n), "mu": np.ones(n)}
    with Simulation(ic, make_params(n_target=50.0, eos_mode=0, soft_mode=1, eps=0.01, ngb_cap=cap)) as sim:
        sim.sort_bodies()
        sim.find_ngb()
        cnt, off, lst = sim.neighbours()
        order = sim.order()
    x, y, z, r = (np.asarray(ic[k])[order] for k in ("x", "y", "z", "range"))
    c2, off2, l2 = O.find_ngb(x, y, z, r)
    assert np.array_equal(cnt[order], c2)
    for s in range(n):
        i, m = order[s], min(c2[s], cap or 232)
        assert np.array_equal(lst[off[i]:off[i] + m], order[l2[off2[s]:off2[s] + m]])
