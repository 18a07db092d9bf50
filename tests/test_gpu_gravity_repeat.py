"""Sets of one tile repeat bit for bit, although their sums are cut into slices:
the stand-alone sum and the gravity phase of a context, eager and replayed."""
import numpy as np
import pytest

from cudasph_b200 import ics
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("soft", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 129, 500, 1000, 1024])
def test_direct_sum_of_one_tile_repeats(n, soft, precision):
    import torch
    from cudasph_b200._capi import lib
    rs = np.random.default_rng(n)
    p, m, r = rs.normal(size=(n, 3)), rs.uniform(0.5, 1.5, n) / n, rs.uniform(0.2, 0.4, n) * n ** (-1 / 3)
    src, tr = torch.from_numpy(np.column_stack([p, m])).cuda(), torch.from_numpy(r).cuda()
    first = None
    for _ in range(20):
        out = torch.full((n, 4), np.nan, dtype=torch.float64, device="cuda")
        assert lib().cudasph_gravity_direct(n, src.data_ptr(), tr.data_ptr(), out.data_ptr(), soft, 0.05, 1.0, precision,
                                            torch.cuda.current_stream().cuda_stream) == 0
        got = out.cpu().numpy()
        first = got if first is None else first
        assert np.array_equal(got, first)
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=soft, eps=0.05)), 1)
    tol = 1e-12 if precision == 0 else 1e-5
    assert np.max(np.abs(first - ref)) <= tol * np.max(np.abs(ref))


@pytest.mark.parametrize("soft", [0, 1])
def test_gravity_phase_of_one_tile_repeats(soft):
    from cudasph_b200.simulation import Simulation, make_params
    ic = ics.polytrope(900, n_ngb=40, seed=2)
    sim = Simulation(ic, make_params(n_target=40.0, eos_mode=0, soft_mode=soft, eps=0.02))
    sim.sort_bodies()
    res = []
    for _ in range(20):
        sim.CUDA_gravity()
        res.append(np.stack([sim.get(k) for k in ("gx", "gy", "gz", "phi")]))
    assert all(np.array_equal(r, res[0]) for r in res)
    sim.set_graph(True)
    sim.step(4)
    g = np.stack([sim.get(k) for k in ("gx", "gy", "gz", "phi")])
    ref = O.gravity(*(sim.get(k) for k in ("x", "y", "z", "m", "range")), O.make_params(soft_mode=soft, eps=0.02))
    assert np.max(np.abs(g - np.stack(ref))) <= 1e-12 * np.max(np.abs(ref))
    sim.close()
