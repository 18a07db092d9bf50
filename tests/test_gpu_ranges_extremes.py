"""The smoothing-length solve at the ends of what it accepts: units of length
whose squares leave FP32, starting ranges of every size, parameters at the edge.

Lengths multiplied by a power of two give the same solve bit for bit (every
FP64 operation of it scales exactly), so the ranges must be equal after
division and the evaluation counts and lists must be the same."""
import numpy as np
import pytest

from cudasph_b200 import ics

pytestmark = pytest.mark.gpu


def _solve(ic, scale=1.0, wide=1.0, **kw):
    from cudasph_b200.simulation import Simulation, make_params
    ic = dict(ic)
    for k in "xyz":
        ic[k] = np.asarray(ic[k]) * scale
    ic["range"] = np.asarray(ic["range"]) * (scale * wide)
    with Simulation(ic, make_params(**dict(dict(n_target=50.0, eos_mode=0, soft_mode=1, eps=0.01), **kw))) as sim:
        sim.sort_bodies()
        order = sim.order()
        sim.CUDA_solve_range()
        cnt, _, lst = sim.neighbours()
        return sim.get("range") / scale, sim.solve_evals(), cnt, lst, order


@pytest.mark.parametrize("wide", [3.0, 6.0])
@pytest.mark.parametrize("log2", [64, 66, 68, -66])
def test_solve_from_wide_ranges_in_any_unit(log2, wide):
    """ranges far too large, whose sums are first taken in FP32"""
    ic = ics.polytrope(8200, n_ngb=50, seed=8200)
    a, b = _solve(ic, 1.0, wide), _solve(ic, 2.0 ** log2, wide)
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])
    assert np.array_equal(a[2], b[2])


def _cloud(n):
    rs = np.random.default_rng(n)
    x, y, z = rs.uniform(-1, 1, (3, n))
    return {"x": x, "y": y, "z": z, "range": np.full(n, 0.4), "m": np.full(n, 1.0 / n), "u": np.ones(n),
            "mu": np.full(n, 0.6)}


@pytest.mark.parametrize("n", [1, 5, 100, 1001, 2045])
def test_ranges_whose_square_is_infinite_in_fp32(n):
    """sets that fit one list of cells, with a part-filled last cell and chunk"""
    a, b = _solve(_cloud(n)), _solve(_cloud(n), 2.0 ** 70)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("log2", [130, 128, -68, -72, -130])
@pytest.mark.parametrize("n", [1001, 9000])
def test_lengths_at_the_ends_of_fp32(n, log2):
    """coordinates beyond FP32 and ranges whose squares are denormal in it"""
    ic = _cloud(n)
    ic["range"] = np.full(n, 0.4 * (1001 / n) ** (1 / 3))
    a, b = _solve(ic), _solve(ic, 2.0 ** log2)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("n", [100, 3000])
def test_infinite_starting_range(n):
    """Every particle is inside and all weights are those of u = 0: the bracket
    runs to its last iteration without a root and the range stays infinite."""
    ic = _cloud(n)
    ic["range"] = np.full(n, 0.4 * (1001 / n) ** (1 / 3))
    a = _solve(ic)
    ic["range"][5] = np.inf
    b = _solve(ic)
    assert b[0][5] == np.inf and b[2][5] == n and b[1][5] == 21
    others = np.arange(n) != 5
    for k in range(3):
        assert np.array_equal(a[k][others], b[k][others])


@pytest.mark.parametrize("f_scale", [1.0, 1.5, 3.0])
@pytest.mark.parametrize("wide", [0.3, 1.0, 5.0, 6.0])
def test_steps_larger_than_the_range(f_scale, wide):
    """Newton steps clamped to more than the range pass through negative ranges
    (about a third of the particles at five times the range, where ig is flat)."""
    from oracle import oracle as O
    ic = _cloud(2000)
    r, ev, cnt, _, order = _solve(ic, 1.0, wide, f_scale=f_scale)
    assert np.all(cnt[r == 0] == 0)
    x, y, z = (ic[k][order] for k in "xyz")
    r_o, _, ev_o = O.solve_range(x, y, z, wide * ic["range"][order], O.make_params(n_target=50.0, f_scale=f_scale))
    assert np.mean(r[order] == np.where(r_o > 0, r_o, 0.0)) >= 0.999  # a negative or undefined end is stored as 0
    assert np.mean(ev[order] == ev_o) >= 0.999


@pytest.mark.parametrize("n", [8200, 90001])
def test_solve_far_from_the_origin(n):
    """At 1e6 the coordinates' FP32 copies say nothing about neighbours; the
    solve is the oracle's there too, and takes about as long (a tenth of the
    allowance is usual) as at the origin."""
    from cudasph_b200.simulation import Simulation, make_params
    from oracle import oracle as O
    ms = []
    for shift in (0.0, 1e6):
        ic = ics.polytrope(n, n_ngb=50, seed=n)
        ic["x"] = ic["x"] + shift
        with Simulation(ic, make_params(n_target=50.0, eos_mode=0, soft_mode=1, eps=0.01)) as sim:
            sim.sort_bodies()
            order = sim.order()
            sim.CUDA_solve_range()
            r = sim.get("range")
            sim.set_profiling(True)
            t = []
            for _ in range(5):
                sim.reset_counters()
                sim.CUDA_solve_range()
                t.append(sim.phase_times()["solve_range"][0])
            ms.append(min(t))
        if n < 10000 or shift:
            x, y, z = (np.asarray(ic[k])[order] for k in "xyz")
            r_o, _, _ = O.solve_range(x, y, z, np.asarray(ic["range"])[order], O.make_params(n_target=50.0))
            assert np.mean(r[order] == r_o) >= 0.999
    assert ms[1] < 10 * ms[0]


@pytest.mark.parametrize("wide,rel_err", [(1.0, 1e-3), (1.02, 1e-3), (0.9, 1e-10)])
def test_groups_of_four_solve_as_single_targets(wide, rel_err):
    """Four targets to a warp and one (a shard of half the set takes the latter)
    give the same ranges, counts and evaluations, also with targets of no range,
    of ranges that are not a number, infinite, tiny and huge among the four."""
    from cudasph_b200.sharded import ShardedSimulation
    from cudasph_b200.simulation import Simulation, make_params
    n = 90_003
    ic = ics.polytrope(n, n_ngb=50, seed=5)
    rs = np.random.default_rng(5)
    r = np.asarray(ic["range"]) * wide
    for value in (0.0, np.nan, -0.1, np.inf, 1e-12, 3.0):
        r[rs.integers(0, n, 5 if value in (np.inf, 3.0) else 500)] = value
    ic["range"] = r
    par = make_params(n_target=50.0, eos_mode=0, soft_mode=1, eps=0.01, rel_err=rel_err)
    with Simulation(ic, par) as sim:
        sim.sort_bodies()
        sim.CUDA_solve_range()
        order, want = sim.order(), (sim.get("range"), sim.n_ngb(), sim.solve_evals())
        status = sim.device_status()
    for rank in range(2):
        with ShardedSimulation(ic, par, rank, 2) as half:
            half.sort_bodies()
            half.CUDA_solve_range()
            assert np.array_equal(half.order(), order)
            lo, hi = half.leaves()
            own = order[lo * 32:min(hi * 32, n)]
            for a, b in zip((half.get("range"), half.n_ngb(), half.solve_evals()), want):
                assert np.array_equal(a[own], b[own])
            assert half.device_status() & ~status == 0
