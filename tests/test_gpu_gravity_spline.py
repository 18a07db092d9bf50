"""Spline-softened direct sum where its kernels change their way: one tile,
ragged last tiles of the symmetric form, launches cut into source slices, and
ranges from zero (Newtonian, coincident pairs included) to the whole cloud
(every pair near), unequal and equal masses.  Reference: the FP64 oracle.

Bounds: FP64 1e-12 of the largest value, as for the Plummer form (rounding of
sums of n terms); mixed 1e-5 RMS, FP32 pair terms."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _case(n, kind, equal):
    rs = np.random.default_rng(n)
    p = rs.normal(size=(n, 3)) * 0.4
    p[1::97] = p[0::97][: p[1::97].shape[0]]  # coincident pairs
    m = np.full(n, 1.0 / n) if equal else rs.uniform(0.5, 1.5, n) / n
    r = {"near": 0.3 * n ** (-1.0 / 3.0) * rs.uniform(0.5, 2.0, n), "all": np.full(n, 10.0),
         "zero": np.where(rs.random(n) < 0.5, 0.0, 0.05)}[kind]
    return p, m, r


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,kind", [(1, "near"), (31, "near"), (1000, "near"), (1024, "near"), (1025, "near"),
                                    (2049, "zero"), (2100, "all"), (5000, "near"), (9000, "zero"), (20001, "near")])
def test_spline_gravity_matches_oracle(n, kind, precision):
    import torch
    from cudasph_b200._capi import lib
    p, m, r = _case(n, kind, equal=False)
    src = torch.from_numpy(np.column_stack([p, m]).copy()).cuda()
    tr = torch.from_numpy(r.copy()).cuda()
    out = torch.full((n, 4), np.nan, dtype=torch.float64, device="cuda")
    rc = lib().cudasph_gravity_direct(n, src.data_ptr(), tr.data_ptr(), out.data_ptr(), 0, 0.0, 1.3, precision,
                                      torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    got = out.cpu().numpy()
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=0, G=1.3)), 1)
    if precision == 0:
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    else:
        scale = np.sqrt(np.mean(np.sum(ref[:, :3] ** 2, 1))) + (n == 1)
        assert np.sqrt(np.mean(np.sum((got - ref)[:, :3] ** 2, 1))) < 1e-5 * scale
        assert np.max(np.abs(got[:, 3] - ref[:, 3])) < 1e-5 * np.max(np.abs(ref[:, 3]))


@pytest.mark.parametrize("n", [1025, 4000])
def test_spline_gravity_equal_mass_step(n):
    """the step's gravity phase takes the equal-mass form"""
    from cudasph_b200.simulation import Simulation, make_params
    p, m, r = _case(n, "near", equal=True)
    ic = {"x": p[:, 0], "y": p[:, 1], "z": p[:, 2], "m": m, "range": r, "u": np.ones(n), "mu": np.full(n, 0.6)}
    sim = Simulation(ic, make_params(n_target=24.0, soft_mode=0, use_psi=1))
    sim.sort_bodies()
    sim.CUDA_gravity()
    got = np.stack([sim.get(k) for k in ("gx", "gy", "gz", "phi")], 1)
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=0)), 1)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    sim.close()


@pytest.mark.parametrize("n", [1025, 4096, 9001])
def test_spline_gravity_separated_clumps(n):
    """Tiles that hold no near pair beside tiles that do, and a few particles
    whose range reaches across: the batches with and without the per-pair test."""
    import torch
    from cudasph_b200._capi import lib
    rs = np.random.default_rng(n + 1)
    p = np.concatenate([rs.normal(size=(n - n // 2, 3)) * 0.1, rs.normal(size=(n // 2, 3)) * 0.1 + 4.0])
    m, r = rs.uniform(0.5, 1.5, n) / n, np.full(n, 0.02)
    r[rs.integers(0, n, 5)] = 5.0
    src = torch.from_numpy(np.column_stack([p, m]).copy()).cuda()
    tr = torch.from_numpy(r.copy()).cuda()
    out = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    assert lib().cudasph_gravity_direct(n, src.data_ptr(), tr.data_ptr(), out.data_ptr(), 0, 0.0, 1.0, 0,
                                        torch.cuda.current_stream().cuda_stream) == 0
    got = out.cpu().numpy()
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=0)), 1)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


def _direct(p, m, r):
    import torch
    from cudasph_b200._capi import lib
    n = m.size
    src = torch.from_numpy(np.column_stack([p, m]).copy()).cuda()
    tr = torch.from_numpy(np.asarray(r, np.float64).copy()).cuda()
    out = torch.full((n, 4), np.nan, dtype=torch.float64, device="cuda")
    assert lib().cudasph_gravity_direct(n, src.data_ptr(), tr.data_ptr(), out.data_ptr(), 0, 0.0, 1.0, 0,
                                        torch.cuda.current_stream().cuda_stream) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [1000, 1030, 2079, 5001])
@pytest.mark.parametrize("odd", [np.nan, 2e150, -0.3])
def test_spline_gravity_odd_ranges(n, odd):
    """Ranges of single particles that are no number (the pair is Newtonian on
    that side), beyond the place of the padding sources, and negative (the
    square counts), where the last batch of sources is part-filled."""
    p, m, r = _case(n, "near", equal=False)
    r[[0, 3, n // 2, n - 1]] = odd
    got = _direct(p, m, r)
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=0)), 1)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [1000, 1030, 5001])
def test_spline_gravity_infinite_range(n):
    """A pair inside an infinite range has no force and no potential from that side."""
    p, m, r = _case(n, "near", equal=False)
    r[[0, 3, n // 2, n - 1]] = np.inf
    got = _direct(p, m, r)
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=0)), 1)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [1000, 1030, 5001])
def test_spline_gravity_separations_with_denormal_squares(n):
    p, m, r = _case(n, "near", equal=False)
    p[0] = 0.0
    for k, d in ((1, [1e-160, 0, 0]), (n // 2, [0, 3e-158, -2e-159]), (n - 1, [-1e-154, 1e-155, 0])):
        p[k] = d
    got = _direct(p, m, r)
    ref = np.stack(O.gravity(p[:, 0], p[:, 1], p[:, 2], m, r, O.make_params(soft_mode=0)), 1)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
