"""The radix sort at the edges of its tiles and of its three forms (direct
counting; small tiles; large tiles with the counts added up by the passes or by
a launch of their own): keys and permutation equal to a stable CPU sort, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 255, 2047, 2048, 2049, 4095, 4096, 4097, 6144, 8191, 8192, 8193, 12287, 12288, 12289,
         524287, 524288, 524289, 1048576, 1048577, 1300001]


def _keys(n, kind):
    rs = np.random.default_rng(n)
    k = rs.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + rs.integers(0, 2, n, dtype=np.uint64)
    if kind == "ties":
        k &= np.uint64(0x8001000300000701)
    if kind == "ones":  # the value that pads a part-filled tile
        k[::3] = np.uint64(0xFFFFFFFFFFFFFFFF)
    return k


@pytest.mark.parametrize("kind", ["random", "ties", "ones"])
@pytest.mark.parametrize("n", SIZES)
def test_radix_sort_is_the_stable_order(n, kind):
    import torch
    from cudasph_b200._capi import check, lib
    k = _keys(n, kind)
    order = np.argsort(k, kind="stable")
    dk = torch.from_numpy(k.view(np.int64).copy()).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    # a scratch buffer aligned to 8 bytes only, filled with rubbish
    scratch = torch.full((lib().cudasph_sort_scratch_bytes(n) // 8 + 2,), -1, dtype=torch.int64, device="cuda")[1:]
    s = torch.cuda.current_stream().cuda_stream
    check(lib().cudasph_radix_sort_u64(n, dk.data_ptr(), dv.data_ptr(), scratch.data_ptr(), s))
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(dv.cpu().numpy(), order)


@pytest.mark.parametrize("key_mode", [0, 1])
@pytest.mark.parametrize("n", [1, 33, 2049, 8193, 12288, 12289])
def test_sort_moves_every_record(n, key_mode):
    """A step's sort: the order is the stable sort of the oracle's keys (some
    particles coincide), and every field still belongs to its particle."""
    from cudasph_b200.simulation import FIELDS, Simulation, make_params
    from oracle import oracle as O
    rs = np.random.default_rng(n)
    ic = {k: rs.normal(size=n) for k in FIELDS}
    ic["m"] = np.full(n, 1.0 / n)
    ic["range"] = rs.uniform(0.1, 0.2, n)
    for k in ("x", "y", "z"):
        ic[k][1::5] = ic[k][0::5][: ic[k][1::5].size]
    sim = Simulation(ic, make_params(key_mode=key_mode))
    sim.sort_bodies()
    keys = (O.peano_keys if key_mode else O.morton_keys)(ic["x"], ic["y"], ic["z"])[0]
    np.testing.assert_array_equal(sim.order(), np.argsort(keys, kind="stable"))
    got = sim.get_state()
    for k in FIELDS:
        np.testing.assert_array_equal(got[k], ic[k], err_msg=k)
