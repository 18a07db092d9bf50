"""The torch binding's rollout with its inputs on the CPU, on the device, and on
the device while the caller works on a stream of its own: the same gradients
(order of FP64 atomics: 1e-11), on the inputs' device, also when the backward
pass runs twice on one graph and after the simulation is closed."""
import numpy as np
import pytest
import torch

from cudasph_b200 import ics

pytestmark = pytest.mark.gpu


def _grads(where, side):
    from cudasph_b200.autograd import RolloutContext, rollout
    from cudasph_b200.simulation import make_params
    ic = ics.polytrope(700, n_ngb=40, seed=4)
    ic["dt"] = 1e-3
    rc = RolloutContext(ic, make_params(n_target=40.0, eos_mode=0, soft_mode=1, eps=0.02), steps=3, every=2)
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    with torch.cuda.stream(stream):
        x, v, u = (torch.from_numpy(a).to(where) for a in (
            np.stack([ic[k] for k in "xyz"], 1), 0.1 * np.stack([ic[k] for k in "yzx"], 1), ic["u"].copy()))
        if where != "cpu":
            torch.cuda._sleep(20_000_000)  # the inputs are late
        x, v, u = (t.clone().requires_grad_(True) for t in (x, v, u))
        vk, rho = rollout(x, v, u, rc)
        loss = (vk * vk).sum() + rho[:50].mean()
        g = torch.autograd.grad(loss, (x, v, u), retain_graph=True)
        g2 = torch.autograd.grad(loss, (x, v, u))
    rc.close()
    assert all(t.device.type == torch.device(where).type for t in (vk, rho) + g)
    res = [t.detach().cpu() for t in (vk, rho) + g]
    torch.cuda.synchronize()
    for a, b in zip(g, g2):
        assert (a - b).abs().max() <= 1e-11 * a.abs().max()
    return res


def test_rollout_is_the_same_from_every_device_and_stream():
    ref = _grads("cpu", False)
    for where, side in (("cuda", False), ("cuda", True)):
        for a, b in zip(_grads(where, side), ref):
            assert (a - b).abs().max() <= 1e-11 * b.abs().max()


def test_rollout_of_a_closed_context_is_refused():
    from cudasph_b200._capi import SphError
    from cudasph_b200.autograd import RolloutContext, rollout
    from cudasph_b200.simulation import make_params
    ic = ics.polytrope(700, n_ngb=40, seed=4)
    rc = RolloutContext(ic, make_params(n_target=40.0, eos_mode=0, soft_mode=1, eps=0.02), steps=1)
    x = torch.from_numpy(np.stack([ic[k] for k in "xyz"], 1)).requires_grad_(True)
    v, u = torch.zeros(700, 3, dtype=torch.float64), torch.from_numpy(ic["u"])
    vk, _ = rollout(x, v, u, rc)
    rc.close()
    with pytest.raises(SphError):
        torch.autograd.grad(vk.sum(), x)
    with pytest.raises(SphError):
        rollout(x, v, u, rc)


@pytest.mark.parametrize("states", [0, 2])
def test_states_beyond_the_device_memory_are_held_on_the_host(states):
    from cudasph_b200.autograd import RolloutContext, rollout
    from cudasph_b200.simulation import make_params
    ic = ics.polytrope(700, n_ngb=40, seed=4)
    ic["dt"] = 1e-3
    res = []
    for limit in (None, states * 700 * 96):
        rc = RolloutContext(ic, make_params(n_target=40.0, eos_mode=0, soft_mode=1, eps=0.02), steps=6, every=3,
                            device_bytes=limit)
        free = rc.budget.left
        assert limit is not None or free > 1 << 30
        x, v, u = (torch.from_numpy(a).requires_grad_(True) for a in (
            np.stack([ic[k] for k in "xyz"], 1), 0.1 * np.stack([ic[k] for k in "yzx"], 1), ic["u"].copy()))
        vk, rho = rollout(x, v, u, rc)
        ckpt = vk.grad_fn.ckpt
        assert [s.rows.is_cuda for s in ckpt.values()] == [limit is None or k < states for k in range(2)]
        assert free - rc.budget.left == 700 * 96 * sum(s.rows.is_cuda for s in ckpt.values())
        res.append([vk.detach(), rho.detach(), *torch.autograd.grad((vk * vk).sum() + rho[:50].mean(), (x, v, u))])
        del vk, rho, ckpt
        assert rc.budget.left == free
        rc.close()
    for a, b in zip(*res):
        assert (a - b).abs().max() <= 1e-11 * b.abs().max()
