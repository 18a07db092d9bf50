"""What the torch rollout refuses and accepts as inputs (host logic, no GPU): a
state of another size than the context's would be read past its end."""
import numpy as np
import pytest
import torch

from cudasph_b200.autograd import _Budget, _checked, _State

N = 7


def _inputs(**kw):
    d = dict(x0=torch.zeros(N, 3), v0=torch.zeros(N, 3), u0=torch.arange(float(N)),
             ic={"range": np.ones(N), "ax": np.zeros(N)})
    d.update(kw)
    return d


@pytest.mark.parametrize("kw", [
    {"x0": torch.zeros(N - 1, 3)}, {"x0": torch.zeros(N + 1, 3)}, {"x0": torch.zeros(N, 2)}, {"x0": torch.zeros(3 * N)},
    {"x0": torch.zeros(1, 3)}, {"v0": torch.zeros(1, 3)}, {"v0": torch.zeros(3)}, {"v0": torch.zeros(N, 3, 2)},
    {"u0": torch.zeros(1)}, {"u0": torch.zeros(N + 1)}, {"u0": torch.tensor(1.0)},
    {"ic": {"range": np.ones(1)}}, {"ic": {"range": np.ones(N), "du": np.ones(N + 1)}},
    {"ic": {"range": 1.0}}])
def test_wrong_sizes_are_refused(kw):
    with pytest.raises(ValueError):
        _checked(N, **_inputs(**kw))


def test_initial_ranges_are_required():
    with pytest.raises(KeyError):
        _checked(N, **_inputs(ic={"ax": np.zeros(N)}))


def test_accepted_forms():
    x, v, u, f = _checked(N, **_inputs(x0=torch.arange(4.0 * N).reshape(N, 4), u0=torch.arange(float(N)).reshape(N, 1),
                                       ic={"range": [1.0] * N, "m": np.ones(3)}))
    assert _checked(N, **_inputs(v0=torch.zeros(N, 3, 1)))[1].shape == (N, 3, 1)
    assert x.shape == v.shape == (N, 3) and x[1, 0] == 4 and u.shape == (N,) and u[3] == 3
    assert set(f) == {"range"} and f["range"].shape == (N,)


def test_budget_of_the_states():
    b = _Budget(200)
    rows = torch.zeros(2, 10, dtype=torch.float64)  # 160 bytes
    first = _State(rows, 0.0, 0.0, b)
    second = _State(rows, 0.0, 0.0, b)
    assert first.held == 160 and second.held == 0 and b.left == 40
    del second
    assert b.left == 40
    with b._lock:  # freed by the garbage collector while a state is being made
        del first
    assert b.left == 200 and b.take(200) and not b.take(1)
