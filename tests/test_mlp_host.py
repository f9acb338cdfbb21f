"""Host logic of the MLP engines: the module and parameter lists they walk."""
import gc

import pytest
import torch
import torch.nn as nn

from voxurf_gb300 import _abi, mlp
from voxurf_gb300.mlp import _grad_buffers, _linears, _modules, _parameters


def _stacks():
    shared = nn.Linear(4, 4)
    yield nn.Sequential(nn.Linear(3, 4), nn.ReLU(), nn.Sequential(nn.Linear(4, 4), nn.ReLU()), nn.Linear(4, 3))
    yield nn.Sequential(shared, nn.Sequential(nn.Linear(4, 4, bias=False), shared, nn.ReLU()), nn.Linear(4, 3))
    yield nn.Linear(2, 3)


def test_walks_equal_torch():
    for net in _stacks():
        assert [id(m) for m in _modules(net)] == [id(m) for m in net.modules()]
        assert [id(p) for p in _parameters(net)] == [id(p) for p in net.parameters()]
        assert [id(m) for m in _linears(net)] == [id(m) for m in net.modules() if isinstance(m, nn.Linear)]


def test_walks_leave_no_cycles():
    """A cycle per call would hold the modules until the collector runs, which
    may be in the middle of a stream capture."""
    net = next(_stacks())
    gc.collect()
    gc.disable()
    try:
        for _ in range(10):
            _linears(net), _parameters(net)
        assert gc.collect() == 0
    finally:
        gc.enable()


def test_gradients_are_tensors_of_their_own():
    """Keeping or saving one gradient keeps no other alive, and changing one in
    place leaves what autograd saved of the others valid."""
    lin = _linears(next(_stacks()))
    grads = _grad_buffers(lin)
    assert [g.shape for g in grads] == [t.shape for m in lin for t in (m.weight, m.bias)]
    assert all(g.untyped_storage().nbytes() == 4 * g.numel() for g in grads)
    assert len({g.untyped_storage().data_ptr() for g in grads}) == len(grads)
    w = torch.ones_like(grads[2], requires_grad=True)
    loss = (grads[2].fill_(2.0) * w).sum()
    grads[3].zero_()
    loss.backward()
    assert bool((w.grad == 2.0).all())


def test_preallocated_buffers_are_checked(monkeypatch):
    """Buffers made for one row count serve fewer rows, with the capacities
    they have, and refuse more before anything is launched."""
    launched = []
    monkeypatch.setattr(_abi, "call_struct", lambda name, a, st: launched.append((name, a)))
    monkeypatch.setattr(mlp, "stream_ptr", lambda *a: 0)
    eng = mlp.TcTrainMLP(nn.Sequential(nn.Linear(20, 32), nn.ReLU(), nn.Linear(32, 32), nn.ReLU(), nn.Linear(32, 3)), 32)
    saved, work = {}, {}

    def one_pass(n, saved, work):
        x = torch.zeros((n, 32), dtype=torch.bfloat16)
        _, st = eng.forward(x, saved=saved)
        return eng.backward_chain(st, torch.zeros((n, 3)), work=work)[2]

    caps = [g.part_cap for g, *_ in one_pass(40_000, saved, work)]
    assert [g.part_cap for g, *_ in one_pass(500, saved, work)] == caps
    launched.clear()
    with pytest.raises(ValueError, match="too small"):
        one_pass(40_200, saved, {})
    with pytest.raises(ValueError, match="too small"):
        one_pass(40_200, {}, work)
    assert [name for name, _ in launched] == ["vx_mlp_train_forward"]   # the second one's own
