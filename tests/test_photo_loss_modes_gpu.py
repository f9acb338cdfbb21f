"""fine_loss where its kernels may not stand for the chain of torch operations:
under what sees every operation, and in backward passes of a batch of upstream
gradients.  The chain below is the reference (run.py:604-627)."""
import pytest
import torch
import torch.nn.functional as F
from torch.fx.experimental.proxy_tensor import make_fx
from torch.utils._python_dispatch import TorchDispatchMode

from voxurf_gb300 import train
from voxurf_gb300.train import fine_loss

pytestmark = pytest.mark.gpu

KEYS = ("rgb_marched", "rgb_marched0", "alphainv_cum")


def _chain(ret, target):
    p = ret["alphainv_cum"][..., -1].clamp(1e-6, 1 - 1e-6)
    entropy = -(p * torch.log(p) + (1 - p) * torch.log(1 - p)).mean()
    return (F.mse_loss(ret["rgb_marched"], target) + 0.001 * entropy
            + F.mse_loss(ret["rgb_marched0"], target) * 0.5)


def _inputs(seed, dev, n=40):
    g = torch.Generator().manual_seed(seed)
    x = [torch.rand((n, 3), generator=g), torch.rand((n, 3), generator=g), torch.rand(n, generator=g) * 0.8 + 0.1]
    return [t.to(dev).requires_grad_() for t in x], torch.rand((n, 3), generator=g).to(dev)


def _loss(f, xs, target):
    return f(dict(zip(KEYS, xs)), target)


@pytest.mark.parametrize("backward", [False, True])
def test_traced_graph_follows_its_inputs(cuda, backward):
    """A graph traced with real tensors gives the loss (and the gradients) of
    the inputs it is replayed on."""
    def f(a, b, c, target):
        loss = _loss(fine_loss, (a, b, c), target)
        return (loss, *torch.autograd.grad(loss, (a, b, c))) if backward else (loss,)

    xs, target = _inputs(0, cuda)
    graph = make_fx(f)(*xs, target)
    xs, target = _inputs(1, cuda)
    got = graph(*xs, target)
    loss = _loss(_chain, xs, target)
    want = (loss, *torch.autograd.grad(loss, xs)) if backward else (loss,)
    for a, b in zip(got, want):
        torch.testing.assert_close(a.detach(), b.detach(), rtol=1e-5, atol=1e-9)


def test_traced_backward_of_an_outer_loss(cuda):
    """The backward alone, traced, of a loss formed outside the trace."""
    xs, target = _inputs(2, cuda)
    loss = _loss(fine_loss, xs, target)
    graph = make_fx(lambda g: torch.autograd.grad(loss, xs, g, retain_graph=True))(torch.ones((), device=cuda))
    got = graph(torch.full((), 3.0, device=cuda))
    want = torch.autograd.grad(3.0 * _loss(_chain, xs, target), xs)
    for a, b in zip(got, want):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-9)


class _Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.ops = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.ops.append(str(func))
        return func(*args, **(kwargs or {}))


def test_dispatch_mode_sees_the_operations(cuda):
    xs, target = _inputs(3, cuda)
    with _Seen() as seen:
        _loss(fine_loss, xs, target)
    assert any("mse_loss" in op for op in seen.ops)


def test_default_device_keeps_the_kernels(cuda, monkeypatch):
    used = []
    orig = train._PhotoLoss.apply
    monkeypatch.setattr(train._PhotoLoss, "apply", lambda *a: (used.append(1), orig(*a))[1])
    xs, target = _inputs(4, cuda)
    with torch.device(cuda):
        _loss(fine_loss, xs, target)
    assert used


@pytest.mark.parametrize("how", ["is_grads_batched", "vmap", "jacobian"])
def test_batched_upstream_gradients(cuda, how):
    """A batch of upstream gradients through one loss: each one's own result."""
    xs, target = _inputs(5, cuda)
    ups = torch.tensor([1.0, -2.5, 0.0], device=cuda)
    want = [torch.autograd.grad(u * _loss(_chain, xs, target), xs) for u in ups]
    loss = _loss(fine_loss, xs, target)
    if how == "is_grads_batched":
        got = torch.autograd.grad(loss, xs, ups, is_grads_batched=True)
    elif how == "vmap":
        got = torch.func.vmap(lambda u: torch.autograd.grad(loss, xs, u, retain_graph=True))(ups)
    else:
        got = torch.autograd.functional.jacobian(
            lambda *x: ups * _loss(fine_loss, x, target), tuple(t.detach() for t in xs), vectorize=True)
    for k in range(3):
        torch.testing.assert_close(got[k], torch.stack([w[k] for w in want]), rtol=1e-5, atol=1e-9)
