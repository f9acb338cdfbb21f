"""fine_loss in one launch against the chain of torch operations it stands for
(run.py:604-627), in 64 bits and by the cases that keep the chain."""
import pytest
import torch
import torch.nn.functional as F

from voxurf_gb300 import train
from voxurf_gb300.train import fine_loss

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _chain(ret, target, wm, we, w0):
    loss = wm * F.mse_loss(ret["rgb_marched"], target)
    if we > 0:
        p = ret["alphainv_cum"][..., -1].clamp(1e-6, 1 - 1e-6)
        loss = loss + we * (-(p * torch.log(p) + (1 - p) * torch.log(1 - p)).mean())
    if w0 > 0 and "rgb_marched0" in ret:
        loss = loss + F.mse_loss(ret["rgb_marched0"], target) * w0
    return loss


def _batch(n, last, cuda, with0=True):
    g = torch.Generator().manual_seed(n)
    ret = {"rgb_marched": torch.rand((n, 3), generator=g), "alphainv_cum": torch.rand(n, generator=g)}
    if with0:
        ret["rgb_marched0"] = torch.rand((n, 3), generator=g)
    ret["alphainv_cum"][-1] = last
    target = torch.rand((n, 3), generator=g).to(cuda)
    return {k: v.to(cuda).requires_grad_() for k, v in ret.items()}, target


# one block up to 65536 elements, several beyond; the entropy inside and outside its clamp
@pytest.mark.parametrize("last", [0.3, 0.0, 1.0, 1e-6, 0.999999])
@pytest.mark.parametrize("n", [1, 5, 341, 342, 21845, 21846, 100_003])
@pytest.mark.parametrize("weights", [(1.0, 0.001, 0.5), (0.7, 0.0, 0.0), (2, 0.01, 1.5)])
def test_loss_and_gradients(cuda, weights, n, last):
    ret, target = _batch(n, last, cuda)
    used = []
    orig = train._PhotoLoss.apply
    train._PhotoLoss.apply = lambda *a: (used.append(1), orig(*a))[1]
    try:
        loss = fine_loss(ret, target, *weights)
    finally:
        train._PhotoLoss.apply = orig
    assert used and loss.shape == () and loss.dtype == torch.float32
    (3.0 * loss).backward()
    ref = {k: v.detach().double().requires_grad_() for k, v in ret.items()}
    exact = _chain(ref, target.double(), *weights)
    (3.0 * exact).backward()
    # per term: the rounded difference, its square, the mean, the weight, the sums
    assert abs(float(loss.detach()) - float(exact.detach())) <= 8 * EPS * abs(float(exact.detach())) + 1e-12
    for k in ret:
        if ref[k].grad is None:
            assert ret[k].grad is None
            continue
        d = (ret[k].grad.double() - ref[k].grad).abs()
        # difference, norm, two products; the entropy's logarithms are within 2 ulp
        # of values up to 14 and cancel at p = 1/2, its clamp is compared in 32 bits
        if k == "alphainv_cum" and last in (1e-6, 0.999999):
            continue
        tol = 6 * EPS * ref[k].grad.abs() + (60 * EPS * 3 * weights[1] if k == "alphainv_cum" else 0)
        tol = tol + (4 * EPS * 2 / (3 * n) * 3 * 2 if k != "alphainv_cum" else 0)
        assert bool((d <= tol).all()), (k, float(d.max()))
    # the 32-bit chain itself, where the clamp's edge decides
    ret32 = {k: v.detach().clone().requires_grad_() for k, v in ret.items()}
    (3.0 * _chain(ret32, target, *weights)).backward()
    if weights[1] > 0:
        torch.testing.assert_close(ret["alphainv_cum"].grad, ret32["alphainv_cum"].grad, rtol=1e-5, atol=1e-7)


def test_nan_and_no_second_term(cuda):
    ret, target = _batch(100, float("nan"), cuda, with0=False)
    assert bool(fine_loss(ret, target).isnan())
    ret, target = _batch(100, 0.5, cuda, with0=False)
    torch.testing.assert_close(fine_loss(ret, target), _chain(ret, target, 1.0, 0.001, 0.5), rtol=1e-6, atol=0)


def test_second_derivatives_match_the_chain(cuda):
    outs = []
    for f in (lambda r, t: fine_loss(r, t), lambda r, t: _chain(r, t, 1.0, 0.001, 0.5)):
        ret, target = _batch(50, 0.3, cuda)
        xs = [ret["rgb_marched"], ret["rgb_marched0"], ret["alphainv_cum"]]
        g = torch.autograd.grad(f(ret, target), xs, create_graph=True)
        h = torch.autograd.grad(sum((v * v).sum() for v in g), xs)
        outs.append([*g, *h])
    for a, b in zip(*outs):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-9)


@pytest.mark.parametrize("how", ["strided", "float64", "target_grad", "vmap", "forward_mode"])
def test_other_callers_keep_the_chain(cuda, how, monkeypatch):
    """Inputs that the kernels do not take run as torch operations, as before."""
    monkeypatch.setattr(train._PhotoLoss, "apply", lambda *a: pytest.fail("the kernels took it"))
    ret, target = _batch(40, 0.3, cuda)
    want = _chain(ret, target, 1.0, 0.001, 0.5)
    if how == "strided":
        got = fine_loss({**ret, "rgb_marched": ret["rgb_marched"].t().contiguous().t()}, target)
    elif how == "float64":
        got = fine_loss({k: v.double() for k, v in ret.items()}, target.double()).float()
    elif how == "target_grad":
        t = target.clone().requires_grad_()
        got = fine_loss(ret, t)
        got.backward()
        assert t.grad is not None
    elif how == "vmap":
        det = {k: v.detach() for k, v in ret.items()}
        got = torch.func.vmap(lambda r: fine_loss({**det, "rgb_marched": r}, target))(det["rgb_marched"][None])[0]
    else:
        with torch.autograd.forward_ad.dual_level():
            x = torch.autograd.forward_ad.make_dual(ret["rgb_marched"].detach(), torch.ones_like(target))
            out = fine_loss({**{k: v.detach() for k, v in ret.items()}, "rgb_marched": x}, target)
            got, tangent = torch.autograd.forward_ad.unpack_dual(out)
            assert tangent is not None
    torch.testing.assert_close(got.detach(), want.detach(), rtol=1e-5, atol=0)
