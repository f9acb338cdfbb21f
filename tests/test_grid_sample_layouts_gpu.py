"""DenseGrid lookups in the float4 layout (channel-last, C % 4 == 0) against the
scalar kernels, which serve channel-first grids and unaligned buffers.

The corner order and weights are the same in both, so forward values are equal
bit for bit.  For the gradient the points lie on a dyadic lattice and the
upstream gradients are small integers: every contribution and every partial sum
is exact in FP32, whatever the order of the reductions."""
import pytest
import torch

from voxurf_gb300.grid import DenseGrid

pytestmark = pytest.mark.gpu

BOX = ([-1.0, -1.0, -1.0], [1.0, 1.0, 1.0])


def _pair(C, shape, cuda):
    """The same grid channel-last (float4 kernels) and channel-first (scalar)."""
    a = DenseGrid(C, shape, *BOX).to(cuda)
    b = DenseGrid(C, shape, *BOX, channel_last=False).to(cuda)
    with torch.no_grad():
        v = torch.randn(a.grid.shape, generator=torch.Generator().manual_seed(C)).to(cuda)
        a.grid.copy_(v)
        b.grid.copy_(v)
    assert a.grid.stride() != b.grid.stride()
    return a, b


@pytest.mark.parametrize("n", [0, 1, 85, 86, 4099])
@pytest.mark.parametrize("C", [4, 12, 20])
def test_float4_forward_equals_scalar(cuda, C, n):
    a, b = _pair(C, (17, 9, 33), cuda)
    # some points outside the box, on its faces and on grid points
    pts = 2.4 * torch.rand((n, 3), generator=torch.Generator().manual_seed(n)) - 1.2
    pts[:n // 3] = (pts[:n // 3] * 8).round() / 8
    with torch.no_grad():
        assert torch.equal(a(pts.to(cuda)), b(pts.to(cuda)))


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("C,n", [(4, 1), (12, 85), (12, 4099), (20, 333)])
def test_float4_gradient_is_exact(cuda, C, n, offset):
    a, b = _pair(C, (17, 9, 33), cuda)
    g = torch.Generator().manual_seed(3)
    pts = (torch.randint(-18, 19, (n, 3), generator=g).float() / 16).to(cuda)   # half and quarter voxels
    buf = torch.randint(-4, 5, (n * C + 1,), generator=g).float().to(cuda)
    up = buf[offset:offset + n * C].view(n, C)     # offset 1: rows that are not 16-byte aligned
    for net in (a, b):
        net(pts).backward(up)
    assert torch.equal(a.grid.grad, b.grid.grad)
    assert float(a.grid.grad.abs().sum()) > 0
