"""The rule that sends a grid to the row kernel of the smoothing, at its edges:
z extents on both sides of each limit, against the same values off a 16-byte
boundary (the tile kernel), bit for bit."""
import numpy as np
import pytest
import torch

from voxurf_gb300 import _abi
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _smooth(name, src, taps, *more):
    out = torch.empty_like(src)
    _abi.call(name, ptr(src), ptr(out), None, None, *src.shape, taps.ctypes.data, len(taps), *more, stream_ptr())
    return out


@pytest.mark.parametrize("X,Y,Z", [(270, 251, 32), (270, 251, 36), (190, 181, 64), (190, 181, 68), (130, 127, 128),
                                   (133, 127, 132), (161, 151, 132), (150, 131, 160), (117, 113, 164)])
@pytest.mark.parametrize("k", [1, 3, 5])
def test_rule_edges(cuda, X, Y, Z, k):
    src = torch.randn((X, Y, Z), generator=torch.Generator().manual_seed(Z)).to(cuda)
    off = torch.empty(src.numel() + 1, device=cuda)[1:].view(src.shape)
    off.copy_(src)
    taps = np.linspace(0.1, 0.7, k).astype(np.float32)
    assert torch.equal(_smooth("vx_smooth3d", src, taps), _smooth("vx_smooth3d", off, taps))
    adj = [_smooth("vx_smooth3d_adjoint", x, taps, 0) for x in (src, off)]
    assert torch.equal(*adj)
