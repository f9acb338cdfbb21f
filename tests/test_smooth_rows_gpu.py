"""The two smoothing kernels sum the same products in the same order: large
grids of aligned float4 rows (the row kernel) against the same values in a
buffer that starts off a 16-byte boundary (the tile kernel), bit for bit."""
import numpy as np
import pytest
import torch

from voxurf_gb300 import _abi
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu

# y tiles of 4 and 16, z tiles of 128, short axes, chunks of x
SHAPES = [(129, 131, 132), (5, 421, 1000), (420, 5, 1004), (330, 637, 12), (133, 128, 124), (9, 130, 2052)]


def _smooth(adjoint, src, taps, into=None):
    X, Y, Z = src.shape
    out = torch.empty_like(src) if into is None else into
    args = [ptr(src), ptr(out), None, None, X, Y, Z, taps.ctypes.data, len(taps)]
    if adjoint:
        _abi.call("vx_smooth3d_adjoint", *args, int(into is not None), stream_ptr())
    else:
        _abi.call("vx_smooth3d", *args, stream_ptr())
    return out


@pytest.mark.parametrize("k", [1, 3, 5])
@pytest.mark.parametrize("shape", SHAPES)
def test_row_kernel_equals_tile_kernel(cuda, shape, k):
    X, Y, Z = shape
    assert X * Y * Z >= 128 ** 3 and Z % 4 == 0
    g = torch.Generator().manual_seed(k)
    src = torch.randn(shape, generator=g).to(cuda)
    off = torch.empty(X * Y * Z + 1, device=cuda)[1:].view(shape)     # 4 bytes past a 16-byte boundary
    off.copy_(src)
    taps = np.linspace(0.1, 0.7, k).astype(np.float32)                # not symmetric
    assert torch.equal(_smooth(False, src, taps), _smooth(False, off, taps))
    assert torch.equal(_smooth(True, src, taps), _smooth(True, off, taps))
    base = torch.randn(shape, generator=g).to(cuda)
    other = torch.empty(X * Y * Z + 1, device=cuda)[1:].view(shape)
    other.copy_(base)
    assert torch.equal(_smooth(True, src, taps, base), _smooth(True, off, taps, other))
