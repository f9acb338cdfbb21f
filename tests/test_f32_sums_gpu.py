"""vx_mlp_f32_reduce where its loads change from floats to float4s: output
counts around the limit, row lengths and offsets that do not allow float4s, few
and many partials.  Integers, so that every order of the sum is exact."""
import pytest
import torch

from voxurf_gb300 import _abi
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 64), (1, 192), (1, 2044), (1, 2048), (32, 64), (31, 64), (192, 70), (64, 33)])
@pytest.mark.parametrize("n_part,pad,offset", [(1, 0, 0), (7, 4, 0), (152, 0, 4), (2047, 4, 1), (33, 1, 0)])
def test_sums_are_exact(cuda, n_part, pad, offset, rows, cols):
    ld = cols + pad
    g = torch.Generator().manual_seed(cols)
    buf = torch.randint(-3, 4, (offset + n_part * rows * ld,), generator=g).float().to(cuda)
    part = buf[offset:].view(n_part, rows, ld)
    out = torch.full((rows, cols + 1), 7.0, device=cuda)
    _abi._declare()
    job = _abi.MlpSumJob(part.data_ptr(), n_part, rows * ld, ld, rows, cols, ptr(out), cols + 1)
    _abi.call("vx_mlp_f32_reduce", (_abi.MlpSumJob * 1)(job), 1, stream_ptr(cuda))
    assert torch.equal(out[:, :cols].double(), part[:, :, :cols].double().sum(0))
    assert bool((out[:, cols] == 7).all())
