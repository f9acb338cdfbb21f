"""Exclusive scans at the edges of the one-launch kernel (steps of 8192 counts,
at most 32768) and of the tiled one beyond it."""
import pytest
import torch

from voxurf_gb300 import _native
from voxurf_gb300._torch import ptr, scratch, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,name", [(torch.int32, "vx_exclusive_scan_i32"), (torch.int64, "vx_exclusive_scan_i64")])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 8191, 8192, 8193, 16385, 32767, 32768, 32769, 70001])
def test_scan_equals_cumsum(cuda, n, dtype, name):
    v = torch.randint(0, 1000, (n,), generator=torch.Generator().manual_seed(n)).to(cuda, dtype)
    out = torch.full((n + 2,), -7, dtype=torch.int64, device=cuda)
    nb = _native.load().vx_scan_scratch_bytes(n)
    tmp = scratch(nb, cuda)
    _native.call(name, ptr(v), n, ptr(out), ptr(tmp), nb, stream_ptr(cuda))
    assert int(out[0]) == 0 and int(out[n + 1]) == -7
    assert torch.equal(out[1:n + 1], torch.cumsum(v.long(), 0))
