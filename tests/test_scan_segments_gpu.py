"""alpha2weight's segment search at sizes around its powers of 16, and its
scans at the lengths where the number of chunks in flight changes, against the
C restatement of render_utils_kernel.cu:577-707."""
import numpy as np
import pytest
import torch

from oracle import cref
from voxurf_gb300 import render_utils_cuda as ru

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


@pytest.mark.parametrize("n_pts", [1, 15, 16, 17, 255, 256, 257, 4095, 4096, 4097, 70_001])
@pytest.mark.parametrize("rays", [1, 40, 3000])
def test_segment_bounds(cuda, n_pts, rays):
    rng = np.random.default_rng(n_pts + rays)
    ray_id = np.sort(rng.integers(0, rays, n_pts))
    alpha = np.zeros(n_pts, np.float32)
    _, _, _, i0, i1 = ru.alpha2weight(torch.from_numpy(alpha).to(cuda), torch.from_numpy(ray_id).to(cuda), rays)
    beg, end = (np.searchsorted(ray_id, np.arange(rays), side) for side in ("left", "right"))
    empty = beg == end
    assert np.array_equal(i0.cpu().numpy(), np.where(empty, 0, beg))
    assert np.array_equal(i1.cpu().numpy(), np.where(empty, 0, end))


@pytest.mark.parametrize("stop_at", [None, 0, 31, 32, 62])
def test_short_segments(cuda, stop_at):
    rng = np.random.default_rng(3)
    lens = np.array([1, 5, 31, 32, 33, 63, 64, 65, 95, 96, 97, 0, 2])
    ray_id = np.repeat(np.arange(lens.size), lens)
    alpha = rng.uniform(0, 0.02, ray_id.size).astype(np.float32)
    if stop_at is not None:
        first = np.cumsum(lens) - lens
        alpha[(first + stop_at)[lens > stop_at]] = 0.9999
    gw, gl = rng.normal(size=alpha.size).astype(np.float32), rng.normal(size=lens.size).astype(np.float32)
    to = lambda x: torch.from_numpy(x).to(cuda)
    out = ru.alpha2weight(to(alpha), to(ray_id), lens.size)
    ref = cref.alpha2weight(alpha, ray_id, lens.size)
    # a factor, five scan levels and up to three carries more than the serial loop's roundings
    for got, want in zip(out[:3], ref[:3]):
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=2 * (97 + 9) * EPS, atol=0)
    assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip(out[3:], ref[3:]))
    g = ru.alpha2weight_backward(to(alpha), *out, lens.size, to(gw), to(gl)).cpu().numpy()
    want = cref.alpha2weight_backward(alpha, *ref, lens.size, gw, gl)
    # both sum at most 97 terms of |gw w| <= 0.1 and one of 5 after |gl last|, over 1 - alpha
    scale = np.abs(gw) + (np.abs(gl)[ray_id] + 97 * 0.1 + 5) / (1 - alpha + 1e-10)
    assert np.all(np.abs(g - want) <= 4 * (97 + 12) * EPS * scale)
