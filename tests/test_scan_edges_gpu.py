"""alpha2weight and its backward at the edges of their chunks: segment
lengths around the 32-sample scans, the 128-sample steps and the
512-sample switch of the accumulator, empty segments, and stops in the first
and last lanes of a scan (render_utils_kernel.cu:577-707 in 64 bits)."""
import numpy as np
import pytest
import torch

from voxurf_gb300 import render_utils_cuda as ru

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24
LENGTHS = (1, 31, 32, 33, 127, 128, 129, 256, 511, 512, 513, 640, 1025, 2303)


def _exact(alpha, gw, glast):
    """One segment in 64 bits: w, T, last, samples up to the stop, gradient."""
    a = alpha.astype(np.float64)
    incl = np.cumprod(1 - a)
    hit = np.nonzero(incl < 1e-3)[0]
    n = int(hit[0]) + 1 if hit.size else a.size
    T = np.ones_like(a)
    T[:n] = np.concatenate([[1.0], incl[:n - 1]])
    w = np.where(np.arange(a.size) < n, T * a, 0.0)
    last = incl[n - 1]
    t = gw[:n] * w[:n]
    back = glast * last + (np.cumsum(t[::-1])[::-1] - t)
    g = np.zeros_like(a)
    g[:n] = gw[:n] * T[:n] - back / (1 - a[:n] + 1e-10)
    mag = np.zeros_like(a)     # what the gradient's roundings scale with
    mag[:n] = np.abs(gw[:n] * T[:n]) + (abs(glast) * last + np.sum(np.abs(t))) / (1 - a[:n] + 1e-10)
    return w, T, last, n, g, mag


@pytest.mark.parametrize("stop_at", [None, 0, 31, 32, 127, 128, 300, 600])
def test_scan_edges_match_64_bits(cuda, stop_at):
    rng = np.random.default_rng(17)
    lens, segs = [], []
    for n in LENGTHS:
        a = rng.uniform(0, 1.5 / max(n, 8), size=n).astype(np.float32)
        if stop_at is not None and stop_at < n:
            a[stop_at] = 0.9999
        segs += [a, np.zeros(0, np.float32)]
        lens += [n, 0]
    ray_id = np.repeat(np.arange(len(lens), dtype=np.int64), lens)
    alpha = np.concatenate(segs)
    gw = rng.normal(size=alpha.size).astype(np.float32)
    gl = rng.normal(size=len(lens)).astype(np.float32)
    to = lambda x: torch.from_numpy(x).to(cuda)
    w, T, last, i0, i1 = ru.alpha2weight(to(alpha), to(ray_id), len(lens))
    g = ru.alpha2weight_backward(to(alpha), w, T, last, i0, i1, len(lens), to(gw), to(gl))
    w, T, last, i0, i1, g = [x.cpu().numpy() for x in (w, T, last, i0, i1, g)]
    at = 0
    for r, n in enumerate(lens):
        if n == 0:
            assert (i0[r], i1[r], last[r]) == (0, 0, 1.0)
            continue
        ew, eT, el, live, eg, mag = _exact(segs[r], gw[at:at + n].astype(np.float64), float(gl[r]))
        s = slice(at, at + n)
        assert (i0[r], i1[r]) == (at, at + live), (n, stop_at)
        # FP32: every factor and every product on the way rounds once (n factors,
        # five scan levels, n / 32 carries, the weight); the pair: the last roundings
        k = 3 if n > 512 else n + 5 + n // 32 + 3
        np.testing.assert_allclose(T[s], eT, rtol=k * EPS, atol=0)
        np.testing.assert_allclose(w[s], ew, rtol=(k + 1) * EPS, atol=0)
        assert abs(last[r] - el) <= k * EPS * abs(el)
        # the gradient is formed from the rounded w and T above, and in FP32 its
        # suffix sums and its quotient round on the way too
        assert np.all(np.abs(g[s] - eg) <= (2 * k + 8) * EPS * mag)
        at += n
