"""The FP32 MLP backward's split-operand tensor-core GEMMs against 64 bits and
against the CUDA-core kernels, which take the calls whose rows are not aligned
for them (an odd row stride): no less exact, and the same values where an
operand has no BF16 parts (infinite, NaN, or beyond BF16's rounding range)."""
import pytest
import torch

from voxurf_gb300 import _abi, _native
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _rows(x, ld):
    buf = torch.zeros((x.shape[0], ld), device=x.device)
    buf[:, :x.shape[1]] = x
    return buf[:, :x.shape[1]]


def _rowgemm(A, Bt, H=None, n_store=None):
    M, K = A.shape
    Np = Bt.shape[1]
    n = Np if n_store is None else n_store
    C = torch.empty((M, Np), device=A.device)
    rows = int(_native.load().vx_mlp_f32_rowgemm_grid(M))
    colsum = torch.empty((rows, Np), device=A.device)
    g = _abi.MlpF32RowGemmArgs()
    g.M, g.K, g.A, g.lda = M, K, ptr(A), A.stride(0)
    g.Bt, g.Np, g.mode = ptr(Bt), Np, 2 if H is None else 1
    g.H, g.ldh, g.C, g.ldc, g.n_store = ptr(H), 0 if H is None else H.stride(0), ptr(C), C.stride(0), n
    g.colsum, g.colsum_cap = ptr(colsum), colsum.numel()
    _abi.call_struct("vx_mlp_f32_rowgemm", g, stream_ptr(A.device))
    assert _native.device_error(stream_ptr(A.device)) == 0
    return C, colsum


def _wgrad(A, B, MP, NP):
    rows, M = A.shape
    N = B.shape[1]
    grid = int(_native.load().vx_mlp_f32_wgrad_grid(rows))
    part = torch.full((grid, MP, NP), float("nan"), device=A.device)
    g = _abi.MlpF32WgradArgs()
    g.rows, g.A, g.lda, g.B, g.ldb = rows, ptr(A), A.stride(0), ptr(B), B.stride(0)
    g.M, g.N, g.part, g.part_cap = M, N, ptr(part), part.numel()
    _abi.call_struct("vx_mlp_f32_wgrad", g, stream_ptr(A.device))
    assert _native.device_error(stream_ptr(A.device)) == 0
    return part[:, :M, :N]


def _gradients(M, K, seed, dev):
    """Rows as a backward pass has them: magnitudes over six decades, and a
    third of the values zero (behind a ReLU)."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn((M, K), generator=g) * torch.exp(torch.empty((M, 1)).uniform_(-14, 0, generator=g))
    return (x * (torch.rand((M, K), generator=g) > 0.33)).to(dev)


def _err(x, ref):
    return float((x.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("K,Np", [(192, 192), (192, 80), (128, 128), (128, 64)])
def test_rowgemm_no_less_exact_than_cuda_cores(cuda, K, Np):
    A = _gradients(20_000, K, 1, cuda)
    Bt = (torch.randn((K, Np), generator=torch.Generator().manual_seed(2)) / K ** 0.5).to(cuda)
    H = torch.randn((A.shape[0], Np), generator=torch.Generator().manual_seed(3)).to(cuda) if K == Np else None
    ref = A.double() @ Bt.double()
    ref = ref if H is None else ref * (H > 0)
    split, sums = _rowgemm(_rows(A, K + 4), Bt, H)
    plain, plain_sums = _rowgemm(_rows(A, K + 1), Bt, H)
    assert not torch.equal(split, plain)          # two different kernels
    e = (_err(split, ref), _err(plain, ref))
    print(K, Np, "split %.3g plain %.3g" % e)
    assert e[0] <= e[1]
    # row by row too: the small rows are as exact as the large ones
    n = ref.norm(dim=1).clamp(min=1e-30)
    r = [((x.double() - ref).norm(dim=1) / n).quantile(0.99).item() for x in (split, plain)]
    assert r[0] <= 1.1 * r[1], r
    if H is not None:
        exact = ref.sum(0)
        e = [_err(x.double().sum(0), exact) for x in (sums, plain_sums)]
        assert e[0] <= max(e[1], 2.0 ** -22), e


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38, 1e-40])
@pytest.mark.parametrize("where", ["row", "weight"])
def test_rowgemm_values_without_parts(cuda, where, value):
    K = N = 192
    A = _gradients(400, K, 4, cuda)
    Bt = torch.randn((K, N), generator=torch.Generator().manual_seed(5)).to(cuda)
    H = torch.randn((400, N), generator=torch.Generator().manual_seed(6)).to(cuda)
    if where == "row":
        A[150, 7] = value
    else:
        Bt[7, 100] = value
    for h in (None, H):
        split, _ = _rowgemm(_rows(A, K), Bt, h)
        plain, _ = _rowgemm(_rows(A, K + 1), Bt, h)
        if abs(value) > 1:      # summed plainly: the same bits, in the tile (rows 128..255) or everywhere
            rows = slice(128, 256) if where == "row" else slice(None)
            assert torch.equal(split[rows].view(torch.int32), plain[rows].view(torch.int32))
        torch.testing.assert_close(split, plain, rtol=1e-4, atol=1e-5, equal_nan=True)


@pytest.mark.parametrize("M,N,NP", [(192, 192, 192), (192, 70, 80), (128, 128, 128), (128, 60, 64)])
def test_wgrad_no_less_exact_than_cuda_cores(cuda, M, N, NP):
    rows = 60_001
    A = _gradients(rows, M, 7, cuda)
    B = torch.randn((rows, N), generator=torch.Generator().manual_seed(8)).clamp(min=0).to(cuda)
    ref = A.double().t() @ B.double()
    split, plain = (_wgrad(_rows(A, M + p), _rows(B, (N + 3) // 4 * 4 + p), M, NP) for p in (0, 1))
    e = [_err(x.double().sum(0), ref) for x in (split, plain)]
    print(M, N, "split %.3g plain %.3g" % tuple(e))
    assert e[0] <= e[1]
    # and partial by partial (a CTA's own rows)
    per = -(-rows // split.shape[0])
    part = torch.stack([A[i * per:(i + 1) * per].double().t() @ B[i * per:(i + 1) * per].double()
                        for i in range(split.shape[0])])
    e = [_err(x, part) for x in (split, plain)]
    assert e[0] <= e[1]


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 127, 128, 129, 160, 255, 513, 152 * 256 + 7])
@pytest.mark.parametrize("M,N,NP", [(192, 192, 192), (192, 70, 80), (192, 64, 64), (128, 128, 128), (128, 75, 80),
                                    (128, 60, 64), (64, 64, 64)])
def test_wgrad_is_exact_on_integers(cuda, M, N, NP, rows):
    g = torch.Generator().manual_seed(rows)
    A = torch.randint(-3, 4, (rows, M), generator=g).float().to(cuda)
    B = torch.randint(-3, 4, (rows, N), generator=g).float().to(cuda)
    for pad in (0, 1):
        got = _wgrad(_rows(A, M + pad), _rows(B, (N + 3) // 4 * 4 + pad), M, NP)
        assert torch.equal(got.double().sum(0), A.double().t() @ B.double())


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.0e38])
@pytest.mark.parametrize("where", ["A", "B"])
def test_wgrad_values_without_parts(cuda, where, value):
    A = _gradients(700, 192, 9, cuda)
    B = torch.randn((700, 192), generator=torch.Generator().manual_seed(10)).to(cuda)
    (A if where == "A" else B)[300, 100] = value
    split, plain = (_wgrad(_rows(A, 192 + p), _rows(B, 192 + p), 192, 192) for p in (0, 1))
    i = 300 // -(-700 // split.shape[0])          # the CTA whose rows hold it (and its column half for B)
    cols = slice(96, 192) if where == "B" else slice(None)
    assert torch.equal(split[i][:, cols].view(torch.int32), plain[i][:, cols].view(torch.int32))
    torch.testing.assert_close(split, plain, rtol=1e-4, atol=1e-4, equal_nan=True)


@pytest.mark.parametrize("offset", [0, 4, 8])
def test_wgrad_partials_within_a_buffer(cuda, offset):
    """Partials that start 16 but not 32 bytes into a sector are summed on the
    CUDA cores (the tensor-core kernel stores whole sectors): exact either way,
    and nothing beside them is written."""
    rows, W = 1000, 192
    g = torch.Generator().manual_seed(offset)
    A, B = (torch.randint(-3, 4, (rows, W), generator=g).float().to(cuda) for _ in range(2))
    grid = int(_native.load().vx_mlp_f32_wgrad_grid(rows))
    buf = torch.full((offset + grid * W * W + 8,), 7.0, device=cuda)
    part = buf[offset:offset + grid * W * W]
    a = _abi.MlpF32WgradArgs()
    a.A, a.lda, a.B, a.ldb, a.M, a.N, a.rows = ptr(A), W, ptr(B), W, W, W, rows
    a.part, a.part_cap = part.data_ptr(), part.numel()
    _abi.call_struct("vx_mlp_f32_wgrad", a, stream_ptr(cuda))
    assert torch.equal(part.view(grid, W, W).double().sum(0), A.double().t() @ B.double())
    assert (buf[:offset] == 7).all() and (buf[-8:] == 7).all()
