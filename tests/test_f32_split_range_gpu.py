"""The split-operand backward GEMMs at the ends of FP32's range, against the
CUDA-core kernels (an odd row stride sends a call there) and 64 bits."""
import pytest
import torch

from test_f32_split_gpu import _err, _rowgemm, _rows, _wgrad
from voxurf_gb300 import _abi
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _bits(x):
    return x.view(torch.int32)


# products that overflow although each operand is far from it, with both signs
# of the parts after the first (1.003 and 0.999 round down and up to BF16)
@pytest.mark.parametrize("a,b", [(1.003e25, 1.003e25), (0.999e25, 1.003e25), (1.003e25, -0.999e25), (3e19, 3e19),
                                 (1.003e30, 1.003e12)])
def test_products_that_overflow(cuda, a, b):
    n = 400
    A = torch.randn((n, 192), generator=torch.Generator().manual_seed(0)).to(cuda)
    B = torch.randn((n, 192), generator=torch.Generator().manual_seed(1)).to(cuda)
    A[150, 7], B[150, 20] = a, b
    split, plain = (_wgrad(_rows(A, 192 + p), _rows(B, 192 + p), 192, 192) for p in (0, 1))
    torch.testing.assert_close(split, plain, rtol=1e-4, atol=1e-4 * max(abs(a), abs(b)))
    big = ~plain.isfinite()
    assert torch.equal(_bits(split)[big], _bits(plain)[big]) and not split.isnan().any()
    Bt = torch.randn((192, 192), generator=torch.Generator().manual_seed(2)).to(cuda)
    Bt[7, 100] = b
    split, plain = (_rowgemm(_rows(A, 192 + p), Bt)[0] for p in (0, 1))
    big = ~plain.isfinite()
    assert torch.equal(_bits(split)[big], _bits(plain)[big]) and not split.isnan().any()
    # every other sum: rounding of its largest products
    scale = A.abs().double() @ Bt.abs().double()
    assert bool(((split.double() - plain.double()).abs()[~big] <= 192 * 2.0 ** -23 * scale[~big]).all())


@pytest.mark.parametrize("a,b", [(1e-36, 1.0), (1.0, 1e-36), (3e-34, 1.0), (1e-30, 1e-3), (1e-20, 1e-17)])
def test_tiny_operands_no_less_exact_than_cuda_cores(cuda, a, b):
    """Values whose second and third BF16 parts would be below BF16's range."""
    g = torch.Generator().manual_seed(4)
    A = (a * torch.randn((3000, 192), generator=g)).to(cuda)
    Bt = (b / 14 * torch.randn((192, 192), generator=g)).to(cuda)
    split, plain = (_rowgemm(_rows(A, 192 + p), Bt)[0] for p in (0, 1))
    ref = A.double() @ Bt.double()
    e = _err(split, ref), _err(plain, ref)
    print("rows %.3g %.3g" % e)
    assert e[0] <= e[1]
    B = (b * torch.randn((3000, 192), generator=g)).to(cuda)
    split, plain = (_wgrad(_rows(A, 192 + p), _rows(B, 192 + p), 192, 192) for p in (0, 1))
    ref = A.double().t() @ B.double()
    e = [_err(x.double().sum(0), ref) for x in (split, plain)]
    print("wgrad %.3g %.3g" % tuple(e))
    assert e[0] <= e[1]


def test_tiny_rows_among_others(cuda):
    """Each row is as exact as its own magnitude asks, also beside larger ones."""
    g = torch.Generator().manual_seed(5)
    A = (torch.randn((4000, 192), generator=g) * 10.0 ** -torch.randint(0, 37, (4000, 1), generator=g)).to(cuda)
    Bt = (torch.randn((192, 192), generator=g) / 14).to(cuda)
    ref = A.double() @ Bt.double()
    r = [((x.double() - ref).norm(dim=1) / ref.norm(dim=1)).quantile(0.99).item()
         for x in (_rowgemm(_rows(A, 192 + p), Bt)[0] for p in (0, 1))]
    assert r[0] <= 1.1 * r[1], r


def _reduced(part):
    """The engine's own ordered sum of the partials."""
    grid, M, N = part.shape
    part, out = part.contiguous(), torch.empty((M, N), device=part.device)
    job = _abi.MlpSumJob(ptr(part), grid, M * N, N, M, N, ptr(out), N)
    _abi.call("vx_mlp_f32_reduce", (_abi.MlpSumJob * 1)(job), 1, stream_ptr(part.device))
    return out


@pytest.mark.parametrize("rows", [33, 65, 700, 60_001, 131_003])
@pytest.mark.parametrize("M,N,NP", [(192, 192, 192), (128, 60, 64)])
def test_wgrad_of_one_sign(cuda, M, N, NP, rows):
    """Products of one sign, whose sums truncation always leaves short: the
    gradient that the engine returns is as exact as the CUDA-core kernels'.
    (Both end in the same ordered FP32 sum of up to 152 partials, about 5e-8;
    a tenth is left for which way its roundings fall.)"""
    g = torch.Generator().manual_seed(rows)
    A, B = torch.rand((rows, M), generator=g).to(cuda), torch.rand((rows, N), generator=g).to(cuda)
    ref = A.double().t() @ B.double()
    e = [_err(_reduced(_wgrad(_rows(A, M + p), _rows(B, (N + 3) // 4 * 4 + p), M, NP)), ref) for p in (0, 1)]
    print(M, N, rows, "%.3g %.3g" % tuple(e))
    assert e[0] <= max(1.1 * e[1], 2.0 ** -24)


def test_rowgemm_of_one_sign(cuda):
    """Rows are more exact than the CUDA-core kernels' here too; their column
    sums keep the truncation of 8 and 4 MMAs: at most (4.5 * 2 / 3 + 2.5 / 3)
    units of 2^-23, half of it on average."""
    g = torch.Generator().manual_seed(6)
    A, Bt = torch.rand((60_001, 192), generator=g).to(cuda), torch.rand((192, 192), generator=g).to(cuda)
    H = torch.ones((A.shape[0], 192), device=cuda)
    ref = A.double() @ Bt.double()
    (split, sums), (plain, _) = (_rowgemm(_rows(A, 192 + p), Bt, H) for p in (0, 1))
    assert _err(split, ref) <= _err(plain, ref)
    assert _err(sums.double().sum(0), ref.sum(0)) <= 3.9 / 2 * 2.0 ** -23
