"""The split-operand backward GEMMs at the ends of FP32's range, against the
CUDA-core kernels (an odd row stride sends a call there) and 64 bits."""
import pytest
import torch

from test_f32_split_gpu import _err, _rowgemm, _rows, _wgrad
from voxurf_gb300 import _abi, _native
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


@pytest.mark.parametrize("where", [(0,), (1,), (0, 1), (0, 2), (1, 2)])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 1e30])
def test_plain_tiles_between_others(cuda, value, where):
    """A CTA that takes several 128-row tiles, with values that send some of
    them to the plain sums: those are the CUDA-core kernel's bits, the tiles
    before and after them and their column sums stay what they are without."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    M = 128 * (2 * sms + 5) + 77                 # three tiles on the first CTAs
    g = torch.Generator().manual_seed(7)
    A = torch.randn((M, 192), generator=g).to(cuda)
    Bt = (torch.randn((192, 192), generator=g) / 14).to(cuda)
    H = torch.randn((M, 192), generator=g).to(cuda)
    clean, _ = _rowgemm(_rows(A, 192), Bt, H)
    tiles = [w * sms + 3 for w in where]         # all on CTA 3
    for t in tiles:
        A[128 * t + 5, 17] = value
        H[128 * t + 5] = 0                       # the row itself stays out of the column sums
    split, sums = _rowgemm(_rows(A, 192), Bt, H)
    plain, plain_sums = _rowgemm(_rows(A, 193), Bt, H)
    special = torch.zeros(M, dtype=torch.bool, device=cuda)
    for t in tiles:
        special[128 * t:128 * (t + 1)] = True
    assert torch.equal(_bits(split[special]), _bits(plain[special]))
    assert torch.equal(_bits(split[~special]), _bits(clean[~special]))
    # up to 2 * sms * 128 + rows of |c| <= 6: each side's additions round
    assert bool(((sums.double().sum(0) - plain_sums.double().sum(0)).abs() <= 1e-6 * plain.abs().double().sum(0)).all())


def test_plain_tiles_do_not_depend_on_timing(cuda):
    """Large finite values: the column sums of a tile that is summed plainly
    are added in one order, its even rows, then its odd rows."""
    g = torch.Generator().manual_seed(8)
    A = torch.randn((39 * 128, 192), generator=g).to(cuda)
    A[::100, 3] = 1e12                           # one in every tile
    Bt = torch.randn((192, 192), generator=g).to(cuda)
    H = torch.randn(A.shape, generator=g).to(cuda)
    split, sums = _rowgemm(_rows(A, 192), Bt, H)
    plain, _ = _rowgemm(_rows(A, 193), Bt, H)
    assert torch.equal(_bits(split), _bits(plain))
    c = split.view(39, 64, 2, 192)
    want = torch.zeros((39, 2, 192), device=cuda)
    for r in range(64):
        want += c[:, r]
    assert torch.equal(sums[:39], want[:, 0] + want[:, 1])


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("mode", [1, 2])
def test_rowgemm_in_place(cuda, mode, special):
    """C over A, as the CUDA-core kernel allows: every row from its own values
    before the call."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    M = 128 * (sms + 3)
    g = torch.Generator().manual_seed(9)
    A = torch.randint(-3, 4, (M, 192), generator=g).float().to(cuda)
    Bt = torch.randint(-3, 4, (192, 192), generator=g).float().to(cuda)
    H = torch.randint(-1, 2, (M, 192), generator=g).float().to(cuda)
    if special:
        A[::200, 9] = float("inf")
        Bt[9] = Bt[9].abs() + 1                  # infinite rows, no NaN
    want, _ = _rowgemm(_rows(A, 193), Bt, H if mode == 1 else None)
    colsum = torch.empty((int(_native.load().vx_mlp_f32_rowgemm_grid(M)), 192), device=cuda)
    a = _abi.MlpF32RowGemmArgs()
    a.M, a.K, a.A, a.lda, a.Bt, a.Np, a.mode = M, 192, ptr(A), 192, ptr(Bt), 192, mode
    a.H, a.ldh, a.C, a.ldc, a.n_store, a.colsum, a.colsum_cap = ptr(H), 192, ptr(A), 192, 192, ptr(colsum), colsum.numel()
    _abi.call_struct("vx_mlp_f32_rowgemm", a, stream_ptr(cuda))
    assert torch.equal(_bits(A), _bits(want))
