"""The FP32 MLP engine's GEMM kernels at the edges of their tiles.

Operands are small integers, so every product and every partial sum is exact in
FP32 (|sum| < 2^24) and the results must equal the integer result bit for bit,
whatever the order of the sums: a dropped, doubled or misplaced term shows."""
import pytest
import torch

from voxurf_gb300 import _abi, _native
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _ints(shape, lo, hi, seed, dev):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(lo, hi + 1, shape, generator=g).float().to(dev)


def _strided(rows, ld, dev):
    """rows [M, K] as the leading columns of a NaN-filled [M, ld] buffer."""
    buf = torch.full((rows.shape[0], ld), float("nan"), device=dev)
    buf[:, :rows.shape[1]] = rows
    return buf


def _grid(lib, M):
    return int(lib.vx_mlp_f32_rowgemm_grid(M))


@pytest.mark.parametrize("M", [1, 63, 64, 65, 127, 128, 129, 1000, 152 * 128 + 1])
@pytest.mark.parametrize("K,Np,n_store,pad", [(70, 192, 192, 2), (192, 192, 192, 0), (192, 80, 70, 2), (192, 64, 60, 1),
                                              (128, 128, 128, 0), (128, 80, 75, 1), (64, 64, 64, 0), (32, 32, 32, 0),
                                              (80, 80, 80, 0), (192, 192, 192, 3)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_rowgemm_is_exact_on_integers(cuda, mode, K, Np, n_store, pad, M):
    if mode == 1 and n_store != Np:
        pytest.skip("hidden layers store every column")
    lib = _native.load()
    _abi._declare()
    A = _strided(_ints((M, K), -3, 3, 1, cuda), K + pad, cuda)
    Kp = (K + 15) // 16 * 16
    Bt = torch.zeros((Kp, Np), device=cuda)
    Bt[:K, :n_store] = _ints((K, n_store), -3, 3, 2, cuda)
    H = _strided(_ints((M, Np), -1, 1, 3, cuda), Np + pad, cuda)
    bias = _ints((Np,), -5, 5, 4, cuda)
    C = torch.full((M, n_store + pad), 7.0, device=cuda)
    colsum = torch.full((_grid(lib, M) * Np,), float("nan"), device=cuda)
    live = torch.tensor([max(1, M - 5)], device=cuda) if M > 64 else None
    g = _abi.MlpF32RowGemmArgs()
    g.M, g.m_dev, g.K, g.A, g.lda = M, ptr(live), K, ptr(A), A.stride(0)
    g.Bt, g.Np, g.mode, g.bias = ptr(Bt), Np, mode, ptr(bias)
    g.H, g.ldh, g.C, g.ldc, g.n_store = ptr(H), H.stride(0), ptr(C), C.stride(0), n_store
    g.colsum, g.colsum_cap = ptr(colsum), colsum.numel()
    _abi.call_struct("vx_mlp_f32_rowgemm", g, stream_ptr(cuda))
    m = M if live is None else int(live)
    # float64 products of small integers are exact
    ref = A[:m, :K].double() @ Bt[:K].double()
    if mode == 0:
        ref = (ref + bias.double()).clamp(min=0)
    elif mode == 1:
        ref = ref * (H[:m, :Np] > 0)
        assert torch.equal(colsum.view(-1, Np).double().sum(0), ref.sum(0))
        assert bool((colsum.view(-1, Np)[int(lib.vx_mlp_f32_colsum_rows(g)):] == 0).all())
    assert torch.equal(C[:m, :n_store].double(), ref[:, :n_store])
    assert bool((C[m:] == 7).all()) and bool((C[:, n_store:] == 7).all())
    assert _native.device_error(stream_ptr(cuda)) == 0
