"""The 32-row tiles of the FP32 row GEMM (forward and input gradient of small
batches) against integers, at the row counts around the tiles and around the
one where 64-row tiles take over."""
import pytest
import torch

from voxurf_gb300 import _abi, _native
from voxurf_gb300._torch import ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("K,Np,pad", [(70, 192, 2), (39, 128, 1), (192, 80, 1), (64, 64, 0), (32, 32, 3)])
@pytest.mark.parametrize("tiles,extra", [(0, 1), (0, 31), (0, 32), (0, 33), (1, 0), (1, 1), (-1, -1), (-1, 0), (-1, 1)])
def test_small_tiles_are_exact_on_integers(cuda, tiles, extra, K, Np, pad, mode):
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    M = (64 * tiles if tiles >= 0 else 64 * (sms - 1)) + extra
    g = torch.Generator().manual_seed(M)
    ints = lambda *s: torch.randint(-3, 4, s, generator=g).float().to(cuda)
    A = torch.full((M, K + pad), float("nan"), device=cuda)
    A[:, :K] = ints(M, K)
    Bt = torch.zeros(((K + 15) // 16 * 16, Np), device=cuda)
    Bt[:K] = ints(K, Np)
    bias = ints(Np)
    C = torch.full((M + 1, Np), 7.0, device=cuda)
    a = _abi.MlpF32RowGemmArgs()
    a.M, a.K, a.A, a.lda, a.Bt, a.Np, a.mode, a.bias = M, K, ptr(A), K + pad, ptr(Bt), Np, mode, ptr(bias)
    a.C, a.ldc, a.n_store = ptr(C), Np, Np
    _abi.call_struct("vx_mlp_f32_rowgemm", a, stream_ptr(cuda))
    ref = A[:, :K].double() @ Bt[:K].double()
    ref = (ref + bias.double()).clamp(min=0) if mode == 0 else ref
    assert torch.equal(C[:M].double(), ref) and bool((C[M:] == 7).all())
    assert _native.device_error(stream_ptr(cuda)) == 0
