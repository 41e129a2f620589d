"""The GEMM seam at sizes that take each of its tiles (16, 32, 40, 48, 56, 64:
by the number of matrices, then by padded area), on both sides of the lines
between them, with remainders in every dimension, against torch float64
matmul: relative error within a small multiple of K eps, as each entry is a
chain of K products."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [0, 1])
@pytest.mark.parametrize("M,N,K,batch", [
    (1, 1, 1, 1), (15, 17, 33, 3), (64, 64, 64, 64), (64, 64, 64, 65), (100, 100, 100, 40), (100, 99, 101, 90),
    (75, 75, 75, 130), (80, 40, 31, 160), (111, 57, 40, 130), (144, 143, 145, 70), (128, 64, 70, 140),
    (33, 31, 300, 700)])
def test_gemm_tiles_match_torch(cplx, M, N, K, batch):
    torch = pytest.importorskip("torch")
    from dqmc_b200 import lib
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 13 * K + cplx)
    dt = torch.complex128 if cplx else torch.float64
    A = torch.randn(batch, K, M, dtype=dt, device="cuda", generator=g)
    B = torch.randn(batch, N, K, dtype=dt, device="cuda", generator=g)
    Cm = torch.randn(batch, N, M, dtype=dt, device="cuda", generator=g)
    nt = np.complex128 if cplx else np.float64
    alpha, beta = np.array([1.25], nt), np.array([-0.5], nt)
    ref = 1.25 * (B @ A) - 0.5 * Cm
    rc = lib.load().dqmc_gpu_gemm(batch, M, N, K, cplx, alpha.ctypes.data, A.data_ptr(), M,
                                  C.c_longlong(M * K), B.data_ptr(), K, C.c_longlong(K * N), beta.ctypes.data,
                                  Cm.data_ptr(), M, C.c_longlong(M * N), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert (Cm - ref).abs().max().item() < 50 * K * 2.2e-16 * max(1.0, ref.abs().max().item())
