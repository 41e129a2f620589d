"""The pre-sorted QR (k_qrb, src/greens.c:119-146) through the calc_eq_g seam:
N where the panel's rows per lane and warps, the 8-column panels and row tiles
and the shared-memory form end, and factors whose columns are zero below the
diagonal (reflectors with tau = 0), real and complex.

Three factors with singular values in about [0.1, 1.7]: the dense FP64 inverse
and the seam's chain both round at a few N eps times the condition numbers,
below 1e-11 for N <= 256; 1e-10 as the other calc_eq_g tests require.  Diagonal
factors are exact up to a few roundings: 1e-14 relative to G <= 1.
"""
import numpy as np
import pytest

from test_gpu_recombine import _call

pytestmark = pytest.mark.gpu


def _random(shape, cplx, seed):
    r = np.random.RandomState(seed)
    a = r.standard_normal(shape)
    return a + 1j * r.standard_normal(shape) if cplx else a


@pytest.mark.parametrize("cplx,N", [(0, 2), (0, 15), (0, 16), (0, 17), (0, 32), (0, 96), (0, 97), (0, 160), (0, 163),
                                    (0, 164), (0, 193), (0, 225), (0, 256), (1, 2), (1, 15), (1, 17), (1, 33),
                                    (1, 65), (1, 112), (1, 118), (1, 130), (1, 225), (1, 256)])
def test_three_factors(cplx, N):
    pytest.importorskip("torch")
    C = 0.8 * np.eye(N) + 0.3 * _random((2, 3, N, N), cplx, N) / np.sqrt(N)
    rc, G, ph = _call(C)
    assert rc == 0
    for b in range(2):
        A = np.eye(N) + C[b, 2] @ C[b, 1] @ C[b, 0]
        assert np.max(np.abs(G[b] - np.linalg.inv(A))) < 1e-10
        assert abs(ph[b] - np.linalg.slogdet(A)[0]) < 1e-10


@pytest.mark.parametrize("cplx,N", [(0, 9), (0, 64), (0, 144), (0, 200), (1, 9), (1, 100), (1, 150)])
def test_diagonal_factors(cplx, N):
    pytest.importorskip("torch")
    d = np.exp(_random((1, 3, N), 0, N))
    C = np.zeros((1, 3, N, N), dtype=complex if cplx else float)
    C[..., np.arange(N), np.arange(N)] = d
    rc, G, _ = _call(C)
    assert rc == 0
    assert np.max(np.abs(G[0] - np.diag(1 / (1 + d[0].prod(0))))) < 1e-14


@pytest.mark.parametrize("cplx,lo,hi", [(0, 140, 168), (1, 92, 124)])
def test_every_size_where_the_matrix_leaves_one_sm(cplx, lo, hi):
    pytest.importorskip("torch")
    for N in range(lo, hi):
        C = 0.8 * np.eye(N) + 0.3 * _random((1, 2, N, N), cplx, N) / np.sqrt(N)
        rc, G, _ = _call(C)
        assert rc == 0, N
        assert np.max(np.abs(G[0] - np.linalg.inv(np.eye(N) + C[0, 1] @ C[0, 0]))) < 1e-10, N
