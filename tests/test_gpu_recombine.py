"""The recombine's blocked LU and its solves (k_recb, src/greens.c:157-207)
through the calc_eq_g seam against a dense inverse, at the sizes where its
tiles, panels and row slots end: N below, at and past 8-row tiles, one and four
panel warps, one and two rows a lane, leading dimension equal to N, matrices in
shared and in global memory, real and complex, several items.

C = two random factors with singular values of I + C_1 C_0 in about [0.1, 10]:
the dense FP64 inverse and the seam's chain (two factorisations, two products,
an LU) both round at a few N eps times the condition number, below 1e-11 for
N <= 256; 1e-10 as the other calc_eq_g tests require.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G_TOL = 1e-10


def _call(C, l=0):
    import torch
    from dqmc_b200 import lib
    nb, F, N, _ = C.shape
    dC = torch.from_numpy(np.ascontiguousarray(C.swapaxes(-1, -2))).cuda()
    dG = torch.zeros(nb, N, N, dtype=dC.dtype, device="cuda")
    ph = torch.zeros(nb, dtype=dC.dtype, device="cuda")
    rc = lib.load().dqmc_gpu_calc_eq_g(nb, N, F, l, int(C.dtype.kind == "c"), dC.data_ptr(), dG.data_ptr(),
                                       ph.data_ptr(), None)
    return rc, dG.cpu().numpy().swapaxes(-1, -2), ph.cpu().numpy()


def _factors(N, nb, cplx, seed):
    r = np.random.RandomState(seed)
    a = r.standard_normal((nb, 2, N, N))
    if cplx:
        a = a + 1j * r.standard_normal((nb, 2, N, N))
    return 0.8 * np.eye(N) + 0.4 * a / np.sqrt(N)


@pytest.mark.parametrize("cplx,N,nb", [(0, 1, 2), (0, 7, 3), (0, 8, 1), (0, 9, 2), (0, 31, 1), (0, 33, 2), (0, 64, 2),
                                       (0, 65, 1), (0, 100, 2), (0, 128, 1), (0, 129, 1), (0, 144, 3), (0, 161, 1),
                                       (0, 255, 1), (1, 5, 2), (1, 36, 1), (1, 97, 1), (1, 100, 2), (1, 129, 1),
                                       (1, 200, 1)])
def test_matches_dense_inverse(cplx, N, nb):
    pytest.importorskip("torch")
    C = _factors(N, nb, cplx, 3 * N + cplx)
    rc, G, ph = _call(C)
    assert rc == 0
    for b in range(nb):
        A = np.eye(N) + C[b, 1] @ C[b, 0]
        assert np.max(np.abs(G[b] - np.linalg.inv(A))) < G_TOL
        assert abs(ph[b] - np.linalg.slogdet(A)[0]) < 1e-10


@pytest.mark.parametrize("cplx,N", [(0, 20), (0, 144), (1, 50)])
def test_bad_values_are_reported(cplx, N):
    """A NaN in one item sets the error status and leaves the other items."""
    pytest.importorskip("torch")
    C = _factors(N, 2, cplx, 9)
    good = C[1].copy()
    C[0, 1, N // 2, N // 3] = np.nan
    rc, G, _ = _call(C)
    assert rc == -13
    assert np.max(np.abs(G[1] - np.linalg.inv(np.eye(N) + good[1] @ good[0]))) < G_TOL
