"""The delayed update in windows of 16 sites (k_update, k_update_cl) against
the oracle's update_delayed (src/updates.c:7-84) through the seam, at the sizes
where its splits end: N below, at and past a window, odd N (no 16-byte
columns), slabs of 8-column tiles with a short or empty last slab, both forms,
real and complex; delay ranks below and above a window's accepts.

Fields and RNG state must be equal.  G and the phase: both sides apply the
same N rank-1 updates to O(1) entries; each rounds its entries a few times per
update, so they agree to 1e-10 as the other tests of this seam require.
"""
import ctypes as C

import numpy as np
import pytest

from oracle_ctl import oracle_lib

pytestmark = pytest.mark.gpu

G_TOL = 1e-10


def _inputs(N, batch, cplx, seed):
    """fields and a well-conditioned G = (I + M)^-1 of both spins per chain"""
    r = np.random.RandomState(seed)
    nt = np.complex128 if cplx else np.float64
    a = r.standard_normal((batch, 2, N, N))
    if cplx:
        a = a + 1j * r.standard_normal((batch, 2, N, N))
    G = np.linalg.inv(np.eye(N) + np.eye(N) * 0.9 + 0.3 * a / np.sqrt(N)).astype(nt)
    el = np.exp(0.35)
    del_ = np.tile(np.concatenate([np.full(N, el ** 2 - 1), np.full(N, el ** -2 - 1)]), (batch, 1))
    del_[:, 3 % N] = del_[:, N + 3 % N] = 0.0     # a site that draws nothing
    hs = r.randint(0, 2, (batch, N)).astype(np.int32)
    rng = np.zeros((batch, 17), np.uint64)
    rng[:, :16] = r.randint(1, 1 << 62, (batch, 16)).astype(np.uint64) * np.uint64(2) + np.uint64(1)
    rng[:, 16] = r.randint(0, 16, batch)
    return nt, G, del_, hs, rng


@pytest.mark.parametrize("form", ["global", "cluster"])
@pytest.mark.parametrize("cplx,N,n_delay,batch", [
    (0, 1, 4, 2), (0, 15, 16, 1), (0, 16, 16, 3), (0, 17, 5, 2), (0, 33, 32, 9), (0, 90, 16, 8),
    (0, 97, 16, 2), (0, 100, 12, 20), (0, 145, 16, 2), (0, 193, 16, 1), (0, 256, 20, 1),
    (1, 13, 16, 2), (1, 65, 16, 3), (1, 91, 7, 9), (1, 113, 16, 1)])
def test_update_windows_match_oracle(monkeypatch, form, cplx, N, n_delay, batch):
    torch = pytest.importorskip("torch")
    from dqmc_b200 import lib
    monkeypatch.setenv("DQMC_UPDATE", form)
    nt, G, del_, hs, rng = _inputs(N, batch, cplx, 7 * N + cplx)
    # column-major, back to back
    dG = torch.from_numpy(np.ascontiguousarray(G.swapaxes(-1, -2))).cuda()
    dhs, drng = torch.from_numpy(hs.copy()).cuda(), torch.from_numpy(rng.view(np.int64).copy()).cuda()
    ddel, dph = torch.from_numpy(del_).cuda(), torch.ones(batch, dtype=dG.dtype, device="cuda")
    rc = lib.load().dqmc_gpu_update_delayed(batch, N, n_delay, cplx, ddel.data_ptr(), drng.data_ptr(),
                                            dhs.data_ptr(), dG.data_ptr(), dph.data_ptr(), None)
    assert rc == 0
    o = oracle_lib(bool(cplx))
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    got = dG.cpu().numpy()
    for c in range(batch):
        g = [np.ascontiguousarray(G[c, s].T).reshape(-1) for s in (0, 1)]
        order, ph = np.zeros(N, np.int32), np.ones(1, nt)
        r, h, d = rng[c].copy(), hs[c].copy(), del_[c].copy()
        o.orc_shuffle(p(r), N, p(order))
        o.orc_update_delayed(N, min(n_delay, N), p(d), p(order), p(r), p(h), p(g[0]), p(g[1]), p(ph))
        assert np.array_equal(dhs.cpu().numpy()[c], h)
        assert np.array_equal(drng.cpu().numpy()[c].view(np.uint64), r)
        for s in (0, 1):
            assert np.max(np.abs(got[c, s].reshape(-1) - g[s])) < G_TOL
        assert abs(dph.cpu().numpy()[c] - ph[0]) < 1e-12
