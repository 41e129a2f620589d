"""The instances of k_update (by N's CTA and by whether the chains outnumber the
SMs) and k_update_cl with more clusters than run at once: every chain bit for bit
the same in both forms, and in a batch as alone in it.  Two chains of different
fields fill the batch by turns, so that two runs of one chain each stand for all.
"""
import numpy as np
import pytest

from test_gpu_update_window import _inputs

pytestmark = pytest.mark.gpu


def _call(lib, torch, monkeypatch, form, cplx, N, n_delay, batch, inp):
    nt, G, del_, hs, rng = inp
    monkeypatch.setenv("DQMC_UPDATE", form)
    rep = lambda a: np.ascontiguousarray(np.concatenate([a] * (batch // len(a))))  # noqa: E731
    d = [torch.from_numpy(rep(x)).cuda() for x in (del_, rng.view(np.int64), hs, G.swapaxes(-1, -2))]
    ph = torch.ones(batch, dtype=d[3].dtype, device="cuda")
    rc = lib.load().dqmc_gpu_update_delayed(batch, N, n_delay, cplx, *[x.data_ptr() for x in d], ph.data_ptr(), None)
    assert rc == 0
    return [x.cpu().numpy() for x in (*d[1:], ph)]


# the edges of k_update's instances (64, 96, 128, 160 rows), beyond 148 chains; a
# cluster form's first waves: 74 clusters of 2 CTAs, 36 of 4, 15 of 8
@pytest.mark.parametrize("cplx,N,batch", [
    (0, 64, 150), (0, 65, 150), (0, 96, 150), (0, 97, 150), (0, 128, 150), (0, 129, 150), (0, 160, 150),
    (0, 161, 150), (0, 146, 40), (0, 206, 18), (1, 64, 150), (1, 65, 150), (1, 160, 150), (1, 161, 20),
    (1, 95, 40), (1, 133, 18)])
def test_forms_agree_beyond_one_wave(monkeypatch, cplx, N, batch):
    torch = pytest.importorskip("torch")
    from dqmc_b200 import lib
    inp = _inputs(N, 2, cplx, 5 * N + cplx)
    a = _call(lib, torch, monkeypatch, "global", cplx, N, 16, batch, inp)
    b = _call(lib, torch, monkeypatch, "cluster", cplx, N, 16, batch, inp)
    one = _call(lib, torch, monkeypatch, "global", cplx, N, 16, 2, inp)
    for x, y, z in zip(a, b, one):
        assert np.array_equal(x, y)
        for c in range(0, batch, 2):
            assert np.array_equal(x[c:c + 2], z)
