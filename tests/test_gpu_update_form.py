"""The form of the delayed update that an engine reports is the one it runs, also
for lattices whose G takes the shared memory of several SMs per spin, and the
tuner times both forms for them."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dqmc_b200 import batch, engine, gen
    return batch, engine, gen


def _sim(mods, n, nflux=0):
    _, engine, gen = mods
    return engine.SimData(gen.make_sim(Nx=n, Ny=n, U=4.0, dt=0.1, L=10, n_matmul=5, n_delay=8, period_eqlt=5,
                                       nflux=nflux, n_sweep_warm=0, n_sweep_meas=4))


# one SM holds G and panels of 8 columns / two to four do: complex N = 100 takes
# 232,192 of the 232,384 bytes of one
@pytest.mark.parametrize("n,nflux,code", [(4, 0, 1), (12, 0, 1), (13, 0, 2), (16, 0, 2), (9, 1, 1), (10, 1, 1),
                                          (11, 1, 2)])
def test_reported_form(mods, monkeypatch, n, nflux, code):
    batch, engine, _ = mods
    monkeypatch.delenv("DQMC_UPDATE", raising=False)
    for form, want in (("cluster", code), ("global", 0)):
        e = engine.Engine([_sim(mods, n, nflux)], update=form)
        assert e.lib.dqmc_engine_update_on_chip(e.h) == want
        assert e.update_form == form
        e.close()


def test_both_forms_are_tuned_where_g_is_spread(mods, monkeypatch):
    batch, engine, _ = mods
    sims = [_sim(mods, 16)]
    assert batch.update_forms(sims, spread=True) == ["global", "cluster"]
    timed = []
    monkeypatch.setattr(batch, "time_sweep", lambda *a, update=None, **k: timed.append(update) or len(timed))
    assert batch.autotune_update(sims) == "global"      # the first of the two fake times
    assert timed == ["global", "cluster"]
