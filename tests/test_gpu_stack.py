"""The sweep's stack of decompositions (one factorisation per recalculation on
each side, src/greens.c:69-208 for the algorithm it replaces) against the
oracle: cluster counts F from 1 up (no stack, one entry, several; even and
odd), N around the GEMM tiles' edges, odd N (no tensor maps), the global-memory
factorisations, real and complex; and an engine that finds no room for the
stack, which takes the whole chain at every recalculation.

Fields and RNG state must be equal.  G: both sides carry the rounding of a
stabilised chain at beta <= 3, U = 4, whose G is known to about 1e-12 there,
so they agree to 1e-10 as the other engine tests require.
"""
import numpy as np
import pytest

from oracle_ctl import Sim

pytestmark = pytest.mark.gpu

G_TOL = 1e-10


@pytest.fixture(scope="module")
def eng():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dqmc_b200 import engine, lib
    lib.load()
    return engine


@pytest.mark.parametrize("Nx,Ny,L,nmul,nflux", [
    (4, 4, 5, 5, 0), (4, 3, 10, 5, 0), (5, 3, 15, 5, 0), (7, 7, 20, 5, 0), (8, 4, 24, 4, 0), (5, 5, 30, 5, 0),
    (11, 5, 10, 5, 0), (13, 13, 10, 5, 0), (5, 3, 15, 5, 1), (6, 6, 20, 4, 1), (9, 7, 10, 5, 1),
    (12, 11, 10, 5, 1)])
def test_sweeps_match_oracle(eng, Nx, Ny, L, nmul, nflux, tmp_path):
    from dqmc_b200 import gen, simfile
    d = gen.make_sim(Nx=Nx, Ny=Ny, U=4.0, mu=-0.5, dt=0.1, L=L, n_matmul=nmul, n_delay=12, period_eqlt=nmul,
                     nflux=nflux, n_sweep_warm=0, n_sweep_meas=2, seed=31 + Nx)
    path = str(tmp_path / "s.h5")
    simfile.write(path, d)
    o = Sim(path)
    gu_o, gd_o, ph_o = o.run(stop_sweep=2)
    s = eng.SimData.read(path)
    e = eng.Engine([s])
    e.init()
    e.sweeps(2)
    e.pull()
    assert e.errors() == 0
    assert np.array_equal(s.hs, o.hs)
    assert np.array_equal(s.rng, o.rng)
    gu, gd, ph = e.g(0)
    assert np.max(np.abs(gu - gu_o)) < G_TOL
    assert np.max(np.abs(gd - gd_o)) < G_TOL
    assert abs(ph - ph_o) < 1e-12
    e.close()


def test_engine_without_room_for_the_stack(eng):
    import torch
    from dqmc_b200 import gen
    N, F, n = 64, 8, 256
    d = gen.make_sim(Nx=8, Ny=8, U=4.0, mu=-0.5, dt=0.1, L=40, n_matmul=5, n_delay=16, period_eqlt=5,
                     n_sweep_warm=0, n_sweep_meas=2, seed=5)
    stack = (F - 1) * 2 * n * 2 * N * N * 8            # bytes of its two matrices per entry

    def run():
        sims = [eng.SimData(dict(d)) for _ in range(n)]
        for c, s in enumerate(sims):
            s.hs[:] = np.roll(s.hs, 13 * c)
        free0 = torch.cuda.mem_get_info()[0]
        e = eng.Engine(sims, lanes=1)
        used = free0 - torch.cuda.mem_get_info()[0]
        e.init()
        e.sweeps(2)
        e.pull()
        assert e.errors() == 0
        g = [e.g(c) for c in (0, n - 1)]
        e.close()
        return sims, g, used

    a, ga, used = run()
    assert used > stack
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    # the rest fits, half of the stack does not
    hold = torch.empty(free - (used - stack // 2), dtype=torch.uint8, device="cuda")
    try:
        b, gb, used_b = run()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert used_b < used - stack // 2
    for x, y in zip(a, b):
        assert np.array_equal(x.hs, y.hs)
        assert np.array_equal(x.rng, y.rng)
    for x, y in zip(ga, gb):
        assert np.max(np.abs(x[0] - y[0])) < G_TOL
        assert np.max(np.abs(x[1] - y[1])) < G_TOL
