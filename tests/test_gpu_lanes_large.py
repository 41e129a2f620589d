"""Matrices beyond one SM's shared memory (real N > 154, complex N > 103): the
QR takes the form over a cluster's shared memory or the one with the matrix in L2
by the items of a launch, which the lane count changes.  33 chains lie on one
side of that line in one lane (66 items) and on the other in two (34 and 32),
and every chain must come out bit for bit the same; the first and the last agree
with the oracle (fields and RNG state equal, G to 1e-10 as in the other engine
tests).  33 clusters of the on-chip update take more than one wave for the
complex lattice.
"""
import numpy as np
import pytest

from oracle_ctl import Sim

pytestmark = pytest.mark.gpu

G_TOL = 1e-10


@pytest.mark.parametrize("Nx,Ny,nflux", [(14, 14, 0), (13, 12, 0), (12, 12, 1)])
def test_lanes_on_both_sides_of_the_qr_line(Nx, Ny, nflux, tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dqmc_b200 import engine, gen, simfile
    n, L = 33, 10
    rngs = gen.chain_rngs(17, n)
    base = gen.make_sim(Nx=Nx, Ny=Ny, U=4.0, mu=-0.5, dt=0.1, L=L, n_matmul=5, n_delay=16, period_eqlt=5,
                        nflux=nflux, n_sweep_warm=0, n_sweep_meas=1, init_rng=rngs[0])
    dicts = [base]
    for r in rngs[1:]:
        d = dict(base)
        d["state/hs"], d["state/rng"] = gen.initial_hs(r, L, Nx * Ny)
        dicts.append(d)
    runs = []
    for lanes in (1, 2):
        sims = [engine.SimData(dict(d)) for d in dicts]
        e = engine.Engine(sims, lanes=lanes)
        e.init()
        e.sweeps(1)
        e.pull()
        assert e.errors() == 0
        runs.append((sims, [e.g(c) for c in range(n)]))
        e.close()
    (a, ga), (b, gb) = runs
    for c in range(n):
        assert np.array_equal(a[c].hs, b[c].hs), c
        assert np.array_equal(a[c].rng, b[c].rng), c
        assert np.array_equal(a[c].eq_acc, b[c].eq_acc), c
        for x, y in zip(ga[c], gb[c]):
            assert np.array_equal(np.asarray(x), np.asarray(y)), c
    for c in (0, n - 1):
        path = str(tmp_path / f"c{c}.h5")
        simfile.write(path, dicts[c])
        o = Sim(path)
        gu, gd, ph = o.run(stop_sweep=1)
        assert np.array_equal(a[c].hs, o.hs)
        assert np.array_equal(a[c].rng, o.rng)
        assert np.max(np.abs(ga[c][0] - gu)) < G_TOL
        assert np.max(np.abs(ga[c][1] - gd)) < G_TOL
        assert abs(ga[c][2] - ph) < 1e-12
