"""Panel QRs of the unequal-time Green's functions: the block reflector is
applied 8 columns and 4 rows at a time, so N around the multiples of 8 and 4
(ragged last panels, columns and rows), the smallest N, one panel only
(E = 1, 2) and the largest N the unequal-time path takes; real and complex.

The measurements carry G(0,t), G(t,0) and G(t,t) of a chain at beta = 1, whose
entries are known to about 1e-12, against the oracle: 1e-9 as the other
unequal-time tests require."""
import numpy as np
import pytest

from oracle_ctl import Sim

pytestmark = pytest.mark.gpu

MEAS_RTOL = 1e-9


@pytest.fixture(scope="module")
def eng():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dqmc_b200 import engine, lib
    lib.load()
    return engine


@pytest.mark.parametrize("Nx,Ny,F,nflux", [
    (2, 2, 5, 0), (3, 3, 4, 0), (5, 3, 6, 0), (7, 7, 5, 0), (13, 5, 3, 0), (16, 10, 4, 0),
    (3, 3, 1, 0), (3, 3, 2, 0), (3, 3, 4, 1), (5, 3, 6, 1), (11, 3, 5, 1), (14, 8, 4, 1)])
def test_unequal_time_matches_oracle(eng, Nx, Ny, F, nflux, tmp_path):
    from dqmc_b200 import gen, simfile
    d = gen.make_sim(Nx=Nx, Ny=Ny, U=4.0, mu=-0.5, dt=0.1, L=2 * F, n_matmul=2, n_delay=8, period_eqlt=2,
                     period_uneqlt=1, nflux=nflux, n_sweep_warm=0, n_sweep_meas=1, seed=11 + Nx)
    path = str(tmp_path / "s.h5")
    simfile.write(path, d)
    o = Sim(path)
    o.run()
    s = eng.SimData.read(path)
    e = eng.Engine([s])
    e.init()
    e.sweeps(1)
    e.pull()
    assert e.errors() == 0
    assert np.array_equal(s.hs, o.hs)
    m = s.measurements()
    for key in (k for k in m if k.startswith("meas_uneqlt/") and k[12:] in o.ue):
        k = key[12:]
        v, r = np.asarray(m[key]).reshape(-1), o.ue[k].reshape(-1)
        np.testing.assert_allclose(v, r, rtol=MEAS_RTOL, atol=MEAS_RTOL * max(np.max(np.abs(r)), 1.0), err_msg=k)
    e.close()
