"""Device memory of the sweep's stack of decompositions.

With its stack an engine holds 2 F + 7 matrices an item, no more than the
2 F + 8 it held before there was one (clusters, their pair products, work), so
what fitted a GPU then fits now.  Where the stack finds no room, no lane of an
engine takes one: chains of one engine never round differently by what memory
was free when their lane was made.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, F, L, CH = 64, 8, 40, 256
UNIT = 2 * CH * N * N * 8              # one matrix per item


@pytest.fixture(scope="module")
def mods():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dqmc_b200 import engine, gen
    d = gen.make_sim(Nx=8, Ny=8, U=4.0, mu=-0.5, dt=0.1, L=L, n_matmul=5, n_delay=16, period_eqlt=5,
                     n_sweep_warm=0, n_sweep_meas=4, seed=5)
    return torch, engine, d


def _run(mods, lanes, leave=None, sweeps=2):
    """an engine of CH chains (the second half the first half's copies), with
    `leave` bytes of the device free when it is made; its chains, G of all of them
    and the bytes it took"""
    torch, engine, d = mods
    sims = [engine.SimData(dict(d)) for _ in range(CH)]
    for c, s in enumerate(sims):
        s.hs[:] = np.roll(s.hs, 13 * (c % (CH // 2)))
    hold = None
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    if leave is not None:
        hold = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    try:
        free0 = torch.cuda.mem_get_info()[0]
        e = engine.Engine(sims, lanes=lanes)
        used = free0 - torch.cuda.mem_get_info()[0]
        e.init()
        e.sweeps(sweeps)
        e.pull()
        assert e.errors() == 0
        g = [e.g(c) for c in range(CH)]
        e.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    return sims, g, used


def test_memory_with_the_stack(mods):
    _run(mods, 1)                                          # module loading takes memory once
    _, _, used = _run(mods, 1)
    other = 2 * CH * 2 * L * N * 8 + CH * L * N * 4        # field diagonals, fields
    assert used < (2 * F + 8) * UNIT + other + (16 << 20)


def test_all_lanes_have_a_stack_or_none(mods):
    _run(mods, 2)
    a, ga, used = _run(mods, 2)
    st = (F - 1) * UNIT
    # room for none of the lanes' stacks, and for one of the two
    n, gn, used_n = _run(mods, 2, used - st + st // 8)
    b, gb, used_b = _run(mods, 2, used - st // 4)
    assert used_n <= used - st and used_b == used_n
    for x, y, z in zip(a, b, n):
        assert np.array_equal(x.hs, y.hs) and np.array_equal(x.rng, y.rng)
        assert np.array_equal(y.hs, z.hs) and np.array_equal(y.rng, z.rng)
    for g in (ga, gn, gb):
        for c in range(CH // 2):                           # the same chain in either lane
            for x, y in zip(g[c], g[c + CH // 2]):
                assert np.array_equal(np.asarray(x), np.asarray(y)), c
    for c in range(CH):
        for x, y in zip(gb[c], gn[c]):
            assert np.array_equal(np.asarray(x), np.asarray(y)), c
        assert np.max(np.abs(ga[c][0] - gb[c][0])) < 1e-10


def test_clusters_stand_after_gradients(mods):
    """the gradient's update-free sweep and the sweeps share the clusters' place:
    sweeps after a gradient are those without one, a repeated gradient the same"""
    torch, engine, d = mods
    out = []
    for grad in (0, 2):
        s = [engine.SimData(dict(d)) for _ in range(3)]
        e = engine.Engine(s)
        e.init()
        e.sweeps(1)
        lg = [e.logdet_grad() for _ in range(grad)]
        if grad:
            e.obs_grad()
            for x, y in zip(*lg):
                assert np.array_equal(np.asarray(x), np.asarray(y))
        e.sweeps(2)
        e.pull()
        assert e.errors() == 0
        out.append((s[1].hs.copy(), s[1].rng.copy()))
        e.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_gradient_with_and_without_a_place_for_q(mods):
    """the gradient's stack keeps its Q beside the clusters while half of the device
    is free, else in their place: the same bits, and sweeps after it too"""
    torch, engine, d = mods
    out = []
    for full in (False, True):
        free, total = torch.cuda.mem_get_info()
        hold = torch.empty(free - total // 2 + (64 << 20), dtype=torch.uint8, device="cuda") if full else None
        s = [engine.SimData(dict(d)) for _ in range(3)]
        for c, x in enumerate(s):
            x.hs[:] = np.roll(x.hs, 13 * c)
        e = engine.Engine(s)
        e.init()
        e.sweeps(1)
        used0 = torch.cuda.mem_get_info()[0]
        ld, S = e.logdet_grad()
        took = used0 - torch.cuda.mem_get_info()[0]
        ld2, S2 = e.logdet_grad()
        assert np.array_equal(ld, ld2) and np.array_equal(S, S2)
        e.sweeps(2)
        e.pull()
        assert e.errors() == 0
        out.append((np.asarray(ld), np.asarray(S), s[2].hs.copy(), s[2].rng.copy(), e.g(2)[0], took))
        e.close()
        del hold
        torch.cuda.empty_cache()
    assert out[0][5] > out[1][5]                           # the place was taken only with room
    for x, y in zip(out[0][:5], out[1][:5]):
        assert np.array_equal(x, y)
