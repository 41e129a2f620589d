"""Performance cases of the engine: what a user of this framework has it do,
from a single small chain to the benchmark's batch, through the public entry
points (Engine, RaggedBatch, SquareModel and the kernel seams of the C ABI).

A case is a dict of plain values.  Its "kind" says which entry point it goes
through:

  sweep    Engine.sweeps on resident chains, then the state and accumulators
           (what a sim file stores) back on the host, and G of every chain
           where there are only a few
  resume   the same after the chains' state has been uploaded again, as a
           run that continues from its files does (G follows the fields)
  ragged   RaggedBatch: chains of different lattices and L in one batch
  grad     SquareModel.evaluate and evaluate_obs at a new theta
  eq_g, update, mul_seq, gemm
           the kernel seams on device pointers
"""
from __future__ import annotations

import copy
import ctypes
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dqmc-dev_b200"))

from dqmc_b200 import batch, engine, gen, grad, lib  # noqa: E402

SWEEPS_MAX = 10 ** 8      # n_sweep of the chains: a state never completes
NORB = {"square": 1, "triangular": 1, "honeycomb": 2, "kagome": 3}


def _sweep(name, chains, Nx, Ny, L, n_matmul, **kw):
    c = dict(name=name, kind="sweep", chains=chains, geometry="square", Nx=Nx, Ny=Ny, tp=0.0, U=4.0,
             mu=-1.0, nflux=0, dt=0.05, L=L, n_matmul=n_matmul, n_delay=16, period_eqlt=n_matmul,
             period_uneqlt=0, bond=0, sweeps=1)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: one multiplication of a wrap, few chains, odd sizes
        dict(name="gemm_small", kind="gemm", batch=6, M=50, N=45, K=50, cplx=0, beta=0.0),
        # calc_eq_g alone, as a program with its own sweep calls it
        dict(name="eq_g_seam", kind="eq_g", batch=64, Nx=10, Ny=10, nflux=0, F=8, n_matmul=8, dt=0.1, U=4.0, l=3),
        # the plain single-chain configuration: latency and launches count
        _sweep("chain1_4x4", 1, 4, 4, 40, 5, mu=0.0, dt=0.1, n_delay=8, period_eqlt=8),
        # one chain of the benchmark's lattice alone on the GPU
        _sweep("chain1_12x12", 1, 12, 12, 120, 10, period_eqlt=8),
        # one chain with unequal-time measurements every fourth sweep
        _sweep("chain1_uneq8x8", 1, 8, 8, 80, 8, tp=-0.25, mu=-0.5, dt=0.1, period_eqlt=8, period_uneqlt=4,
               sweeps=4),
        # an odd lattice (N = 75), a moderate number of chains
        _sweep("chains24_kagome5x5", 24, 5, 5, 42, 7, geometry="kagome", mu=0.5, dt=0.1, n_delay=12),
        # the largest matrices the dense kernels take (N = 256)
        _sweep("chains4_16x16", 4, 16, 16, 40, 10),
        # complex hopping: every sweep with unequal-time and bond correlators
        _sweep("complex64_10x10", 64, 10, 10, 50, 5, mu=0.0, dt=0.1, nflux=1, period_uneqlt=1, bond=1),
        # the benchmark's batch
        _sweep("chains256_12x12", 256, 12, 12, 120, 10, period_eqlt=8),
        # chains continued from their stored state
        _sweep("resume16_12x10", 16, 12, 10, 40, 10, kind="resume"),
        # uneven lattices and lengths in one batch
        dict(name="ragged8", kind="ragged", chains=8, sides="6,8,10,14", L="20,40,60", dt=0.05, U=4.0),
        # gradients of 128 configurations of the 8x8 lattice at fixed fields
        dict(name="grad128_8x8", kind="grad", n_cfg=128, Nx=8, Ny=8, U=4.0, dt=0.1, L=40, n_matmul=8),
    ]


def _between(rng, lo, hi):
    """a whole number from lo to hi, spread over its logarithm"""
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choices(["sweep", "resume", "grad", "eq_g", "update", "mul_seq", "gemm"],
                       [8, 2, 1, 2, 2, 1, 2])[0]
    if kind == "gemm":
        return dict(kind=kind, batch=_between(rng, 2, 2000), M=_between(rng, 16, 160), N=_between(rng, 16, 160),
                    K=_between(rng, 16, 256), cplx=rng.choice([0, 0, 1]), beta=rng.choice([0.0, 0.5]))
    if kind in ("eq_g", "update", "mul_seq"):
        nflux = rng.choice([0, 0, 1])
        Nx, Ny = rng.randint(4, 12), rng.randint(4, 12)
        c = dict(kind=kind, batch=_between(rng, 1, 256), Nx=Nx, Ny=Ny, nflux=nflux, dt=0.1, U=rng.uniform(2.0, 4.0))
        if kind == "update":
            c.update(n_delay=rng.choice([4, 8, 12, 16, 20]))
        else:
            c.update(n_matmul=rng.randint(3, 8))
        if kind == "eq_g":
            F = rng.randint(2, 8)
            c.update(F=F, l=rng.randrange(F))
        return c
    if kind == "grad":
        F = rng.randint(2, 5)
        return dict(kind=kind, n_cfg=_between(rng, 2, 96), Nx=rng.randint(4, 8), Ny=rng.randint(4, 8),
                    U=rng.uniform(2.0, 4.0), dt=0.1, L=8 * F, n_matmul=8)
    nflux = rng.choice([0, 0, 0, 1])
    geo = rng.choice(["square", "square", "triangular", "honeycomb", "kagome"])
    most = 144 if nflux else 256
    while True:
        Nx, Ny = rng.randint(3, 16), rng.randint(3, 16)
        if 16 <= NORB[geo] * Nx * Ny <= most:
            break
    N = NORB[geo] * Nx * Ny
    n_matmul = rng.randint(4, 10)
    dt = rng.choice([0.05, 0.08])
    F = rng.randint(2, max(2, min(12, int(6.0 / (dt * n_matmul)))))
    if N > 150:
        F = min(F, 4)
    L = F * n_matmul
    uneq = rng.choice([0, 0, 1]) if N <= 100 else 0
    cost = (4 if nflux else 1) * (3 if uneq else 1) * L * N ** 3
    chains = _between(rng, 1, max(1, min(256, int(2.5e10 / cost))))
    c = _sweep("", chains, Nx, Ny, L, n_matmul, kind=kind, geometry=geo, U=rng.uniform(2.0, 4.0),
               mu=rng.choice([0.0, -0.5, -1.0]), nflux=nflux, dt=dt, n_delay=rng.choice([8, 12, 16, 20]),
               period_uneqlt=uneq, bond=uneq * rng.choice([0, 1]))
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _model(geometry, Nx, Ny, tp, U, mu, nflux, dt, L, n_matmul, n_delay, period_eqlt, period_uneqlt, bond):
    return gen.make_sim(geometry=geometry, Nx=Nx, Ny=Ny, tp=tp, U=U, mu=mu, nflux=nflux, dt=dt, L=L,
                        n_matmul=n_matmul, n_delay=n_delay, period_eqlt=period_eqlt,
                        period_uneqlt=period_uneqlt, meas_bond_corr=bond, n_sweep_warm=0,
                        n_sweep_meas=SWEEPS_MAX)


def _model_of(case):
    return _model(*[case[k] for k in ("geometry", "Nx", "Ny", "tp", "U", "mu", "nflux", "dt", "L", "n_matmul",
                                      "n_delay", "period_eqlt", "period_uneqlt", "bond")])


def _fields(seed, shape):
    """random Hubbard-Stratonovich fields, and an RNG state per chain"""
    r = np.random.RandomState(seed % (1 << 32))
    rng = np.zeros((shape[0], 17), np.uint64)
    rng[:, :16] = r.randint(1, 1 << 62, size=(shape[0], 16)).astype(np.uint64) * np.uint64(2) + np.uint64(1)
    return r.randint(0, 2, size=shape).astype(np.int32), rng


def _sims(d, hs, rng):
    base = engine.SimData(d)
    out = []
    for h, r in zip(hs, rng):
        s = copy.copy(base)
        s.p = dict(base.p)
        s.hs, s.rng = h.reshape(-1).copy(), r.copy()
        s.eq_acc, s.ue_acc = base.eq_acc.copy(), base.ue_acc.copy()
        out.append(s)
    return out


def _pinned(shape, dtype):
    t = torch.zeros(int(np.prod(shape)) * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True)
    a = t.numpy().view(dtype).reshape(shape)
    return a, t


def _hopping(case):
    """(exp(-dt K), exp(dt K)) of the seams' square lattice as the engine reads them (column-major), exp(dt lambda)"""
    d = _model("square", case["Nx"], case["Ny"], 0.0, case["U"], -0.5, case["nflux"], case["dt"], 8, 8, 8, 8, 0, 0)
    return d["params/exp_Ku"].T, d["params/exp_lambda"], d["params/del"]


def _ragged_models(case, seed):
    sides = [int(x) for x in case["sides"].split(",")]
    ls = [int(x) for x in case["L"].split(",")]
    out = []
    for c in range(case["chains"]):
        L, n = ls[(c // len(sides)) % len(ls)], sides[c % len(sides)]
        d = _model("square", n, n, 0.0, case["U"], -0.5, 0, case["dt"], L, 10, 16, 10, 0, 0)
        out.append((d, _fields(seed * 97 + c, (1, L, n * n))))
    return out


def _thetas(case, seed):
    r = np.random.RandomState((seed + 7) % (1 << 32))
    n = 2 * case["Nx"] * case["Ny"]
    return [np.concatenate([[1.0, -0.2, -0.5], 0.05 * r.standard_normal(n)]) for _ in range(2)]


def _grad_fields(case, seed):
    return _fields(seed, (case["n_cfg"], case["L"], case["Nx"] * case["Ny"]))[0]


def _seam_inputs(case, seed):
    """inputs of the seams as torch tensors on the GPU, matrices column-major and back to back"""
    k = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    nb = case["batch"]
    if k == "gemm":
        t = torch.complex128 if case["cplx"] else torch.float64
        M, N, K = case["M"], case["N"], case["K"]
        # item b: K x M, N x K and N x M row-major = the column-major operands
        return {"A": torch.randn(nb, K, M, dtype=t, device="cuda", generator=g),
                "B": torch.randn(nb, N, K, dtype=t, device="cuda", generator=g),
                "C": torch.zeros(nb, N, M, dtype=t, device="cuda")}
    eK, el, dl = _hopping(case)
    N = eK.shape[0]
    nt = torch.complex128 if case["nflux"] else torch.float64
    eKt = torch.from_numpy(np.ascontiguousarray(eK)).to("cuda", nt)
    ns = {"update": 8, "mul_seq": case.get("n_matmul"), "eq_g": case.get("F", 1) * case.get("n_matmul", 1)}[k]
    hs, rng = _fields(seed, (nb, ns, N))
    elt = torch.from_numpy(np.ascontiguousarray(el.reshape(2, N))).cuda()
    hst = torch.from_numpy(hs).cuda()
    s = {"eK": eKt, "N": N}
    if k == "mul_seq":
        return s | {"el": elt.reshape(1, -1).expand(nb, -1).contiguous(), "hs": hst,
                    "expK": eKt.T.contiguous(), "C": torch.zeros(nb, N, N, dtype=nt, device="cuda")}

    def product(h):
        """B_{n-1} ... B_0 of the slices h [item, n, N] (field signs)"""
        d = torch.where(h > 0, elt[1], elt[0])
        out = None
        for j in range(h.shape[1]):
            b = eKt * d[:, j, None, :]
            out = b if out is None else b @ out
        return out

    if k == "eq_g":
        m = case["n_matmul"]
        C = torch.stack([product(hst[:, f * m:(f + 1) * m]) for f in range(case["F"])], 1)
        return s | {"C": C.transpose(-1, -2).contiguous(), "G": torch.zeros(nb, N, N, dtype=nt, device="cuda"),
                    "phase": torch.zeros(nb, dtype=nt, device="cuda")}
    eye = torch.eye(N, dtype=nt, device="cuda")
    G = torch.stack([torch.linalg.inv(eye + product(h)) for h in (hst, 1 - hst)], 1)
    return s | {"G0": G.transpose(-1, -2).contiguous(), "hs0": hst[:, 0].contiguous(),
                "rng0": torch.from_numpy(rng.view(np.int64)).cuda(),
                "del": torch.from_numpy(np.tile(dl.reshape(1, -1), (nb, 1))).cuda(),
                "phase0": torch.ones(nb, dtype=nt, device="cuda")}


def prepare(case, seed):
    k = case["kind"]
    if k in ("gemm", "eq_g", "update", "mul_seq"):
        s = _seam_inputs(case, seed)
        if k == "update":
            s |= {x: s[x + "0"].clone() for x in ("G", "hs", "rng", "phase")}
        return {"case": case, "lib": lib.load(), **s}
    if k == "ragged":
        sims = [_sims(d, *f)[0] for d, f in _ragged_models(case, seed)]
        rb = batch.RaggedBatch(sims)
        rb.init()
        return {"case": case, "rb": rb, "sims": sims}
    if k == "grad":
        m = grad.SquareModel(case["Nx"], case["Ny"], case["U"], case["dt"], case["L"], _grad_fields(case, seed),
                             n_matmul=case["n_matmul"])
        return {"case": case, "model": m, "theta": _thetas(case, seed), "i": 0}
    d = _model_of(case)
    n, L, N = case["chains"], case["L"], int(d["params/N"])
    sims = _sims(d, *_fields(seed, (n, L, N)))
    e = engine.Engine(sims)
    e.init()
    s = {"case": case, "engine": e, "keep": []}
    for key, shape, dt in (("rng", (n, 17), np.uint64), ("hs", (n, L * N), np.int32), ("eq_n", (n,), np.int32),
                           ("eq_acc", (n, sims[0].eq_acc.size), sims[0].nt), ("ue_n", (n,), np.int32),
                           ("ue_acc", (n, sims[0].ue_acc.size), sims[0].nt)):
        if key.startswith("ue") and not case["period_uneqlt"]:
            continue
        s[key], t = _pinned(shape, dt)
        s["keep"].append(t)
    if k == "resume":
        s["up"] = []
        for a in e.state_arrays():
            p, t = _pinned(a.shape, a.dtype)
            p[...] = a
            s["up"].append(p)
            s["keep"].append(t)
    return s


# -------------------------------------------------------------------- pass

def run(s):
    case = s["case"]
    k = case["kind"]
    if k in ("sweep", "resume"):
        e = s["engine"]
        if k == "resume":
            e.set_chains(*s["up"], sweep=0)
        e.sweeps(case["sweeps"], sync=False)
        e.get_chains(s["rng"], s["hs"], s["eq_n"], s["eq_acc"], s.get("ue_n"), s.get("ue_acc"))
        # the RNG's 64-bit words as signed numbers
        out = {"hs": s["hs"], "rng": s["rng"].view(np.int64), "eq_n": s["eq_n"], "eq_acc": s["eq_acc"]}
        if case["period_uneqlt"]:
            out |= {"ue_n": s["ue_n"], "ue_acc": s["ue_acc"]}
        if case["chains"] <= 4:
            out["g"] = [e.g(c) for c in range(case["chains"])]
        return out
    if k == "ragged":
        s["rb"].sweeps(1, sync=False)
        s["rb"].pull()
        return [{"hs": x.hs, "rng": x.rng.view(np.int64), "eq_acc": x.eq_acc} for x in s["sims"]]
    if k == "grad":
        # an optimiser's next theta: the hopping changes from pass to pass
        th = s["theta"][s["i"] % 2]
        s["i"] += 1
        ld, g = s["model"].evaluate(th)
        obs, go = s["model"].evaluate_obs(th)
        return {"ld": ld, "grad": g, "obs": obs, "obs_grad": go}
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    L = s["lib"]
    if k == "gemm":
        M, N, K, cx = case["M"], case["N"], case["K"], case["cplx"]
        one, beta = (ctypes.c_double * 2)(1.0, 0.0), (ctypes.c_double * 2)(case["beta"], 0.0)
        lib.check(L.dqmc_gpu_gemm(case["batch"], M, N, K, cx, one, s["A"].data_ptr(), M,
                                  ctypes.c_longlong(M * K), s["B"].data_ptr(), K, ctypes.c_longlong(K * N), beta,
                                  s["C"].data_ptr(), M, ctypes.c_longlong(M * N), st), "dqmc_gpu_gemm")
        return s["C"]
    cx = int(case["nflux"] != 0)
    if k == "eq_g":
        lib.check(L.dqmc_gpu_calc_eq_g(case["batch"], s["N"], case["F"], case["l"], cx, s["C"].data_ptr(),
                                       s["G"].data_ptr(), s["phase"].data_ptr(), st), "dqmc_gpu_calc_eq_g")
        return {"G": s["G"], "phase": s["phase"]}
    if k == "mul_seq":
        lib.check(L.dqmc_gpu_mul_seq(case["batch"], s["N"], case["n_matmul"], 0, cx, s["expK"].data_ptr(),
                                     s["el"].data_ptr(), s["hs"].data_ptr(), s["C"].data_ptr(), st),
                  "dqmc_gpu_mul_seq")
        return s["C"]
    # the update works in place: every pass starts from the same slice
    for x in ("G", "hs", "rng", "phase"):
        s[x].copy_(s[x + "0"])
    lib.check(L.dqmc_gpu_update_delayed(case["batch"], s["N"], case["n_delay"], cx, s["del"].data_ptr(),
                                        s["rng"].data_ptr(), s["hs"].data_ptr(), s["G"].data_ptr(),
                                        s["phase"].data_ptr(), st), "dqmc_gpu_update_delayed")
    return {"G": s["G"], "hs": s["hs"], "rng": s["rng"], "phase": s["phase"]}


# -------------------------------------------------------------------- work

def _sweep_work(chains, N, L, F, cx, uneq, acc, fields_twice=2):
    """One sweep: wraps, cluster products, one factorisation step forward and
    one backward with its two products and one solve per cluster boundary,
    two thirds of the sites accepted; the state and accumulators in and out."""
    n3 = float(N) ** 3
    per = (L - F) * 4 * n3 + (L - F) * 2 * n3 + F * (2 * (8 / 3 + 4) + 8 / 3) * n3 + L * (2 / 3) * 2 * n3
    if uneq:
        per += L * (3 * 2 + 2 + 6 * 2) * n3    # three stacks built and half wrapped
    fl = 2 * chains * per * (4 if cx else 1)
    by = chains * (fields_twice * 4 * L * N + 2 * 17 * 8 + 2 * acc * (16 if cx else 8)) + 16 * N * N * (16 if cx else 8)
    return {"flops": fl, "bytes": by}


def work(case):
    k = case["kind"]
    if k in ("sweep", "resume"):
        N = NORB[case["geometry"]] * case["Nx"] * case["Ny"]
        d = _model_of(case)
        acc = sum(np.size(v) for key, v in d.items() if key.startswith("meas_"))
        n = case["sweeps"]
        w = _sweep_work(case["chains"], N, case["L"], case["L"] // case["n_matmul"], case["nflux"],
                        1.0 / case["period_uneqlt"] if case["period_uneqlt"] else 0, acc)
        return {"flops": n * w["flops"], "bytes": w["bytes"]}
    if k == "ragged":
        sides = [int(x) for x in case["sides"].split(",")]
        ls = [int(x) for x in case["L"].split(",")]
        out = {"flops": 0.0, "bytes": 0.0}
        for c in range(case["chains"]):
            n = sides[c % len(sides)] ** 2
            L = ls[(c // len(sides)) % len(ls)]
            w = _sweep_work(1, n, L, L // 10, 0, 0, 11 * n)
            out = {x: out[x] + w[x] for x in out}
        return out
    if k == "grad":
        N, L, n = case["Nx"] * case["Ny"], case["L"], case["n_cfg"]
        n3 = float(N) ** 3
        # log-det: one update-free sweep; observables: a row and a column of
        # the space-time G per slice and their product, for two weights
        fl = 2 * n * (4 * L * n3 + L * (4 * L * 2 * n3 + 2 * L * 2 * n3))
        return {"flops": fl, "bytes": 4.0 * n * L * N + 8.0 * n * 3 * (3 + 2 * N)}
    if k == "gemm":
        M, N, K, b = case["M"], case["N"], case["K"], case["batch"]
        e = 16 if case["cplx"] else 8
        return {"flops": (8.0 if case["cplx"] else 2.0) * b * M * N * K,
                "bytes": e * float(b) * (M * K + K * N + M * N * (2 if case["beta"] else 1))}
    N = case["Nx"] * case["Ny"]
    e, cx, b, n3 = (16, 4, case["batch"], float(N) ** 3) if case["nflux"] else (8, 1, case["batch"], float(N) ** 3)
    if k == "eq_g":
        # products two clusters at a time, a factorisation and two products per pair, the solve
        p = (case["F"] + 1) // 2
        return {"flops": cx * b * n3 * (2 * (case["F"] // 2) + p * (8 / 3) + (p - 1) * 4 + 8 / 3),
                "bytes": e * float(b) * N * N * (case["F"] + 1)}
    if k == "mul_seq":
        return {"flops": cx * b * n3 * 2 * (case["n_matmul"] - 1),
                "bytes": e * float(N * N) * (b + 1) + 4.0 * b * case["n_matmul"] * N}
    return {"flops": cx * b * 2 * (2 / 3) * 2 * n3, "bytes": e * 4.0 * b * N * N}


# --------------------------------------------- the same values in plain numpy

_M64 = (1 << 64) - 1


class _Rng:
    """xorshift1024*: 16 words and a position"""

    def __init__(self, words):
        self.s, self.p = [int(x) for x in words[:16]], int(words[16])

    def next(self):
        a = self.s[self.p]
        self.p = (self.p + 1) & 15
        b = self.s[self.p]
        b ^= (b << 31) & _M64
        self.s[self.p] = b ^ a ^ (b >> 11) ^ (a >> 30)
        return (self.s[self.p] * 1181783497276652981) & _M64

    def words(self):
        return np.array(self.s + [self.p], np.uint64)


def _phase(x):
    return x / abs(x) if x != 0 else 1.0


def _stable_g(Cs):
    """(G, phase, log |det|) of (I + C_{n-1} ... C_0)^-1 from the factors in order of application: QR with the
    columns in order of norm after each, scales kept apart"""
    N = Cs[0].shape[0]
    Q, d, T = np.eye(N, dtype=Cs[0].dtype), np.ones(N), np.eye(N, dtype=Cs[0].dtype)
    for C in Cs:
        X = (C @ Q) * d
        p = np.argsort(-(np.abs(X) ** 2).sum(0), kind="stable")
        Q, R = np.linalg.qr(X[:, p])
        d = np.abs(np.diag(R)).copy()
        d[d == 0] = 1.0
        T = (R / d[:, None]) @ T[p]
    big, small = np.maximum(d, 1.0), np.minimum(d, 1.0)
    Y = Q.conj().T / big[:, None]
    M = Y + small[:, None] * T
    sm, lm = np.linalg.slogdet(M)
    sq = np.linalg.slogdet(Q)[0]
    return np.linalg.solve(M, Y), sm * sq, lm + np.log(big).sum()


def _update_slice(r, hs, dl, G, order, phase):
    """the Metropolis sweep of one slice's sites, G of both spins changed one rank at a time"""
    for i in order:
        h = hs[i]
        de = (dl[h, i], dl[1 - h, i])
        if de[0] == 0.0 and de[1] == 0.0:
            continue
        u = (r.next() >> 12) * 2.0 ** -52
        rat = [1.0 + (1.0 - G[s][i, i]) * de[s] for s in (0, 1)]
        prob = rat[0] * rat[1]
        if u < abs(prob):
            for s in (0, 1):
                a = G[s][:, i].copy()
                a[i] -= 1.0
                G[s] += np.outer(a * (de[s] / rat[s]), G[s][i])
            phase = phase * _phase(prob)
            hs[i] = 1 - h
    return phase


def _shuffle(r, N):
    order = [0] * N
    for i in range(N):
        j = (r.next() >> 3) % (i + 1)
        order[i] = order[j]
        order[j] = i
    return order


def _meas_eq(d, G, phase, acc):
    """the always-on equal-time set"""
    P = lambda k: np.asarray(d["params/" + k])  # noqa: E731
    N = int(P("N"))
    ni, nij = int(P("num_i")), int(P("num_ij"))
    mi, mij = P("map_i").reshape(-1), P("map_ij").reshape(-1)          # mij[i + N j]
    pu = P("peierlsu").reshape(-1).reshape(N, N)                       # [i, j] = flat[j + N i]
    pd = P("peierlsd").reshape(-1).reshape(N, N)
    gu, gd = G
    nu, nd = 1.0 - np.diag(gu), 1.0 - np.diag(gd)
    one = np.eye(N)

    def add(m, n, v):
        v = np.asarray(v, dtype=acc.dtype)
        if acc.dtype.kind == "c":
            return np.bincount(m, v.real, n) + 1j * np.bincount(m, v.imag, n)
        return np.bincount(m, v, n)

    acc[0] += phase
    o = 1
    for v in (nu + nd, nu, nd, nu * nd):
        acc[o:o + ni] += phase / float(P("degen_i").reshape(-1)[0]) * add(mi, ni, v)
        o += ni
    a, b = gu * pu, gd * pd
    x = one * (2.0 - nu - nd)[:, None] - (gu.T * gu + gd.T * gd)
    dens, sz = nu + nd, nu - nd
    for v in (0.5 * (a + b), a, b, np.outer(dens, dens) + x,
              0.25 * (one * (2.0 - nu - nd)[:, None] - (gu.T * gd + gd.T * gu)),
              0.25 * (np.outer(sz, sz) + x), gu * gd):
        acc[o:o + nij] += phase / float(P("degen_ij").reshape(-1)[0]) * add(mij, nij, v.T.reshape(-1))
        o += nij


def _exact_sweeps(d, hs, rng, n):
    """n sweeps of one chain: (hs, rng, accumulators, G up, G down, phase)"""
    P = lambda k: np.asarray(d["params/" + k])  # noqa: E731
    N, L, nm = int(P("N")), int(P("L")), int(P("n_matmul"))
    F, pe = L // nm, int(P("period_eqlt"))
    m = {k: [P(k + s).T for s in "ud"] for k in ("exp_K", "inv_exp_K", "exp_halfK", "inv_exp_halfK")}
    el, dl = P("exp_lambda").reshape(2, N), P("del").reshape(2, N)
    hs, r = hs.reshape(L, N).astype(np.int64), _Rng(rng)
    nt = m["exp_K"][0].dtype
    acc = np.zeros(1 + 4 * int(P("num_i")) + 7 * int(P("num_ij")), nt)
    at = np.arange(N)

    def cluster(f, s):
        out = None
        for l in range(f * nm, (f + 1) * nm):
            b = m["exp_K"][s] * el[hs[l] ^ s, at]
            out = b if out is None else b @ out
        return out

    C = [[cluster(f, s) for f in range(F)] for s in (0, 1)]

    def fresh(l0):
        g = [_stable_g(C[s][l0:] + C[s][:l0]) for s in (0, 1)]
        return [g[0][0], g[1][0]], g[0][1] * g[1][1]

    G, phase = fresh(0)
    for _ in range(n):
        for l in range(L):
            phase = _update_slice(r, hs[l], dl, G, _shuffle(r, N), phase)
            if (l + 1) % nm == 0:
                for s in (0, 1):
                    C[s][l // nm] = cluster(l // nm, s)
                G, phase = fresh((l // nm + 1) % F)
            else:
                for s in (0, 1):
                    v = el[hs[l] ^ s, at]
                    G[s] = m["exp_K"][s] @ ((v[:, None] * G[s] / v) @ m["inv_exp_K"][s])
            if (l + 1) % pe == 0:
                _meas_eq(d, [m["inv_exp_halfK"][s] @ (G[s] @ m["exp_halfK"][s]) for s in (0, 1)], phase, acc)
    return hs, r.words(), acc, G[0], G[1], phase


def _exact_grad(case, seed):
    """log |det| of both spins, its gradient, and density and double occupancy at the first theta"""
    hs = _grad_fields(case, seed)
    th = _thetas(case, seed)[0]
    Nx, Ny, L, nm, dt = case["Nx"], case["Ny"], case["L"], case["n_matmul"], case["dt"]
    N = Nx * Ny
    nn, nnn = [], []
    for iy in range(Ny):
        for ix in range(Nx):
            i, r, u = ix + Nx * iy, (ix + 1) % Nx + Nx * iy, ix + Nx * ((iy + 1) % Ny)
            nn += [(i, r), (i, u)]
            nnn += [(i, (ix + 1) % Nx + Nx * ((iy + 1) % Ny)), (r, u)]
    E = np.zeros((3 + len(nn), N, N))
    for b, (i, j) in enumerate(nn):
        for q in (0, 3 + b):
            E[q, i, j] -= 1.0
            E[q, j, i] -= 1.0
    for i, j in nnn:
        E[1, i, j] -= 1.0
        E[1, j, i] -= 1.0
    E[2] -= np.eye(N)
    K = np.tensordot(np.asarray(th), E, 1)
    w, V = np.linalg.eigh(K)
    eK, iK = (V * np.exp(-dt * w)) @ V.T, (V * np.exp(dt * w)) @ V.T
    a = -dt * w
    da = a[:, None] - a[None]
    with np.errstate(divide="ignore", invalid="ignore"):
        wt = -dt * np.exp(a[None] - a[:, None]) * np.where(np.abs(da) > 1e-12, np.expm1(da) / da, 1.0)
    Em = np.einsum("ai,kab,bj->kij", V, E, V, optimize=True) * wt
    lam = np.arccosh(np.exp(0.5 * case["U"] * dt))
    ld, S, obs = np.zeros(len(hs)), np.zeros((len(hs), N, N)), np.zeros((len(hs), 2))
    for c, h in enumerate(hs):
        occ = np.zeros((2, L, N))
        for s in (0, 1):
            v = np.exp(lam * np.where((h ^ s) > 0, 1.0, -1.0))
            Cs = []
            for f in range(L // nm):
                P = np.eye(N)
                for l in range(f * nm, (f + 1) * nm):
                    P = eK @ (v[l][:, None] * P)
                Cs.append(P)
            for f in range(L // nm):
                G, _, l0 = _stable_g(Cs[f:] + Cs[:f])
                if f == 0:
                    ld[c] += l0
                for l in range(f * nm, (f + 1) * nm):
                    occ[s, l] = 1.0 - np.diag(G)
                    S[c] += v[l][:, None] * (np.eye(N) - G) / v[l]
                    G = eK @ ((v[l][:, None] * G / v[l]) @ iK)
        obs[c] = occ.sum() / (N * L), (occ[0] * occ[1]).sum() / (N * L)
    g = np.einsum("cab,kba->ck", S, np.einsum("ai,kij,bj->kab", V, Em, V, optimize=True), optimize=True)
    return {"ld": ld, "grad": g, "obs": obs, "obs_grad": None}


def _quick(sites, N):
    """whether numpy takes few seconds over this many site visits"""
    return sites <= 80000 and sites * N * N <= 3e9


def exact(case, seed):
    k = case["kind"]
    if k == "grad":
        return _exact_grad(case, seed)
    if k in ("sweep", "resume"):
        d = _model_of(case)
        n, L, N = case["chains"], case["L"], int(d["params/N"])
        if not _quick(n * case["sweeps"] * L * N, N):
            return None
        hs, rng = _fields(seed, (n, L, N))
        got = [_exact_sweeps(d, hs[c], rng[c], case["sweeps"]) for c in range(n)]
        out = {"hs": None, "rng": None, "eq_n": None, "eq_acc": np.stack([x[2] for x in got])}
        if case["period_uneqlt"]:
            out |= {"ue_n": None, "ue_acc": None}
        if n <= 4:
            out["g"] = [(x[3], x[4], np.asarray(x[5], x[2].dtype)) for x in got]
        return out
    if k == "ragged":
        out = []
        for d, (hs, rng) in _ragged_models(case, seed):
            out.append({"hs": None, "rng": None, "eq_acc": _exact_sweeps(d, hs[0], rng[0], 1)[2]})
        return out
    if k == "update" and not _quick(case["batch"] * case["Nx"] * case["Ny"], case["Nx"] * case["Ny"]):
        return None
    s = {x: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for x, v in _seam_inputs(case, seed).items()}
    if k == "gemm":
        return np.matmul(s["B"], s["A"])          # the transposes: (A B)^T = B^T A^T
    if k == "eq_g":
        C, l = s["C"].swapaxes(-1, -2), case["l"]
        got = [_stable_g([c[(l + f) % case["F"]] for f in range(case["F"])]) for c in C]
        return {"G": np.stack([g[0].T for g in got]), "phase": np.array([g[1] for g in got])}
    if k == "mul_seq":
        N, el = s["N"], s["el"][0].reshape(2, -1)
        out = None
        for j in range(case["n_matmul"]):
            b = s["eK"] * el[s["hs"][:, j], np.arange(N)][:, None, :]
            out = b if out is None else b @ out
        return out.swapaxes(-1, -2)
    N, dl = s["N"], s["del"][0].reshape(2, -1)
    G, hs, ph = [], [], []
    for c in range(case["batch"]):
        r = _Rng(s["rng0"][c].view(np.uint64))
        g, h = [s["G0"][c, q].T.copy() for q in (0, 1)], s["hs0"][c].copy()
        # the order is drawn first, then a uniform per visited site
        ph.append(_update_slice(r, h, dl, g, _shuffle(r, N), 1.0))
        G.append(np.stack([x.T for x in g]))
    return {"G": np.stack(G), "hs": None, "rng": None, "phase": np.array(ph, s["phase0"].dtype)}
