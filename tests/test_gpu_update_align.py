"""dqmc_gpu_update_delayed on a G that is aligned to its 8-byte numbers only (a
view that starts at an odd element of a larger buffer): the copies of G to and
from shared memory take 16 bytes at a time only where G allows it, so the call
gives the same bits as on an aligned G and touches nothing beside it.  N on both
sides of the update forms' lines, even and odd; on the CPU, the rule itself.
"""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_gpu_update_window import _inputs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
def test_wide_copies_only_where_every_column_is_aligned(tmp_path):
    """g_wide over N and the base's offset, against the columns' addresses"""
    src = tmp_path / "w.cu"
    src.write_text('#include "update.cuh"\n'
                   'extern "C" int wide(unsigned long long p, int n) { return dq::g_wide((const void *)p, n); }\n')
    so = str(tmp_path / "w.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "dqmc-dev_b200", "csrc"), "-o", so, str(src)], check=True)
    f = C.CDLL(so).wide
    f.argtypes = [C.c_ulonglong, C.c_int]
    for base in (4096, 4104, 4112, 4120):
        for n in range(1, 20):
            cols = all((base + 8 * n * c) % 16 == 0 for c in range(2 * n))
            assert f(base, n) == int(cols and n % 2 == 0), (base, n)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["global", "cluster"])
@pytest.mark.parametrize("N,batch", [(16, 2), (26, 3), (27, 2), (64, 2), (90, 1), (96, 40), (146, 1), (256, 1)])
def test_update_on_g_aligned_to_8_bytes(monkeypatch, form, N, batch):
    torch = pytest.importorskip("torch")
    from dqmc_b200 import lib
    monkeypatch.setenv("DQMC_UPDATE", form)
    _, G, del_, hs, rng = _inputs(N, batch, 0, 3 * N)
    g = np.ascontiguousarray(G.swapaxes(-1, -2)).reshape(-1)
    pad = 5
    out = []
    for off in (0, 1):
        buf = torch.full((g.size + 2 * pad + 1,), 7.0, dtype=torch.float64, device="cuda")
        lo = pad + 1 - off                       # 16-byte multiple from the base for off = 0
        dG = buf[lo:lo + g.size]
        dG.copy_(torch.from_numpy(g))
        assert dG.data_ptr() % 16 == 8 * off
        dhs, drng = torch.from_numpy(hs.copy()).cuda(), torch.from_numpy(rng.view(np.int64).copy()).cuda()
        ddel, dph = torch.from_numpy(del_).cuda(), torch.ones(batch, dtype=torch.float64, device="cuda")
        rc = lib.load().dqmc_gpu_update_delayed(batch, N, 16, 0, ddel.data_ptr(), drng.data_ptr(),
                                                dhs.data_ptr(), dG.data_ptr(), dph.data_ptr(), None)
        assert rc == 0
        b = buf.cpu().numpy()
        assert np.all(b[:lo] == 7.0) and np.all(b[lo + g.size:] == 7.0)
        out.append((b[lo:lo + g.size], dhs.cpu().numpy(), drng.cpu().numpy(), dph.cpu().numpy()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
