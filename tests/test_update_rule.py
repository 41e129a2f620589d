"""The rule that chooses the delayed update's form (update_split, update_cl.cuh)
against measured sweeps: at every row the form it takes is at most 4% slower than
the fastest one measured.  Rows: scalar, N, chains, then milliseconds a sweep (L =
10, default lanes, one B200) with G in device memory and on chip in 1, 2 and 4 CTAs
per spin (None: not measured, or does not fit).  The times scatter by 1 to 2%.
"""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

ROWS = """
zd 16 8 0.38 0.41 - -
zd 16 32 0.39 0.42 - -
zd 16 64 0.43 0.47 - -
zd 16 100 0.47 0.50 - -
zd 16 128 0.52 0.57 - -
zd 16 192 0.63 0.68 - -
zd 16 256 0.74 0.81 - -
zd 25 8 0.59 0.60 - -
zd 25 32 0.60 0.62 - -
zd 25 64 0.64 0.66 - -
zd 25 100 0.76 0.81 - -
zd 25 128 0.83 0.91 - -
zd 25 192 1.07 1.16 - -
zd 25 256 1.32 1.44 - -
zd 36 8 0.98 0.86 - -
zd 36 32 1.02 0.91 - -
zd 36 64 1.12 0.98 - -
zd 36 100 1.32 1.26 - -
zd 36 128 1.51 1.42 - -
zd 36 192 1.99 1.97 - -
zd 36 256 2.44 2.50 - -
zd 49 8 1.49 1.21 - -
zd 49 32 1.59 1.31 - -
zd 49 64 1.78 1.48 - -
zd 49 100 2.15 1.96 - -
zd 49 128 2.42 2.24 - -
zd 49 192 3.25 3.16 - -
zd 49 256 3.75 3.73 - -
zd 64 8 1.77 1.42 1.36 -
zd 64 32 1.88 1.54 1.48 -
zd 64 64 2.12 1.77 2.28 -
zd 64 100 2.52 2.41 3.48 -
zd 64 128 2.85 2.95 4.22 -
zd 64 192 3.91 4.40 6.26 -
zd 64 256 4.63 5.72 8.13 -
zd 81 8 3.07 2.20 2.05 2.04
zd 81 32 3.45 2.57 2.43 4.39
zd 81 64 3.91 3.07 3.65 6.23
zd 81 100 4.62 4.18 5.58 9.04
zd 81 128 5.16 5.12 6.75 -
zd 81 192 7.10 7.57 10.25 -
zd 81 256 9.28 10.04 13.59 -
zd 100 8 3.98 - 2.88 2.75
zd 100 32 4.66 - 3.56 5.94
zd 100 64 5.34 - 5.43 8.40
zd 100 100 6.47 - 8.18 12.13
zd 100 128 7.61 - 10.17 -
zd 100 192 11.00 - 15.38 -
zd 100 256 14.61 - 20.42 -
zd 121 8 5.65 - 3.85 3.63
zd 121 32 6.62 - 4.81 7.59
zd 121 64 8.31 - 7.93 11.59
zd 121 100 9.74 - 11.55 16.22
zd 121 128 12.52 - 15.24 -
zd 121 192 16.74 - 21.41 -
zd 121 256 21.94 - 28.44 -
zd 144 8 7.98 - - 4.96
zd 144 32 9.20 - - 9.97
zd 144 64 11.46 - - 15.11
zd 144 100 14.02 - - 21.73
zd 144 128 17.90 - - -
zd 144 192 24.49 - - -
zd 144 256 32.34 - - -
zd 169 8 12.95 - - 6.79
zd 169 32 16.11 - - 14.73
zd 169 64 19.99 - - 21.58
zd 169 100 26.90 - - 32.96
zd 169 128 32.05 - - -
zd 169 192 46.37 - - -
zd 169 256 61.94 - - -
d 16 8 0.29 0.29 - -
d 16 32 0.29 0.30 - -
d 16 64 0.30 0.31 - -
d 16 100 0.33 0.33 - -
d 16 128 0.35 0.36 - -
d 16 192 0.40 0.42 - -
d 16 256 0.51 0.53 - -
d 25 8 0.40 0.37 - -
d 25 32 0.41 0.39 - -
d 25 64 0.43 0.41 - -
d 25 100 0.48 0.47 - -
d 25 128 0.50 0.48 - -
d 25 192 0.61 0.60 - -
d 25 256 0.75 0.75 - -
d 36 8 0.63 0.51 - -
d 36 32 0.66 0.55 - -
d 36 64 0.70 0.59 - -
d 36 100 0.76 0.66 - -
d 36 128 0.84 0.72 - -
d 36 192 1.00 0.93 - -
d 36 256 1.28 1.21 - -
d 49 8 0.88 0.65 - -
d 49 32 0.96 0.72 - -
d 49 64 1.01 0.77 - -
d 49 100 1.15 0.94 - -
d 49 128 1.23 0.98 - -
d 49 192 1.54 1.33 - -
d 49 256 2.19 2.08 - -
d 64 8 1.01 0.74 - -
d 64 32 1.06 0.78 - -
d 64 64 1.11 0.84 - -
d 64 100 1.33 1.37 - -
d 64 128 1.36 1.26 - -
d 64 192 1.76 1.74 - -
d 64 256 2.30 2.52 - -
d 81 8 1.44 1.05 1.02 -
d 81 32 1.58 1.17 1.15 -
d 81 64 1.74 1.33 1.75 -
d 81 100 2.36 2.42 3.24 -
d 81 128 2.38 2.23 3.05 -
d 81 192 3.21 3.11 4.43 -
d 81 256 4.22 4.39 6.12 -
d 100 8 1.83 1.39 1.32 1.28
d 100 32 2.03 1.59 1.52 2.55
d 100 64 2.27 1.84 2.36 3.89
d 100 100 3.09 3.32 4.32 5.82
d 100 128 3.15 3.12 4.14 -
d 100 192 4.67 4.49 5.99 -
d 100 256 5.71 6.03 7.95 -
d 121 8 2.69 1.83 1.71 1.64
d 121 32 2.94 2.07 1.94 3.16
d 121 64 3.42 2.56 3.17 4.94
d 121 100 4.47 4.41 5.60 7.28
d 121 128 4.62 4.25 5.43 -
d 121 192 7.14 6.26 8.03 -
d 121 256 8.86 8.36 10.73 -
d 144 8 3.58 2.23 2.12 2.05
d 144 32 3.90 2.56 2.45 3.99
d 144 64 4.32 3.00 3.77 6.03
d 144 100 5.80 5.45 6.97 9.13
d 144 128 5.97 5.28 6.75 -
d 144 192 8.42 7.75 10.02 -
d 144 256 11.29 10.31 13.15 -
d 156 8 4.49 - 2.94 2.84
d 156 32 5.13 - 3.57 5.25
d 156 64 5.63 - 5.07 7.56
d 156 100 7.90 - 9.32 11.68
d 156 128 8.54 - 9.82 -
d 156 192 12.32 - 14.42 -
d 156 256 19.61 - 21.90 -
d 169 8 5.50 - 3.32 3.15
d 169 32 6.42 - 4.21 6.09
d 169 64 7.51 - 6.51 9.23
d 169 100 10.70 - 12.06 14.53
d 169 128 12.12 - 12.38 -
d 169 192 17.45 - 18.82 -
d 169 256 25.03 - 26.02 -
d 196 8 7.09 - 4.19 3.96
d 196 32 8.13 - 5.18 7.56
d 196 64 9.60 - 8.20 11.64
d 196 100 13.39 - 15.01 18.03
d 196 128 15.38 - 16.29 -
d 196 192 22.51 - 24.09 -
d 196 256 31.75 - 32.68 -
d 225 8 10.80 - - 5.16
d 225 32 13.99 - - 11.36
d 225 64 16.60 - - 17.04
d 225 100 23.67 - - 27.26
d 225 128 26.75 - - 31.15
d 225 192 39.84 - - 46.28
d 225 256 52.41 - - 60.95
d 256 8 13.58 - - 6.13
d 256 32 17.63 - - 13.61
d 256 64 20.54 - - 20.05
d 256 100 29.56 - - 31.94
d 256 128 33.58 - - 35.97
d 256 192 48.71 - - 53.26
d 256 256 65.82 - - 70.68
zd 28 8 0.61 0.71 - -
zd 28 32 0.63 0.70 - -
zd 28 64 0.66 0.75 - -
zd 28 100 0.78 0.88 - -
zd 28 128 0.87 1.00 - -
zd 28 192 1.13 1.25 - -
zd 28 256 1.40 1.55 - -
zd 30 8 0.65 0.67 - -
zd 30 32 0.66 0.69 - -
zd 30 64 0.70 0.74 - -
zd 30 100 0.82 0.90 - -
zd 30 128 0.92 1.00 - -
zd 30 192 1.19 1.26 - -
zd 30 256 1.45 1.59 - -
zd 32 8 0.65 0.67 - -
zd 32 32 0.67 0.69 - -
zd 32 64 0.71 0.74 - -
zd 32 100 0.83 0.88 - -
zd 32 128 0.93 0.98 - -
zd 32 192 1.21 1.26 - -
zd 32 256 1.52 1.58 - -
zd 33 8 0.93 0.82 - -
zd 33 32 0.98 0.87 - -
zd 33 64 1.08 0.95 - -
zd 33 100 1.27 1.21 - -
zd 33 128 1.43 1.34 - -
zd 33 192 1.87 1.84 - -
zd 33 256 2.39 2.41 - -
d 20 8 0.34 0.35 - -
d 20 32 0.36 0.36 - -
d 20 64 0.37 0.38 - -
d 20 100 0.42 0.43 - -
d 20 128 0.43 0.45 - -
d 20 192 0.51 0.53 - -
d 20 256 0.62 0.66 - -
d 30 8 0.44 0.42 - -
d 30 32 0.46 0.43 - -
d 30 64 0.48 0.46 - -
d 30 100 0.54 0.54 - -
d 30 128 0.55 0.54 - -
d 30 192 0.66 0.67 - -
d 30 256 0.78 0.78 - -
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("rule")
    (d / "r.cu").write_text(
        '#include "update_cl.cuh"\n'
        'extern "C" int split(int cx, int n, int launch, int chains) {\n'
        '  const int ldp = (n + 15) / 16 * 16 + 4;\n'
        '  return cx ? dq::update_split<dq::zd>(n, dq::update_delay<dq::zd>(n, 16, ldp), launch, chains)\n'
        '            : dq::update_split<double>(n, dq::update_delay<double>(n, 16, ldp), launch, chains); }\n')
    so = str(d / "r.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "dqmc-dev_b200", "csrc"), "-o", so, str(d / "r.cu")], check=True)
    return C.CDLL(so).split


def _lane(cx, chains):
    """chains of the largest lane of a default engine"""
    n = max(1, min(4, chains // 32)) if cx else min(8, chains // 32) if chains >= 256 else max(1, min(4, chains // 64))
    return -(-chains // n)


def test_rule_takes_the_fast_side(split, monkeypatch):
    monkeypatch.delenv("DQMC_UPDATE", raising=False)
    for row in ROWS.split("\n"):
        if not row.strip():
            continue
        s, n, ch, *t = row.split()
        cx, n, ch = int(s == "zd"), int(n), int(ch)
        ms = {p: float(x) for p, x in zip((0, 1, 2, 4), t) if x != "-"}
        p = split(cx, n, _lane(cx, ch), ch)
        assert p in ms, (row, p)
        assert ms[p] <= 1.04 * min(ms.values()), (row, p)


@pytest.mark.parametrize("cx", [0, 1])
def test_forced_forms(split, monkeypatch, cx):
    for n in (4, 24, 64, 144, 186):
        for ch in (1, 64, 300):
            monkeypatch.setenv("DQMC_UPDATE", "global")
            assert split(cx, n, ch, ch) == 0
            monkeypatch.setenv("DQMC_UPDATE", "cluster")
            assert split(cx, n, ch, ch) in (1, 2, 4)
    monkeypatch.setenv("DQMC_UPDATE", "cluster")
    assert split(cx, 256, 1, 1) == (0 if cx else 4)
    assert split(cx, 480, 1, 1) == 0
