"""Status of the delayed update: a launch that the runtime refuses ends the call
with an error instead of a sweep without its update, and an error word that the
kernel has set (a wait that ran out) reaches the seam's caller.

Both come from a fake: the library's objects are linked once more with calls of
the runtime wrapped, and when they are told to, the launch returns an error code
without launching and the wait finds the error word set.
"""
import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_gpu_update_window import _inputs

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "dqmc-dev_b200")
DQMC_E_CUDA, DQMC_E_DEVICE = -11, -13

FAKE = r"""
#include <cuda_runtime.h>
extern "C" {
int fake_refuse = 0;      /* launches to refuse */
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a);
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **a)
{
	if (fake_refuse > 0) {
		fake_refuse--;
		return cudaErrorLaunchOutOfResources;
	}
	return __real_cudaLaunchKernelExC(c, f, a);
}
unsigned fake_word = 0;   /* what the next wait on a stream leaves in the call's error word */
static unsigned *word;
cudaError_t __real_cudaHostAlloc(void **p, size_t n, unsigned flags);
cudaError_t __wrap_cudaHostAlloc(void **p, size_t n, unsigned flags)
{
	const cudaError_t e = __real_cudaHostAlloc(p, n, flags);
	if (e == cudaSuccess && n == sizeof(unsigned)) word = (unsigned *)*p;
	return e;
}
cudaError_t __real_cudaStreamSynchronize(cudaStream_t st);
cudaError_t __wrap_cudaStreamSynchronize(cudaStream_t st)
{
	const cudaError_t e = __real_cudaStreamSynchronize(st);
	if (fake_word && word) {
		*word |= fake_word;
		fake_word = 0;
	}
	return e;
}
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    objs = sorted(glob.glob(os.path.join(PKG, "build", "*.o")))
    if not objs or shutil.which("nvcc") is None:
        pytest.skip("no objects of the library to link")
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.cu").write_text(FAKE)
    so = str(d / "libfake.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "static",
                    "-Xcompiler", "-fPIC", "-Xlinker", "--wrap=cudaLaunchKernelExC", "-Xlinker", "--wrap=cudaHostAlloc", "-Xlinker",
                    "--wrap=cudaStreamSynchronize", "-o", so,
                    str(d / "fake.cu")] + objs, check=True)
    from dqmc_b200 import lib
    own, lib._lib = lib._lib, None
    try:
        h = lib.load(so)
    finally:
        lib._lib = own
    return h, C.c_int.in_dll(h, "fake_refuse")


def _seam(h, N, form, monkeypatch):
    import torch
    monkeypatch.setenv("DQMC_UPDATE", form)
    _, G, del_, hs, rng = _inputs(N, 2, 0, 11)
    dG = torch.from_numpy(np.ascontiguousarray(G.swapaxes(-1, -2))).cuda()
    dhs, drng = torch.from_numpy(hs.copy()).cuda(), torch.from_numpy(rng.view(np.int64).copy()).cuda()
    ddel, dph = torch.from_numpy(del_).cuda(), torch.ones(2, dtype=torch.float64, device="cuda")
    rc = h.dqmc_gpu_update_delayed(2, N, 16, 0, ddel.data_ptr(), drng.data_ptr(), dhs.data_ptr(),
                                   dG.data_ptr(), dph.data_ptr(), None)
    return rc, dG.cpu().numpy(), np.ascontiguousarray(G.swapaxes(-1, -2))


@pytest.mark.parametrize("form", ["global", "cluster"])
def test_seam_reports_a_refused_launch(fake, form, monkeypatch):
    h, refuse = fake
    refuse.value = 1
    rc, got, G = _seam(h, 32, form, monkeypatch)
    assert refuse.value == 0
    assert rc == DQMC_E_CUDA
    assert np.array_equal(got, G)          # nothing ran on it
    rc, got, G = _seam(h, 32, form, monkeypatch)
    assert rc == 0 and not np.array_equal(got, G)


@pytest.mark.parametrize("form", ["global", "cluster"])
def test_sweep_reports_a_refused_update(fake, form, monkeypatch):
    """refused while the sweep's graph is captured: the call fails and nothing is
    kept of it; the next sweeps capture again and are those of a fresh engine"""
    from dqmc_b200 import engine, gen, lib
    h, refuse = fake
    monkeypatch.setattr(lib, "_lib", h)
    monkeypatch.setenv("DQMC_UPDATE", form)
    d = gen.make_sim(Nx=6, Ny=5, U=4.0, mu=-0.5, dt=0.1, L=10, n_matmul=5, n_delay=8, period_eqlt=5,
                     n_sweep_warm=0, n_sweep_meas=4, seed=3)
    out = []
    for n_refuse in (0, 1):
        s = engine.SimData(dict(d))
        e = engine.Engine([s])
        e.init()
        if n_refuse:
            refuse.value = n_refuse
            with pytest.raises(RuntimeError):
                e.sweeps(1)
            assert refuse.value == 0
        e.sweeps(2)
        e.pull()
        assert e.errors() == 0
        out.append((s.hs.copy(), s.rng.copy(), s.eq_acc.copy()))
        e.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("form", ["global", "cluster"])
def test_seam_reports_the_kernels_error_word(fake, form, monkeypatch):
    h, _ = fake
    word = C.c_uint.in_dll(h, "fake_word")
    word.value = 4
    rc, _, _ = _seam(h, 32, form, monkeypatch)
    assert word.value == 0 and rc == DQMC_E_DEVICE
    rc, _, _ = _seam(h, 32, form, monkeypatch)
    assert rc == 0
