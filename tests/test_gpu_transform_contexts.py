"""sx_transform_z in a second context of a process, as on a second device: a
kernel's shared-memory limit holds for one context's copy of it, and lengths
whose block takes more than 48 KB fail where it was not raised.  The second
context is made through the driver, in a process of its own; against numpy's
FFT (1e-14 of the largest value, as for the lengths elsewhere)."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes as C, sys
import numpy as np, torch
import semtex_b200 as sx
nz, n = int(sys.argv[1]), 96
x = np.random.default_rng(nz).standard_normal((nz, n))
d = torch.tensor(x, device="cuda")
sx.transform_z(d.data_ptr(), nz, n, n, 1)
X = d.cpu().numpy()
F = np.fft.rfft(x, axis=0) / nz
want = np.empty_like(x)
want[0], want[1] = F[0].real, F[-1].real
want[2::2], want[3::2] = F[1:-1].real, F[1:-1].imag
cu = C.CDLL("libcuda.so.1")
def do(name, *a):
    assert getattr(cu, name)(*a) == 0, name
ctx, p = C.c_void_p(), C.c_uint64()
do("cuCtxCreate_v2", C.byref(ctx), 0, 0)
do("cuMemAlloc_v2", C.byref(p), C.c_size_t(x.nbytes))
do("cuMemcpyHtoD_v2", p, C.c_void_p(x.ctypes.data), C.c_size_t(x.nbytes))
sx.transform_z(p.value, nz, n, n, 1)
do("cuCtxSynchronize")
Y = np.empty_like(x)
do("cuMemcpyDtoH_v2", C.c_void_p(Y.ctypes.data), p, C.c_size_t(x.nbytes))
sx.transform_z(p.value, nz, n, n, -1)
do("cuCtxSynchronize")
Z = np.empty_like(x)
do("cuMemcpyDtoH_v2", C.c_void_p(Z.ctypes.data), p, C.c_size_t(x.nbytes))
do("cuMemFree_v2", p)
do("cuCtxDestroy_v2", ctx)
for a, b in ((X, want), (Y, want), (Z, x)):
    assert np.abs(a - b).max() <= 1e-14 * np.abs(b).max()
"""


@pytest.mark.parametrize("nz", [24, 96, 128, 240, 256, 512])  # one length of each kernel variant
def test_second_context(nz):
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(nz)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
