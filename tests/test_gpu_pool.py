"""Where band systems' memory comes from and goes: a pool while that is the
quicker way to make and drop them, the device's own allocator beyond.  Systems
of one form solve like the other's, bit for bit, and what is dropped is the
device's again.  In processes of their own: other tests' memory is not in the
counts."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

BEGIN = """
import gc, time
import numpy as np, torch
import semtex_b200 as sx
from semtex_b200.mesh import rect_mesh
MB = 1 << 20
st = torch.cuda.Stream()
def free():
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]
def solve(S, m, nz):
    f = torch.tensor(np.random.default_rng(1).standard_normal((nz, m.nplane)), device="cuda")
    u = torch.zeros_like(f)
    torch.cuda.synchronize()
    S.solve_batched(u.data_ptr(), f.data_ptr(), 0, nz, m.nplane, sx.FP64)
    torch.cuda.synchronize()
    return u
"""


def _run(script):
    r = subprocess.run([sys.executable, "-c", BEGIN + script], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_large_systems_leave_nothing_behind():
    _run("""
m = rect_mesh(64, 64, 11, jitter=0.1, seed=4)
mesh = sx.Mesh(m)
lam = np.linspace(10.0, 40.0, 4)
def systems(modes):
    S = sx.ModalMatrixSys(mesh, base_mode=8, num_modes=modes, method=sx.DIRECT, lambda2_modes=lam[:modes],
                          betak2_modes=np.zeros(modes))
    S.tune(band_cluster=8)
    return S
small = systems(1)  # pooled
u1 = solve(small, m, 2)
del small
before = free()
for _ in range(2):
    S = systems(4)
    assert S.device_bytes > 5 << 30
    u = solve(S, m, 8)
    assert torch.equal(u[:2], u1)
    S.close()
    del u, S
    assert free() > before - 64 * MB
""")


def test_nothing_is_kept_while_the_device_is_short():
    _run("""
m = rect_mesh(24, 24, 9, jitter=0.1, seed=4)
mesh = sx.Mesh(m)
def drop():
    sx.ModalMatrixSys(mesh, num_modes=10, method=sx.DIRECT, lambda2_modes=np.linspace(1.0, 9.0, 10)).close()
drop()
before = free()  # the pool keeps some 600 MB
hold = torch.empty(torch.cuda.mem_get_info()[0] - (6 << 30), dtype=torch.uint8, device="cuda")
time.sleep(0.1)  # the library looks at the device's free memory now and then
drop()
assert free() > before - hold.numel() + 400 * MB  # it kept nothing
""")
