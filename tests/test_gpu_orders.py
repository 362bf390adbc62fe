"""GPU parity of the condensation, the assembly and the condensed forcing at
every order (their kernels are compiled per order): skewed elements, an
essential, a natural and a mixed side, three systems built together, against
the oracle's FP64 direct solve (1e-12, the bar of the other direct-solve
tests)."""
import numpy as np
import pytest

from oracle.oracle import OracleMesh, solve_planes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np_", list(range(3, 13)))
def test_orders_match_oracle(np_):
    import torch

    import semtex_b200 as sx
    from semtex_b200.mesh import rect_mesh
    m = rect_mesh(4, 3, np_, 0.0, 1.0, 0.0, 1.5, jitter=0.2, seed=np_,
                  bc=dict(bottom="D", right=("M", 1.3, 0.4), top="N", left="D"))
    nz, nm = 6, 3
    lam = np.array([5.0, 80.0, 600.0])
    rng = np.random.default_rng(np_)
    f = rng.standard_normal((nz, m.nplane))
    bc = rng.standard_normal((nz, len(m.boundaries), m.np))
    S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=nm, method=sx.DIRECT, lambda2_modes=lam,
                          betak2_modes=np.arange(nm, dtype=np.float64) ** 2)
    uo, _ = solve_planes(OracleMesh(m), 0.0, 1.0, f, bc, lambda2_per_mode=lam)
    sp = [0] + list(range(2, nz))
    fd, u, b = torch.tensor(f, device="cuda"), torch.zeros(f.shape, dtype=torch.float64, device="cuda"), \
        torch.tensor(bc, device="cuda")
    S.solve_batched(u.data_ptr(), fd.data_ptr(), b.data_ptr(), nz, m.nplane, sx.FP64)
    torch.cuda.synchronize()
    a, o = u.cpu().numpy()[sp], uo[sp]
    assert np.linalg.norm(a - o) <= 1e-12 * np.linalg.norm(o)
    assert np.abs(a - o).max() <= 1e-12 * np.abs(o).max()
