"""The kernel count a JACPCG solve reports: 11 launches a plane and 9 an
iteration, and where the mesh has essential nodes one more zeroing at each of
four places (three before the iterations, one in each); boundary lines add
none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walls", ["D", "N"])
@pytest.mark.parametrize("lines", [False, True])
def test_jacpcg_launches(walls, lines):
    import torch

    import semtex_b200 as sx
    from semtex_b200.mesh import rect_mesh
    m = rect_mesh(3, 4, 6, bc=dict.fromkeys(("bottom", "right", "top", "left"), walls))
    S = sx.ModalMatrixSys(sx.Mesh(m), lambda2=1e3, num_modes=1, method=sx.JACPCG)
    f = torch.tensor(np.random.default_rng(3).standard_normal((1, m.nplane)), device="cuda")
    u = torch.zeros_like(f)
    bc = torch.ones((1, len(m.boundaries), m.np), dtype=torch.float64, device="cuda")
    st = S.solve_device(u.data_ptr(), f.data_ptr(), bc.data_ptr() if lines else 0, 1, m.nplane, 1e-10, 500)
    zr = int(walls == "D")
    assert 0 < st["iterations_total"] < 500
    assert st["kernel_launches"] == 11 + 3 * zr + (9 + zr) * st["iterations_total"]
