"""GPU parity of the essential values where the sides' lines disagree at the
corners they share: the later boundary's value holds, as in the reference's
loop over boundaries (src/field.cpp:994-1019), in every form of the solve,
against the oracle (1e-12 for the FP64 direct forms, 1e-10 for the iterative
ones, the bars of their other tests)."""
import numpy as np
import pytest

from oracle.oracle import OracleMesh, solve_planes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sx():
    import semtex_b200
    return semtex_b200


def _close(a, b, tol):
    assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
    assert np.abs(a - b).max() <= tol * np.abs(b).max()


@pytest.mark.parametrize("walls", ["DDDD", "DNDN", "NDDD"])
@pytest.mark.parametrize("form", ["plain", "batched", "mixed", "jacpcg", "static", "nolines"])
def test_corner_values_are_the_later_boundarys(sx, walls, form):
    import torch

    from semtex_b200.mesh import rect_mesh
    m = rect_mesh(3, 4, 6, 0.0, 1.0, 0.0, 1.0, jitter=0.15, seed=6,
                  bc=dict(zip(("bottom", "right", "top", "left"), walls)))
    rng = np.random.default_rng(5)
    nz, lam = 4, np.array([3e4, 5e4])
    f = rng.standard_normal((nz, m.nplane))
    bc = None if form == "nolines" else rng.standard_normal((nz, len(m.boundaries), m.np))
    S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=2, method=sx.JACPCG if form == "jacpcg" else sx.DIRECT,
                          lambda2_modes=lam, betak2_modes=np.zeros(2))
    fd = torch.tensor(f, device="cuda")
    u = torch.zeros_like(fd)
    b = 0 if bc is None else torch.tensor(bc, device="cuda")
    ptrs = (u.data_ptr(), fd.data_ptr(), b if bc is None else b.data_ptr(), nz, m.nplane)
    if form == "mixed":
        S.tune(mixed_route=sx.ROUTE_CG, inner_iters=40)
        S.solve_batched(*ptrs, sx.MIXED_FP32, 1e-13, 30)
    elif form == "static":
        S.solve_device_static(*ptrs)
    elif form in ("plain", "jacpcg"):
        S.solve_device(*ptrs, tol_rel=1e-12, step_max=5000)
    else:
        S.solve_batched(*ptrs, sx.FP64)
    torch.cuda.synchronize()
    uo, _ = solve_planes(OracleMesh(m), 0.0, 0.0, f, bc, lambda2_per_mode=lam)
    sp = [0, 2, 3]
    _close(u.cpu().numpy()[sp], uo[sp], 1e-10 if form in ("mixed", "jacpcg") else 1e-12)
