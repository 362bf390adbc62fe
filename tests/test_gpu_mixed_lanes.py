"""GPU parity of the mixed form for every way its lanes are filled: 32, 16 or 8
planes a chunk, one chunk and several, element counts that leave the last
group of a block short, straight and curved elements side by side, alone and
in a multi-mesh batch; against the oracle (1e-10, the mixed form's bar).
Blocks hold several elements only where 32 planes a chunk would give an SM more
of them, so the meshes that are to be packed have more than 148 elements."""
import numpy as np
import pytest

from oracle.oracle import OracleMesh, solve_planes

pytestmark = pytest.mark.gpu

TOL = 1e-10


@pytest.fixture(scope="module")
def sx():
    import semtex_b200
    return semtex_b200


def _mesh(nx, ny, np_, walls="D"):
    """A rectangle whose right half is distorted: both kinds of element."""
    from semtex_b200.mesh import rect_mesh
    X, Y = np.meshgrid(np.linspace(0, 1, nx + 1), np.linspace(0, 1, ny + 1), indexing="xy")
    X, Y = X.copy(), Y.copy()
    inner = np.zeros(X.shape, dtype=bool)
    inner[1:-1, nx // 2 + 1:-1] = True
    X[inner] += 0.2 / nx
    Y[inner] -= 0.15 / ny
    return rect_mesh(nx, ny, np_, vertex_xy=(X, Y), bc={"bottom": walls, "top": "D"})


def _problem(m, nz, seed):
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((nz, m.nplane))
    bc = rng.standard_normal((nz, len(m.boundaries), 1)) * np.ones(m.np)
    nm = max(nz // 2, 1)
    return f, bc, np.linspace(1e5, 3e5, nm)


def _check(m, nz, f, bc, lam, u):
    uo, _ = solve_planes(OracleMesh(m), 0.0, 0.0, f, bc, lambda2_per_mode=lam)
    for p in ([0] if nz == 1 else [0] + list(range(2, nz))):
        assert np.linalg.norm(u[p] - uo[p]) <= TOL * np.linalg.norm(uo[p]), p
        assert np.abs(u[p] - uo[p]).max() <= TOL * np.abs(uo[p]).max(), p
    if nz > 1:
        assert np.all(u[1] == 0.0)


SIZES = [(1, 1, 1, 5, "D"), (1, 3, 3, 3, "D"), (2, 3, 3, 4, "N"), (8, 5, 1, 12, "D"), (10, 3, 3, 6, "D"),
         (16, 3, 5, 11, "N"), (18, 5, 1, 7, "D"), (24, 3, 3, 9, "N"), (32, 5, 1, 5, "D"), (34, 3, 3, 5, "D")]
#: 8, 8, 8, 16, 16, 8, 8, 8 planes a chunk, and 16 at the lowest order
PACKED = [(1, 19, 9, 5, "D"), (2, 19, 9, 4, "N"), (8, 19, 9, 12, "D"), (10, 17, 9, 6, "D"), (16, 17, 11, 11, "N"),
          (18, 19, 9, 7, "D"), (24, 19, 9, 9, "N"), (34, 13, 13, 5, "D"), (10, 17, 9, 3, "D")]


@pytest.mark.parametrize("nz,nx,ny,np_,walls", SIZES + PACKED)
def test_lane_layouts_match_oracle(sx, nz, nx, ny, np_, walls):
    import torch
    m = _mesh(nx, ny, np_, walls)
    f, bc, lam = _problem(m, nz, nz)
    S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=len(lam), method=sx.JACPCG, lambda2_modes=lam,
                          betak2_modes=np.zeros(len(lam)))
    S.tune(inner_iters=30)
    fd, b = torch.tensor(f, device="cuda"), torch.tensor(bc, device="cuda")
    u = torch.zeros_like(fd)
    S.solve_batched(u.data_ptr(), fd.data_ptr(), b.data_ptr(), nz, m.nplane, sx.MIXED_FP32, 1e-13, 40)
    torch.cuda.synchronize()
    _check(m, nz, f, bc, lam, u.cpu().numpy())


@pytest.mark.parametrize("sizes", [SIZES, SIZES + PACKED], ids=["wide", "packed"])
def test_lane_layouts_in_one_batch(sx, sizes):
    import torch
    B, members, probs = sx.Batch(), [], []
    for nz, nx, ny, _, walls in sizes:  # one order: one launch over every layout
        m = _mesh(nx, ny, 6, walls)
        f, bc, lam = _problem(m, nz, 100 + nz)
        S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=len(lam), method=sx.JACPCG, lambda2_modes=lam,
                              betak2_modes=np.zeros(len(lam)))
        S.tune(inner_iters=30)
        t = [torch.tensor(a, device="cuda") for a in (f, bc)]
        u = torch.zeros_like(t[0])
        members.append((S, u.data_ptr(), t[0].data_ptr(), t[1].data_ptr(), nz, m.nplane))
        probs.append((m, nz, f, bc, lam, u, t))
    B.solve(members, sx.MIXED_FP32, 1e-13, 40)
    torch.cuda.synchronize()
    for m, nz, f, bc, lam, u, _ in probs:
        _check(m, nz, f, bc, lam, u.cpu().numpy())
