"""GPU parity of the band sweeps where their hand-offs change form: one, two
and three block columns; a band of one tile, of the leader's own tiles, and
wide enough that every rank of the widest cluster owns tiles; one right-hand
side and two; every kind of cluster (one CTA; a leader share; more CTAs than
tiles), against the oracle's FP64 direct solve (1e-12, the bar of the other
direct-solve tests: these systems' condition times 1e-16, with a margin)."""
import numpy as np
import pytest

from oracle.oracle import OracleMesh, solve_planes

pytestmark = pytest.mark.gpu

TOL = 1e-12
#: nx, ny, np, planes: block columns x tiles right of the diagonal
MESHES = [(2, 2, 4, 1),     # 1 x 0
          (3, 3, 8, 6),     # 2 x 1
          (5, 4, 8, 4),     # 4 x 2
          (16, 4, 9, 6),    # 13 x 2
          (20, 18, 10, 4)]  # 91 x 9


@pytest.fixture(scope="module")
def sx():
    import semtex_b200
    return semtex_b200


@pytest.mark.parametrize("nx,ny,np_,nz", MESHES)
@pytest.mark.parametrize("cluster,stages,lead", [(0, 0, 0), (1, 1, 0), (2, 4, 0), (3, 2, 2), (5, 3, 1), (9, 2, 4),
                                                 (16, 1, 1)])
def test_band_sweeps_match_oracle(sx, nx, ny, np_, nz, cluster, stages, lead):
    import torch

    from semtex_b200.mesh import rect_mesh
    m = rect_mesh(nx, ny, np_, 0.0, 1.0, 0.0, 1.0, jitter=0.1, seed=4)
    nm = max(nz // 2, 1)
    lam = np.linspace(40.0, 900.0, nm)
    f = np.random.default_rng(nx).standard_normal((nz, m.nplane))
    S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=nm, method=sx.DIRECT, lambda2_modes=lam,
                          betak2_modes=np.arange(nm, dtype=np.float64) ** 2)
    S.tune(band_cluster=cluster, band_stages=stages, band_lead=lead)
    uo, _ = solve_planes(OracleMesh(m), 0.0, 1.0, f, None, lambda2_per_mode=lam)
    sp = [0] + list(range(2, nz))
    f0 = torch.tensor(f, device="cuda")
    fd, u = torch.empty_like(f0), torch.zeros_like(f0)
    for _ in range(2):  # the first call, then the replayed graph
        fd.copy_(f0)
        u.zero_()
        S.solve_batched(u.data_ptr(), fd.data_ptr(), 0, nz, m.nplane, sx.FP64)
        torch.cuda.synchronize()
        S.status()
        a, b = u.cpu().numpy()[sp], uo[sp]
        assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)
        assert np.abs(a - b).max() <= TOL * np.abs(b).max()


def test_wide_band_equals_narrow(sx):
    """A numbering whose band is too wide for a window of all its blocks in
    shared memory (older blocks are read through L2, the diagonal solves run
    between the sweeps): the solution of the same systems under the narrow
    numbering, which the tests above hold against the oracle, to the rounding
    of a full elimination (7,700 unknowns of condition about 1e3: 1e-11)."""
    import dataclasses

    import torch

    from semtex_b200.mesh import rect_mesh
    nz, lam = 4, np.array([300.0, 700.0])
    narrow = rect_mesh(28, 26, 7, 0.0, 1.0, 0.0, 1.0, jitter=0.1, seed=4)
    new = np.arange(narrow.nglobal)
    new[:narrow.nsolve] = np.random.default_rng(8).permutation(narrow.nsolve)
    wide = dataclasses.replace(narrow, btog=new[narrow.btog].astype(np.int32), nband=narrow.nsolve)
    assert -(-(wide.nband - 1) // 64) > 110  # tiles a block column: beyond the window
    f = torch.tensor(np.random.default_rng(3).standard_normal((nz, narrow.nplane)), device="cuda")
    sols = []
    # the last two leave the leader the tile 64 block columns back, whose block's
    # place in the window is the next one stored to, and little after it
    for m, cases in ((narrow, ((0, 0),)), (wide, ((0, 0), (1, 0), (2, 2), (7, 1), (2, 31), (3, 62)))):
        S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=2, method=sx.DIRECT, lambda2_modes=lam, betak2_modes=np.zeros(2))
        for cluster, lead in cases:
            S.tune(band_cluster=cluster, band_stages=4 if lead > 2 else 0, band_lead=lead)
            fd, u = f.clone(), torch.zeros_like(f)
            S.solve_batched(u.data_ptr(), fd.data_ptr(), 0, nz, m.nplane, sx.FP64)
            torch.cuda.synchronize()
            S.status()
            sols.append(u)
    for u in sols[1:]:
        assert float((u - sols[0]).norm()) <= 1e-11 * float(sols[0].norm())


@pytest.mark.parametrize("nm", [148, 149, 300])
def test_more_systems_than_sms(sx, nm):
    """One launch over as many systems as the chip has SMs, and more: the rest
    wait for a place, in the default schedule and in one of three CTAs a system.
    Every system against the oracle."""
    import torch

    from semtex_b200.mesh import rect_mesh
    m = rect_mesh(5, 4, 7, 0.0, 1.0, 0.0, 1.0, jitter=0.1, seed=4)
    nz, lam = 2 * nm, np.linspace(40.0, 900.0, nm)
    f = np.random.default_rng(nm).standard_normal((nz, m.nplane))
    S = sx.ModalMatrixSys(sx.Mesh(m), num_modes=nm, method=sx.DIRECT, lambda2_modes=lam, betak2_modes=np.zeros(nm))
    uo, _ = solve_planes(OracleMesh(m), 0.0, 0.0, f, None, lambda2_per_mode=lam)
    sp = [0] + list(range(2, nz))
    for cluster in (0, 3):
        S.tune(band_cluster=cluster)
        fd = torch.tensor(f, device="cuda")
        u = torch.zeros_like(fd)
        torch.cuda.synchronize()
        S.solve_batched(u.data_ptr(), fd.data_ptr(), 0, nz, m.nplane, sx.FP64)
        torch.cuda.synchronize()
        S.status()
        a, b = u.cpu().numpy()[sp], uo[sp]
        assert (np.linalg.norm(a - b, axis=1) <= TOL * np.linalg.norm(b, axis=1)).all()
