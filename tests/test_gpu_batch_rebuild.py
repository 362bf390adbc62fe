"""A batch kept over members that are closed and built anew with other
constants (a changed time step): the new objects, and their workspaces, may be
given the old ones' addresses, and nothing kept for the old ones may answer for
them.  Every solution equals the new member's own solve: bit for bit in FP64
(one band-sweep schedule for both), to 1e-10 in the mixed form (its bar)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_members_built_anew(form):
    import torch

    import semtex_b200 as sx
    from semtex_b200.mesh import rect_mesh
    ms = [rect_mesh(4, 3, 8), rect_mesh(3, 5, 6)]
    meshes, nz = [sx.Mesh(m) for m in ms], 6
    prec = sx.FP64 if form == "fp64" else sx.MIXED_FP32
    f0 = [torch.tensor(np.random.default_rng(i).standard_normal((nz, m.nplane)), device="cuda")
          for i, m in enumerate(ms)]
    fs, us = [torch.empty_like(f) for f in f0], [torch.zeros_like(f) for f in f0]
    B, last = sx.Batch(), None
    for lam in (2e3, 4e4, 3e3, 6e4, 2e3):
        S = [sx.ModalMatrixSys(mesh, num_modes=3, method=sx.DIRECT if form == "fp64" else sx.JACPCG,
                               lambda2_modes=np.full(3, lam), betak2_modes=np.arange(3.0)) for mesh in meshes]
        for s in S:
            s.tune(band_cluster=2, inner_iters=40)
        for _ in range(3):  # the first call with these members, and what is replayed from it
            for f, g, u in zip(fs, f0, us):
                f.copy_(g)
                u.zero_()
            torch.cuda.synchronize()
            B.solve([(s, u.data_ptr(), f.data_ptr(), None, nz, m.nplane) for s, u, f, m in zip(S, us, fs, ms)],
                    prec, 1e-13, 40)
            torch.cuda.synchronize()
            got = [u.clone() for u in us]
            for s, m, g, u in zip(S, ms, f0, got):
                f, v = g.clone(), torch.zeros_like(g)
                torch.cuda.synchronize()
                s.solve_batched(v.data_ptr(), f.data_ptr(), 0, nz, m.nplane, prec, 1e-13, 40)
                torch.cuda.synchronize()
                if form == "fp64":
                    assert torch.equal(u, v)
                else:
                    assert float((u - v).norm()) <= 1e-10 * float(v.norm())
        assert last is None or float((got[0] - last).abs().max()) > 1e-6 * float(last.abs().max())
        last = got[0]
        for s in S:
            s.close()
