"""Systems built, used and dropped in turn: their memory comes from a pool
that later systems reuse, a build waits once for all its systems, and the
batched form enqueues its first call as it is and replays a graph from the
second on.  Every solution equals the first one bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sx():
    import semtex_b200
    return semtex_b200


def _systems(sx, w, mesh):
    return sx.ModalMatrixSys(mesh, num_modes=w.num_modes, method=sx.DIRECT, lambda2_modes=w.lambda2,
                             betak2_modes=w.betak2)


def test_build_solve_drop_on_another_stream(sx):
    """The solve is on a stream that does not wait for the default one, and the
    systems are dropped without waiting for it: their memory must not be
    reused before it is done."""
    import torch
    from semtex_b200.workloads import small_channel
    w = small_channel(nx=12, ny=9, np_=8, nz=10, lam=50.0, seed=2)
    mesh = sx.Mesh(w.mesh)
    f0 = torch.tensor(w.forcing, device="cuda")
    f, us, st = torch.empty_like(f0), [], torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):
        S = _systems(sx, w, mesh)
        us.append(torch.zeros_like(f0))
        torch.cuda.synchronize()
        for _ in range(3):
            with torch.cuda.stream(st):
                f.copy_(f0)
            S.solve_batched(us[-1].data_ptr(), f.data_ptr(), 0, w.nz, w.mesh.nplane, stream=st.cuda_stream)
        S.close()
    torch.cuda.synchronize()
    for u in us[1:]:
        assert torch.equal(u, us[0])
    assert float(us[0].abs().max()) > 0.0


def test_second_call_inside_a_capture(sx):
    import torch
    from semtex_b200.workloads import small_channel
    w = small_channel(nx=6, ny=5, np_=7, nz=6, lam=50.0, seed=2)
    S = _systems(sx, w, sx.Mesh(w.mesh))
    f0 = torch.tensor(w.forcing, device="cuda")
    f, u = f0.clone(), torch.zeros_like(f0)
    st = torch.cuda.Stream()
    args = (u.data_ptr(), f.data_ptr(), 0, w.nz, w.mesh.nplane)
    torch.cuda.synchronize()
    S.solve_batched(*args, stream=st.cuda_stream)
    st.synchronize()
    want = u.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        S.solve_batched(*args, stream=st.cuda_stream)
    for _ in range(2):
        f.copy_(f0)
        u.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(u, want)
