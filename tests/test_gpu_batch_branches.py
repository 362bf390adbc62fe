"""More members in a batch's FP64 solve than its captured graph has branches:
every member equals its own batched solve bit for bit, in the call that
enqueues the kernels, in the one that captures the graph and in one that
replays it, each with new forcing; with other buffers in between; and in a
capture of the caller's own."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [2, 16, 17, 35])
def test_members_beyond_the_branches(members):
    import torch

    import semtex_b200 as sx
    from semtex_b200.workloads import small_channel
    ws = [small_channel(nx=2 + i % 4, ny=2 + i % 3, np_=4 + i % 5, nz=2 + 2 * (i % 3), lam=1e3, seed=i)
          for i in range(members)]
    S = [sx.ModalMatrixSys(sx.Mesh(w.mesh), num_modes=w.num_modes, method=sx.DIRECT, lambda2_modes=w.lambda2,
                           betak2_modes=w.betak2) for w in ws]
    for s in S:
        s.tune(band_cluster=2)  # one split of the tiles, alone and in the batch
    fs = [torch.empty(w.forcing.shape, dtype=torch.float64, device="cuda") for w in ws]
    us = [torch.zeros_like(f) for f in fs]
    B = sx.Batch()
    for scale in (1.0, -2.5, 0.5):
        want = []
        for s, w, f in zip(S, ws, fs):
            f.copy_(torch.tensor(w.forcing) * scale)
            u = torch.zeros_like(f)
            s.solve_batched(u.data_ptr(), f.data_ptr(), 0, w.nz, w.mesh.nplane, sx.FP64)
            torch.cuda.synchronize()
            want.append(u)
            f.copy_(torch.tensor(w.forcing) * scale)
        torch.cuda.synchronize()
        B.solve([(s, u.data_ptr(), f.data_ptr(), None, w.nz, w.mesh.nplane) for s, u, f, w in zip(S, us, fs, ws)],
                sx.FP64)
        torch.cuda.synchronize()
        for u, v in zip(us, want):
            assert torch.equal(u, v)


def test_new_buffers_and_a_callers_capture():
    import torch

    import semtex_b200 as sx
    from semtex_b200.workloads import small_channel
    ws = [small_channel(nx=2 + i, ny=3, np_=5 + i, nz=4, lam=1e3, seed=i) for i in range(3)]
    S = [sx.ModalMatrixSys(sx.Mesh(w.mesh), num_modes=w.num_modes, method=sx.DIRECT, lambda2_modes=w.lambda2,
                           betak2_modes=w.betak2) for w in ws]
    f0 = [torch.tensor(w.forcing, device="cuda") for w in ws]
    sets = [([torch.empty_like(f) for f in f0], [torch.empty_like(f) for f in f0]) for _ in range(2)]
    B, st, want = sx.Batch(), torch.cuda.Stream(), None

    def solve(fs, us):
        B.solve([(s, u.data_ptr(), f.data_ptr(), None, w.nz, w.mesh.nplane) for s, u, f, w in zip(S, us, fs, ws)],
                sx.FP64, stream=st.cuda_stream)

    def restore(fs, us):
        for f, g, u in zip(fs, f0, us):
            f.copy_(g)
            u.zero_()
        torch.cuda.synchronize()

    for k in (0, 0, 1, 0, 1, 1, 1, 0):
        restore(*sets[k])
        solve(*sets[k])
        torch.cuda.synchronize()
        got = [u.clone() for u in sets[k][1]]
        want = want or got
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    g = torch.cuda.CUDAGraph()  # the last call was the first with its buffers
    with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
        solve(*sets[0])
    for _ in range(2):
        restore(*sets[0])
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(sets[0][1], want))
    assert float(want[0].abs().max()) > 0.0
