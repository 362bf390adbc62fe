"""sx_transform_z at every length it takes up to 512, and two beyond (the
library path): one stage and several, each kernel variant's largest and
smallest block, ragged point counts and padded planes; against numpy's FFT of
the same packing in 64 bits.  Tolerance: the FFT's error grows as log2(nz)
roundings, 2^-53 each; 1e-14 of the largest value is about eight times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lengths():
    out = []
    for n in range(2, 513, 2):
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1:
            out.append(n)
    return out + [540, 768]


@pytest.mark.parametrize("nz", _lengths())
def test_transform_every_length(nz):
    import torch
    import semtex_b200 as sx
    for npts, stride in ((1, 1), (77, 80), (300, 301)):
        x = np.random.default_rng(nz + npts).standard_normal((nz, stride))
        d = torch.tensor(x, device="cuda")
        sx.transform_z(d.data_ptr(), nz, stride, npts, +1)
        X = d.cpu().numpy()
        F = np.fft.rfft(x[:, :npts], axis=0) / nz
        want = np.empty((nz, npts))
        want[0], want[1] = F[0].real, F[nz // 2].real
        want[2::2], want[3::2] = F[1:nz // 2].real, F[1:nz // 2].imag
        assert np.abs(X[:, :npts] - want).max() <= 1e-14 * np.abs(want).max()
        assert np.array_equal(X[:, npts:], x[:, npts:])
        sx.transform_z(d.data_ptr(), nz, stride, npts, -1)
        back = d.cpu().numpy()
        assert np.abs(back[:, :npts] - x[:, :npts]).max() <= 1e-14 * np.abs(x).max()
        assert np.array_equal(back[:, npts:], x[:, npts:])


@pytest.mark.parametrize("npts", [99_999, 100_000, 100_033])
def test_transform_128_on_both_sides_of_its_line(npts):
    """Length 128 takes other kernels from 100,000 points on."""
    import torch
    import semtex_b200 as sx
    nz = 128
    x = torch.randn(nz, npts + 6, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    d = x.clone()
    sx.transform_z(d.data_ptr(), nz, npts + 6, npts, +1)
    torch.cuda.synchronize()
    cols = np.r_[0:40, npts - 40:npts]
    F = np.fft.rfft(x[:, cols].cpu().numpy(), axis=0) / nz
    want = np.empty((nz, len(cols)))
    want[0], want[1] = F[0].real, F[nz // 2].real
    want[2::2], want[3::2] = F[1:nz // 2].real, F[1:nz // 2].imag
    assert np.abs(d[:, cols].cpu().numpy() - want).max() <= 1e-14 * np.abs(want).max()
    assert torch.equal(d[:, npts:], x[:, npts:])
    sx.transform_z(d.data_ptr(), nz, npts + 6, npts, -1)
    torch.cuda.synchronize()
    assert float((d - x).abs().max()) <= 1e-14 * float(x.abs().max())


@pytest.mark.parametrize("nz", [96, 128, 256])
def test_first_transform_inside_a_capture(nz):
    """Nothing is set up on the device before a length's first call, so that it
    may be a captured one.  In a process of its own: it is the first."""
    import subprocess
    import sys
    script = f"""
import numpy as np, torch
import semtex_b200 as sx
nz, n = {nz}, 500
x = torch.randn(nz, n, dtype=torch.float64, device="cuda")
d, st, g = x.clone(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
torch.cuda.synchronize()
with torch.cuda.graph(g, stream=st, capture_error_mode="thread_local"):
    sx.transform_z(d.data_ptr(), nz, n, n, 1, stream=st.cuda_stream)
g.replay()
torch.cuda.synchronize()
F = np.fft.rfft(x.cpu().numpy(), axis=0) / nz
X = d.cpu().numpy()
assert np.abs(X[0] - F[0].real).max() <= 1e-14 * np.abs(F).max()
assert np.abs(X[2::2] - F[1:-1].real).max() <= 1e-14 * np.abs(F).max()
assert np.abs(X[3::2] - F[1:-1].imag).max() <= 1e-14 * np.abs(F).max()
"""
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
