"""radonusfft's two adjoints against the complex128 direct sums that they
approximate, at the operator's own polar tables and at the smallest and odd
sizes of the slice blocks.

Tolerance 1e-6: the gridding window's error (rms below 5e-8 per axis) and FP32
rounding of two FFT passes and of sums over the points of a cell, each below
log2(2N) 2^-24 = 6e-7, as the forward's."""
import numpy as np
import pytest

from oracle.usfft import checker1, circ_mask

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def adjoint_sums(g, x, y, n, exact):
    """f [nz, n, n] from g [ntheta, nz, n]: the detector rows padded (by their edge
    values, or by zeros: the adjoint of the forward's crop), centred FFT, sum over
    the polar points, mask; then the crop, or the fold of the replicated margin."""
    N, (ntheta, nz, _) = n * 3 // 2, g.shape
    c0 = N // 6
    idx = np.clip(np.arange(N), c0, 5 * N // 6 - 1) - c0
    gl = np.zeros((ntheta, nz, N), np.complex128)
    if exact:
        gl[:, :, c0:c0 + n] = g
    else:
        gl[:] = g[:, :, idx]
    s1 = checker1(N)
    gl = np.fft.fft(gl * s1, axis=-1) * s1 / N
    t = np.arange(N) - N // 2
    f = np.zeros((nz, N, N), np.complex128)
    for a in range(ntheta):
        ex, ey = (np.exp(2j * np.pi * v[a].astype(np.float64)[:, None] * t) for v in (x, y))   # [k, t]
        f += np.einsum("zk,ky,kx->zyx", gl[a], ey, ex, optimize=True)
    f *= circ_mask(N)
    if not exact:
        return f[:, c0:c0 + n, c0:c0 + n]
    fold = np.zeros((n, N))
    fold[idx, np.arange(N)] = 1.0
    return fold @ f @ fold.T


@pytest.mark.parametrize("n,nz,nt", [(8, 1, 3), (8, 17, 5), (16, 7, 1), (32, 9, 24), (64, 16, 13), (128, 3, 7)])
def test_radon_adjoints_against_direct_sums(n, nz, nt):
    from ptychotomo_b200 import radonusfft
    rng = np.random.default_rng(n + 10 * nz)
    theta = rng.uniform(-np.pi, np.pi, nt).astype(np.float32)
    g = (rng.standard_normal((nt, nz, n)) + 1j * rng.standard_normal((nt, nz, n))).astype(np.complex64)
    op = radonusfft(nt, nz, n)
    op.setobj(torch.from_numpy(theta).cuda())
    x = torch.empty((nt, op.N), dtype=torch.float32, device="cuda")
    y = torch.empty_like(x)
    op.get_xy(x, y)
    gd = torch.from_numpy(g).cuda()
    for exact, call in ((False, op.adj), (True, op.adj_exact)):
        f = torch.full((nz, n, n), float("nan"), dtype=torch.complex64, device="cuda")
        call(f, gd)
        ref = adjoint_sums(g, x.cpu().numpy(), y.cpu().numpy(), n, exact)
        assert np.linalg.norm(f.cpu().numpy() - ref) <= 1e-6 * np.linalg.norm(ref)
