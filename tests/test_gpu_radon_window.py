"""radonusfft against the complex128 direct sums it approximates, at the
operator's own polar tables: the smallest and odd widths of the gridding
window's tiles and of the slice blocks (1, 8 and 16 slices +- 1).

Tolerance 1e-6: the window's error (rms below 5e-8 per axis) and FP32 rounding
of two FFT passes and 64 + 8 sums, each below log2(2N) 2^-24 = 6e-7."""
import numpy as np
import pytest

from oracle.nudft import radon_fwd_exact

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,nt", [(8, 1, 3), (8, 17, 5), (16, 7, 1), (32, 9, 24), (64, 16, 13), (128, 3, 7)])
def test_radon_fwd_against_direct_sums(n, nz, nt):
    from ptychotomo_b200 import radonusfft
    rng = np.random.default_rng(n + nz)
    theta = rng.uniform(-np.pi, np.pi, nt).astype(np.float32)
    f = (rng.standard_normal((nz, n, n)) + 1j * rng.standard_normal((nz, n, n))).astype(np.complex64)
    op = radonusfft(nt, nz, n)
    op.setobj(torch.from_numpy(theta).cuda())
    x = torch.empty((nt, op.N), dtype=torch.float32, device="cuda")
    y = torch.empty_like(x)
    op.get_xy(x, y)
    g = torch.empty((nt, nz, n), dtype=torch.complex64, device="cuda")
    fd = torch.from_numpy(f).cuda()
    op.fwd(g, fd)
    ref = radon_fwd_exact(f, theta, n, xy=(x.cpu().numpy(), y.cpu().numpy()))
    assert np.linalg.norm(g.cpu().numpy() - ref) <= 1e-6 * np.linalg.norm(ref)
    # the exact adjoint is the adjoint of that: <R f, h> = <f, R^T h>
    h = torch.from_numpy((rng.standard_normal(g.shape) + 1j * rng.standard_normal(g.shape)).astype(np.complex64)).cuda()
    back = torch.empty_like(fd)
    op.adj_exact(back, h)
    a = torch.vdot(g.flatten().cdouble(), h.flatten().cdouble())
    b = torch.vdot(fd.flatten().cdouble(), back.flatten().cdouble())
    assert abs(a - b) <= 1e-6 * g.cdouble().norm() * h.cdouble().norm()
