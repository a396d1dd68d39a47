"""The ptycho kernels against the oracle at the sizes where their trips, lines
and tables can go wrong: odd probes and probes of one pixel, one scan, odd
numbers of scans (two frames per trip), skipped scans anywhere, probes whose
rows fill the shared table partly, and the residual's out-of-range values.

Tolerances: two FFT passes of det <= 128 points round by at most
14 x 2^-24 = 8e-7 relative to the frame and the sums over scans add as much:
2e-6; the residual of counts within a factor of two of |f|^2 is a quarter of f,
so four times that: 1e-5."""
import numpy as np
import pytest

from oracle.ptycho import PtychoFFT

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def crand(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


CASES = [  # ntheta, nz, n, nscan, det, nprb
    (1, 20, 19, 1, 16, 7), (3, 40, 33, 3, 16, 16), (2, 40, 37, 5, 32, 1), (2, 41, 40, 4, 32, 31), (3, 50, 70, 7, 32, 32),
    (1, 70, 66, 1, 64, 16), (2, 70, 66, 5, 64, 17), (2, 66, 70, 6, 64, 33), (2, 70, 71, 3, 64, 63), (2, 90, 64, 9, 64, 64),
    (1, 130, 131, 1, 128, 128), (2, 131, 130, 5, 128, 127), (2, 130, 140, 4, 128, 40), (1, 129, 130, 3, 128, 112)]


@pytest.mark.parametrize("nt,nz,n,ns,det,P", CASES)
@pytest.mark.parametrize("parts", [None, "1", "2"])
def test_frames_against_oracle(nt, nz, n, ns, det, P, parts, monkeypatch):
    from ptychotomo_b200 import ptychofft
    if parts:
        monkeypatch.setenv("PT_PTYCHO_ADJ_PARTS", parts)
    rng = np.random.default_rng(det + 1000 * P + ns)
    scan = np.stack([rng.uniform(0, n - P, (nt, ns)), rng.uniform(0, nz - P, (nt, ns))]).astype(np.float32)
    if ns > 2:
        scan[:, 0, 1] = -1
        scan[:, -1, ns - 1] = -1
    prb, psi = crand(rng, (P, P)), crand(rng, (nt, nz, n))
    op = ptychofft(nt, nz, n, nt, ns, det, det, P)
    op.setobj(T(scan), T(prb))
    orc = PtychoFFT(nt, nz, n, nt, ns, det, det, P)
    orc.setobj(scan, prb)
    g = torch.full((nt, ns, det, det), float("nan"), dtype=torch.complex64, device="cuda")
    op.fwd(g, T(psi))
    ref = orc.fwd(psi)
    assert rel(g.cpu().numpy(), ref) <= 2e-6          # skipped scans: zero frames
    h = crand(rng, g.shape)
    f = torch.full((nt, nz, n), float("nan"), dtype=torch.complex64, device="cuda")
    op.adj(f, T(h))
    assert rel(f.cpu().numpy(), orc.adj(h)) <= 2e-6
    first = f.clone()
    op.adj(f, T(h))
    assert torch.equal(f, first)
    data = (np.abs(h) ** 2 * rng.uniform(0.25, 0.75, h.shape)).astype(np.float32)
    for model, r in ((0, h - data * h / np.abs(h) ** 2), (1, h - np.sqrt(data) * np.exp(1j * np.angle(h)))):
        op.adj_resid(f, T(h), T(data), 1.0, model)
        assert rel(f.cpu().numpy(), orc.adj(r)) <= 1e-5
    gp = torch.empty((P, P), dtype=torch.complex64, device="cuda")
    op.adj_probe(gp, T(h), T(psi))
    assert rel(gp.cpu().numpy(), orc.adj_probe(h, psi)) <= 2e-6


@pytest.mark.parametrize("det", [16, 64, 128])
def test_gaussian_residual_out_of_range_values(det):
    """Zeros, subnormal and huge moduli and counts among ordinary ones: the
    residual in 64 bits, then the oracle's adjoint."""
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(det)
    n = det + 3
    scan = np.zeros((2, 1, 2), np.float32)
    scan[0, 0] = [1, 2]
    prb = crand(rng, (det, det))
    op = ptychofft(1, n, n, 1, 2, det, det, det)
    op.setobj(T(scan), T(prb))
    orc = PtychoFFT(1, n, n, 1, 2, det, det, det)
    orc.setobj(scan, prb)
    h = crand(rng, (1, 2, det, det))
    d = (np.abs(h) ** 2 * rng.uniform(0.25, 0.75, h.shape)).astype(np.float32)
    pick = rng.permutation(h.size)
    flat, dat = h.reshape(-1), d.reshape(-1)
    for i, x in enumerate((0, 1e-20, 3e-16 - 2e-16j, 1e-38j, 5.0)):
        flat[pick[7 * i:7 * i + 7]] = x
        dat[pick[7 * i:7 * i + 7]] = [0, 1e-45, 1e-38, 1e-31, 1e-20, 1.0, 9.0]
    r = h.astype(np.complex128) - np.sqrt(d.astype(np.float64)) * np.exp(1j * np.angle(h.astype(np.complex128)))
    f = torch.empty((1, n, n), dtype=torch.complex64, device="cuda")
    op.adj_resid(f, T(h), T(d), 1.0, 1)
    assert rel(f.cpu().numpy(), orc.adj(r)) <= 1e-5


@pytest.mark.parametrize("nt,nz,n,ns,det,P", [
    (4, 60, 61, 325, 16, 10), (2, 41, 40, 130, 32, 32),       # more than 16 parts
    (33, 61, 60, 14, 16, 13), (6, 50, 47, 20, 32, 31),        # few frames: four threads per line
    (148, 33, 33, 36, 16, 16), (60, 40, 41, 40, 32, 29),      # many
    (1, 70, 71, 887, 64, 32), (8, 70, 71, 111, 64, 32)])      # forward: one and two frames per trip
@pytest.mark.parametrize("uneven", [False, True])
def test_dispatch_edges_against_oracle(nt, nz, n, ns, det, P, uneven):
    """The forms that the numbers of frames and scans choose between.  The
    tolerances of the test above; sums over several hundred scans of one pixel
    add at most sqrt(400) x 2^-24 = 1.2e-6 to the adjoint's: 4e-6."""
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(det + 7 * ns)
    scan = np.stack([rng.uniform(0, n - P, (nt, ns)), rng.uniform(0, nz - P, (nt, ns))]).astype(np.float32)
    if uneven:
        for t in range(nt):
            scan[:, t, ns - rng.integers(0, ns // 2):] = -1
    prb, psi = crand(rng, (P, P)), crand(rng, (nt, nz, n))
    op, orc = ptychofft(nt, nz, n, nt, ns, det, det, P), PtychoFFT(nt, nz, n, nt, ns, det, det, P)
    op.setobj(T(scan), T(prb))
    orc.setobj(scan, prb)
    g = torch.full((nt, ns, det, det), float("nan"), dtype=torch.complex64, device="cuda")
    op.fwd(g, T(psi))
    assert rel(g.cpu().numpy(), orc.fwd(psi)) <= 2e-6
    h = crand(rng, g.shape)
    f = torch.full((nt, nz, n), float("nan"), dtype=torch.complex64, device="cuda")
    op.adj(f, T(h))
    assert rel(f.cpu().numpy(), orc.adj(h)) <= 4e-6
    data = (np.abs(h) ** 2 * rng.uniform(0.25, 0.75, h.shape)).astype(np.float32)
    op.adj_resid(f, T(h), T(data), 1.0, 0)
    assert rel(f.cpu().numpy(), orc.adj(h - data * h / np.abs(h) ** 2)) <= 1e-5
