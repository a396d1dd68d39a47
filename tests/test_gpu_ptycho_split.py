"""The split of the ptycho adjoint over blocks and slabs: what setobj may do to
it, and that every way to choose it gives the oracle's adjoint.

Tolerance 4e-6: two FFT passes of det <= 128 points round by at most 14 x 2^-24
= 8e-7 relative to the frame, and a pixel's sum over at most 200 scans by
sqrt(200) x 2^-24 = 8e-7 in the mean and a few times that in the worst order."""
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


def scans(rng, nt, nz, n, ns, P, valid):
    """Random scans of which the first `valid` of each angle are not skipped."""
    scan = np.stack([rng.uniform(0, n - P, (nt, ns)), rng.uniform(0, nz - P, (nt, ns))]).astype(np.float32)
    scan[:, :, valid:] = -1
    return scan


@pytest.mark.parametrize("nt,nz,n,ns,det,P,few", [(2, 60, 61, 200, 16, 10, 12), (2, 60, 61, 200, 32, 20, 8),
                                                  (3, 70, 71, 60, 64, 32, 6), (5, 131, 130, 40, 128, 64, 3)])
def test_setobj_leaves_the_slabs_of_a_captured_adjoint(nt, nz, n, ns, det, P, few):
    """An adjoint captured with few scans is replayed after setobj with all of
    them, for which a fresh operator would take more parts: the slabs that the
    graph writes must still be there, so the split must not grow (checked
    before the replay)."""
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(det)
    prb, g = crand(rng, (P, P)), crand(rng, (nt, ns, det, det))
    part, full = scans(rng, nt, nz, n, ns, P, few), scans(rng, nt, nz, n, ns, P, ns)
    fresh = ptychofft(nt, nz, n, nt, ns, det, det, P)
    fresh.setobj(T(full), T(prb))
    op = ptychofft(nt, nz, n, nt, ns, det, det, P)
    op.setobj(T(part), T(prb))
    before = op.parts
    assert 1 < before < fresh.parts
    gd = T(g)
    f = torch.empty((nt, nz, n), dtype=torch.complex64, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        op.adj(f, gd)
    torch.cuda.current_stream().wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.adj(f, gd)
    scan = T(full)
    op.setobj(scan, T(prb))
    assert op.parts <= before
    orc = PtychoFFT(nt, nz, n, nt, ns, det, det, P)
    orc.setobj(full, prb)
    ref = orc.adj(g)
    f.fill_(float("nan"))
    graph.replay()
    assert rel(f.cpu().numpy(), ref) <= 4e-6
    f.fill_(float("nan"))
    op.adj(f, gd)
    assert rel(f.cpu().numpy(), ref) <= 4e-6
    # slabs that no launch has used are chosen anew
    op = ptychofft(nt, nz, n, nt, ns, det, det, P)
    op.setobj(T(part), T(prb))
    op.setobj(scan, T(prb))
    assert op.parts == fresh.parts
