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
    assert 1 < op.parts <= few < fresh.parts     # at most a slab for each scan
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
    assert op.parts <= few
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


@pytest.mark.parametrize("nt,nz,n,ns,det,P", [
    (2, 60, 61, 25, 16, 9), (150, 20, 22, 13, 16, 16),         # both kernels' sizes, with blocks that queue
    (3, 50, 47, 31, 32, 25), (150, 37, 35, 7, 32, 32),
    (5, 80, 79, 18, 64, 41), (150, 70, 66, 3, 64, 64), (6, 66, 70, 80, 64, 30)])
@pytest.mark.parametrize("uneven", [False, True])
def test_every_residual_has_a_split(nt, nz, n, ns, det, P, uneven):
    """The plain adjoint and both gradients, each with its own split and kernel.
    Gradients to 1e-5: the residual of counts within a factor of two of |f|^2 is
    a quarter of f."""
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(det + 7 * ns)
    scan = scans(rng, nt, nz, n, ns, P, ns)
    if uneven:
        for t in range(nt):
            scan[:, t, rng.integers(0, ns + 1):] = -1
    prb, h = crand(rng, (P, P)), crand(rng, (nt, ns, det, det))
    op, orc = ptychofft(nt, nz, n, nt, ns, det, det, P), PtychoFFT(nt, nz, n, nt, ns, det, det, P)
    op.setobj(T(scan), T(prb))
    orc.setobj(scan, prb)
    data = (np.abs(h) ** 2 * rng.uniform(0.25, 0.75, h.shape)).astype(np.float32)
    f = torch.full((nt, nz, n), float("nan"), dtype=torch.complex64, device="cuda")
    op.adj(f, T(h))
    assert rel(f.cpu().numpy(), orc.adj(h)) <= 4e-6
    for model, r in ((0, h - data * h / np.abs(h) ** 2), (1, h - np.sqrt(data) * np.exp(1j * np.angle(h)))):
        f.fill_(float("nan"))
        op.adj_resid(f, T(h), T(data), 1.0, model)
        assert rel(f.cpu().numpy(), orc.adj(r)) <= 1e-5


def adjoints(op, h, data, shape):
    """The adjoint and both gradients."""
    out = []
    for run in (lambda f: op.adj(f, h), lambda f: op.adj_resid(f, h, data, 1.0, 0), lambda f: op.adj_resid(f, h, data, 1.0, 1)):
        f = torch.full(shape, float("nan"), dtype=torch.complex64, device="cuda")
        run(f)
        out.append(f)
    return out


FORCED = [(1, 20, 19, 1, 16, 7, 1), (3, 40, 33, 3, 16, 16, 2), (2, 40, 37, 5, 32, 1, 5), (2, 41, 40, 4, 32, 31, 3),
          (3, 50, 70, 7, 32, 32, 4), (1, 70, 66, 1, 64, 16, 1), (2, 66, 70, 6, 64, 33, 5), (2, 70, 71, 3, 64, 63, 1),
          (2, 90, 64, 9, 64, 64, 2)]


@pytest.mark.parametrize("nt,nz,n,ns,det,P,parts", FORCED)
def test_both_kernels_at_forced_splits(nt, nz, n, ns, det, P, parts, monkeypatch):
    """Gradients to 1e-5, as above.  The sub-pixel model's adjoint in one kernel
    against the other."""
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(det + P)
    scan = scans(rng, nt, nz, n, ns, P, ns)
    if ns > 2:
        scan[:, 0, 1] = -1
    prb, h = crand(rng, (P, P)), crand(rng, (nt, ns, det, det))
    data = (np.abs(h) ** 2 * rng.uniform(0.25, 0.75, h.shape)).astype(np.float32)
    orc = PtychoFFT(nt, nz, n, nt, ns, det, det, P)
    orc.setobj(scan, prb)
    ref = [orc.adj(r) for r in (h, h - data * h / np.abs(h) ** 2, h - np.sqrt(data) * np.exp(1j * np.angle(h)))]
    monkeypatch.setenv("PT_PTYCHO_ADJ_PARTS", str(parts))
    sub = []
    for few in ("0", "1"):
        monkeypatch.setenv("PT_PTYCHO_ADJ_FEW", few)
        op = ptychofft(nt, nz, n, nt, ns, det, det, P)
        op.setobj(T(scan), T(prb))
        assert op.parts == parts
        for got, want, tol in zip(adjoints(op, T(h), T(data), (nt, nz, n)), ref, (4e-6, 1e-5, 1e-5)):
            assert rel(got.cpu().numpy(), want) <= tol
        op.set_subpixel(8)
        sub.append(adjoints(op, T(h), T(data), (nt, nz, n)))
    for a, b, tol in zip(*sub, (4e-6, 1e-5, 1e-5)):
        assert rel(a.cpu().numpy(), b.cpu().numpy()) <= tol


@pytest.mark.parametrize("nt,nz,n,ns,det,P", [(9, 36, 50, 36, 16, 16), (150, 30, 31, 40, 16, 9), (40, 40, 41, 20, 32, 29),
                                              (30, 70, 66, 12, 64, 41), (3, 131, 130, 9, 128, 100)])
@pytest.mark.parametrize("valid", [0.5, 1.0])
def test_a_split_is_the_same_however_it_is_set(nt, nz, n, ns, det, P, valid, monkeypatch):
    """By the environment, by the property before and after setobj: the same bits."""
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(nt + det)
    scan = scans(rng, nt, nz, n, ns, P, int(valid * ns))
    prb, h = crand(rng, (P, P)), T(crand(rng, (nt, ns, det, det)))
    data = h.abs().square() * 0.5
    for parts in (1, 3, ns):
        ops = []
        with monkeypatch.context() as m:
            m.setenv("PT_PTYCHO_ADJ_PARTS", str(parts))
            ops.append(ptychofft(nt, nz, n, nt, ns, det, det, P))
            ops[0].setobj(T(scan), T(prb))
        for before in (True, False):
            ops.append(ptychofft(nt, nz, n, nt, ns, det, det, P))
            if before:
                ops[-1].parts = parts
            ops[-1].setobj(T(scan), T(prb))
            if not before:
                ops[-1].parts = parts
        assert [op.parts for op in ops] == [parts] * 3
        a, b, c = (adjoints(op, h, data, (nt, nz, n)) for op in ops)
        for x, y, z in zip(a, b, c):
            assert torch.equal(x, y) and torch.equal(x, z)


@pytest.mark.parametrize("nt,nz,n,ns,det,P", [(4, 60, 61, 325, 16, 10), (60, 40, 41, 40, 32, 29), (6, 80, 79, 18, 64, 41),
                                              (3, 131, 130, 9, 128, 100)])
@pytest.mark.parametrize("few", [None, "0"])
def test_autotuner_starts_from_the_present_split(nt, nz, n, ns, det, P, few, monkeypatch):
    """The present split is among those timed, so the result is it or one that
    was faster: never a split that was not offered.  The gradients keep theirs,
    to the bit, and setobj keeps the tuned one."""
    from ptychotomo_b200 import ptychofft
    if few:
        monkeypatch.setenv("PT_PTYCHO_ADJ_FEW", few)
    rng = np.random.default_rng(nt + det)
    scan = scans(rng, nt, nz, n, ns, P, ns)
    prb, h = crand(rng, (P, P)), crand(rng, (nt, ns, det, det))
    data = T(h).abs().square() * 0.5
    op = ptychofft(nt, nz, n, nt, ns, det, det, P)
    op.setobj(T(scan), T(prb))
    before, default = adjoints(op, T(h), data, (nt, nz, n)), op.parts
    f = torch.empty((nt, nz, n), dtype=torch.complex64, device="cuda")
    tuned = op.autotune(f, T(h), trials=2)
    assert tuned == op.parts and tuned in (1, 2, 3, 4, 6, 8, 12, 16, default)
    op.setobj(T(scan[:, :, ::-1].copy()), T(prb))
    assert op.parts == tuned
    op.setobj(T(scan), T(prb))
    after = adjoints(op, T(h), data, (nt, nz, n))
    orc = PtychoFFT(nt, nz, n, nt, ns, det, det, P)
    orc.setobj(scan, prb)
    assert rel(after[0].cpu().numpy(), orc.adj(h)) <= 4e-6
    assert torch.equal(after[1], before[1]) and torch.equal(after[2], before[2])
