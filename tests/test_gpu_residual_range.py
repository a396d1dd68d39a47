"""The residual that the ptycho gradients form on load, value by value over the
range of FP32: a frame that is zero but for one value transforms into that
value times powers of two, without rounding, so its patch of the object holds
the residual itself.

u = 2^-24.  Poisson x - D x / b, b = |x|^2 + 1e-32: at most seven roundings (two
of |x|^2, the sum, the reciprocal, two products, the difference) and, where 1/b
is subnormal, 2^-150 b < 2 u more: 16 u of |x| + |D x / b|.  Gaussian x - sqrt(D)
x / |x|: rsqrtf (2 ulp = 4 u) and six roundings, or, for |x|^2 < 1e-30, atan2f (3
ulp of an angle up to pi: 12 u) and sincosf (2 ulp: 4 u): 24 u of |x| + sqrt(D).
Sums into the object flush what is below 2^-126."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

U = 2.0 ** -24
X = np.array([0, 1e-38, 1e-20, 3e-16 - 2e-16j, 2e-15j, -1e-3 + 1e-9j, 0.7 - 0.3j, 3e3j, 2e9 - 1e9j, 3e18, 1e19j, -7e18 + 6e18j],
             np.complex64)
D = np.array([0, 1e-45, 1e-38, 1e-31, 3e-30, 1e-20, 1.0, 9.0, 4e6, 1e10, 1e30, 1e37], np.float32)


def expected(x, d, model):
    """The residual in 64 bits, and the size that its error is measured by."""
    x, d = x.astype(np.complex128), d.astype(np.float64)
    t = d * x / (np.abs(x) ** 2 + 1e-32) if model == 0 else np.sqrt(d) * np.exp(1j * np.angle(x))
    return x - t, np.abs(x) + np.abs(t)


def check(got, x, d, model, floor=0.0):
    ref, size = expected(x, d, model)
    ok = (np.abs(ref.real) < 1e37) & (np.abs(ref.imag) < 1e37)      # the others overflow
    assert ok.sum() > 0.8 * ok.size
    err = np.abs(got.astype(np.complex128) - ref)[ok]
    assert (err <= (16, 24)[model] * U * size[ok] + floor).all()


@pytest.mark.parametrize("model", [0, 1])
def test_residual_over_the_range(model):
    from ptychotomo_b200 import kernels as K
    x, d = np.repeat(X, len(D)), np.tile(D, len(X))
    xt = torch.from_numpy(x).cuda()
    out = K.residual(torch.empty_like(xt), xt, torch.from_numpy(d).cuda(), 1.0, model)
    check(out.cpu().numpy(), x, d, model)


def one_value_frames(x, d, det, P, model, parts, few, monkeypatch):
    """adj_resid of one frame per (x, d), over disjoint patches: [frame, P, P]."""
    from ptychotomo_b200 import ptychofft
    if parts:
        monkeypatch.setenv("PT_PTYCHO_ADJ_PARTS", parts)
    if few:
        monkeypatch.setenv("PT_PTYCHO_ADJ_FEW", few)
    side, k = 4, 12
    assert len(x) % k == 0
    nt, n, nz = len(x) // k, side * P, -(-k // side) * P
    s = np.arange(k)
    scan = np.broadcast_to(np.stack([s % side * P, s // side * P])[:, None], (2, nt, k)).astype(np.float32)
    op = ptychofft(nt, nz, n, nt, k, det, det, P)
    op.setobj(torch.from_numpy(scan.copy()).cuda(), torch.ones((P, P), dtype=torch.complex64, device="cuda"))
    fr = torch.zeros((nt * k, det, det), dtype=torch.complex64, device="cuda")
    da = torch.zeros((nt * k, det, det), dtype=torch.float32, device="cuda")
    fr[:, 0, 0], da[:, 0, 0] = torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda()
    f = torch.empty((nt, nz, n), dtype=torch.complex64, device="cuda")
    op.adj_resid(f, fr, da, 1.0, model)
    f = f.reshape(nt, -1, P, side, P).transpose(2, 3).reshape(nt * k, P, P)
    return f.cpu().numpy().astype(np.complex128) * det


# detector, probe, number of parts, kernel for few frames or not (None: chosen)
FRAMES = [(16, 16, None, "1"), (16, 16, "1", "0"), (16, 9, "1", "0"), (32, 32, "2", "0"), (32, 11, "1", "0"), (32, 20, None, "1"),
          (64, 64, None, "0"), (64, 33, None, "0"), (64, 32, "1", "1"), (128, 128, None, None), (128, 100, "1", None)]


@pytest.mark.parametrize("det,P,parts,few", FRAMES)
@pytest.mark.parametrize("model", [0, 1])
def test_gradient_residual_over_the_range(det, P, parts, few, model, monkeypatch):
    x, d = np.repeat(X, len(D)), np.tile(D, len(X))
    got = one_value_frames(x, d, det, P, model, parts, few, monkeypatch)
    for i, j in ((0, 0), (P - 1, 0), (P // 2, P - 1)):
        check(got[:, i, j], x, d, model, floor=det * 2.0 ** -126)


@pytest.mark.parametrize("det,P,parts,few", FRAMES)
def test_counts_that_are_not_numbers_stay_visible(det, P, parts, few, monkeypatch):
    """A count that is NaN or infinite, or negative in the Gaussian model, makes
    its own patch not finite and no other."""
    for model, bad in ((0, [np.nan, np.inf]), (1, [np.nan, np.inf, -1.0])):
        x, d = np.full(24, 0.5 + 1j, np.complex64), np.ones(24, np.float32)
        d[5:5 + len(bad)] = bad
        got = one_value_frames(x, d, det, P, model, parts, few, monkeypatch)
        assert (~np.isfinite(got)).all(axis=(1, 2)).tolist() == [not (np.isfinite(v) and v >= 0) for v in d]
