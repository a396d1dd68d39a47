"""The solver's vector kernels against torch in 64 bits at the sizes where their
wide accesses, unrolled loops and rows end: one element, odd numbers, one more
or less than a trip of the whole grid, arrays that are 8-byte aligned only, an
output that is one of the inputs, rows shorter than a warp and longer than a
block.

u = 2^-24: a complex product and its sum round each component at most four
times by u of sum |c| |x|; J and J* take at most four sums and a product."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

U = 2.0 ** -24
TRIP = 148 * 16 * 256                      # threads of the elementwise grid
SIZES = [1, 2, 3, 255, 513, TRIP * 2 - 1, TRIP * 4 + 2, TRIP * 4 + 3, (1 << 22) - 1, (1 << 22) + 1, (1 << 22) + TRIP * 4 + 2]


def crand(n, seed, shift=0):
    """n complex values, at an address that is 8 and not 16 modulo 16 if shift is odd."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.complex(torch.randn(n + shift, generator=g, device="cuda"), torch.randn(n + shift, generator=g, device="cuda"))[shift:]
    assert x.data_ptr() % 16 == 8 * (shift % 2)
    return x


def close(got, ref, size, rounds):
    d = got.to(torch.complex128) - ref
    bound = rounds * U * size
    return bool((d.real.abs() <= bound).all() and (d.imag.abs() <= bound).all())


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("shift", [None, 0, 1, 2])
def test_lincomb(n, shift):
    """shift: which array is 8-byte aligned only (0: the output); None: none."""
    from ptychotomo_b200 import kernels as K
    coef = [0.5 - 1.25j, -2.0, 0.75j, 1.0 + 0.3j]
    for k in (1, 2, 3, 4):
        for alias in (None, 0, k - 1):
            xs = [crand(n, 10 * k + j, int(shift == j + 1)) for j in range(k)]
            ref = sum(complex(np.complex64(c)) * x.to(torch.complex128) for c, x in zip(coef, xs))
            size = sum(abs(c) * x.abs().double() for c, x in zip(coef, xs))
            out = crand(n, 99, int(shift == 0)) if alias is None else xs[alias]
            K.lincomb(out, list(zip(coef, xs)))
            assert close(out, ref, size, 4 + k), (k, alias)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("shift", [None, 0, 1, 2, 3])
def test_cmul(n, shift):
    from ptychotomo_b200 import kernels as K
    for mode in (0, 1, 2):
        for alias in (None, 0, 1):
            a, b, c = (crand(n, 7 * mode + j, int(shift == j + 1)) for j in range(3))
            x, y, z = (v.to(torch.complex128) for v in (a, b, c))
            y = y - z if mode == 1 else y
            ref, size = (x if mode == 0 else x.conj()) * y, x.abs() * (y.abs() + (b.abs() + c.abs()).double() * (mode == 1))
            out = crand(n, 99, int(shift == 0)) if alias is None else (a, b)[alias]
            K.cmul(out, a, b, c if mode == 1 else None, mode)
            assert close(out, ref, size, 5), (mode, alias)


@pytest.mark.parametrize("nz,ny,nx", [(1, 1, 1), (3, 5, 7), (2, 9, 31), (5, 3, 33), (4, 7, 256), (3, 2, 257), (2, 3, 700),
                                      (40, 130, 3)])
def test_regulariser(nz, ny, nx):
    from ptychotomo_b200 import kernels as K
    s = 2 / np.sqrt(3)
    u, g = crand(nz * ny * nx, 1).reshape(nz, ny, nx), crand(3 * nz * ny * nx, 2).reshape(3, nz, ny, nx)
    ud, gd = u.to(torch.complex128), g.to(torch.complex128)
    sf = float(np.float32(s))
    ref, size = torch.zeros_like(gd), torch.zeros(gd.shape, dtype=torch.float64, device="cuda")
    for c, ax in enumerate((2, 1, 0)):
        m = ud.shape[ax] - 1
        hi, lo = ud.narrow(ax, 1, m), ud.narrow(ax, 0, m)
        ref[c].narrow(ax, 0, m).copy_(sf * (hi - lo))
        size[c].narrow(ax, 0, m).copy_(sf * (hi.abs() + lo.abs()))
    assert close(K.reg_fwd(torch.full_like(g, float("nan")), u, sf), ref, size, 3)
    ref, size = torch.zeros_like(ud), torch.zeros(ud.shape, dtype=torch.float64, device="cuda")
    for c, ax in enumerate((2, 1, 0)):
        m = ud.shape[ax] - 1
        ref += gd[c]
        ref.narrow(ax, 1, m).sub_(gd[c].narrow(ax, 0, m))
        size += gd[c].abs()
        size.narrow(ax, 1, m).add_(gd[c].abs().narrow(ax, 0, m))
    assert close(K.reg_adj(torch.full_like(u, float("nan")), g, sf), sf * ref, sf * size, 8)


@pytest.mark.parametrize("n", [1, 2, 255, 1184 * 256 - 1, 1184 * 256 * 4, 1184 * 256 * 4 + 1, 1184 * 256 * 9 + 77])
def test_reductions(n):
    """FP64 sums of exact products (n 2^-53 of the sum of their sizes); the
    terms of tv are rounded to FP32 (8 u), the angles by atan2f (3 ulp of pi)."""
    from ptychotomo_b200.kernels import Reducer
    red = Reducer("cuda")
    a, b = crand(n, 1), crand(n, 2)
    x, y = a.to(torch.complex128), b.to(torch.complex128)
    na, nb, ab = float((x.abs() ** 2).sum()), float((y.abs() ** 2).sum()), complex((x.conj() * y).sum())
    size, eps = float((x.abs() * y.abs()).sum()), 4 * n * 2.0 ** -53 + 1e-15
    assert abs(red.norm2(a) - na) <= eps * na
    assert abs(red.dot(a, b) - ab) <= 2 * eps * size
    q = red.quad3(a, b)
    assert abs(q[0] - na) <= eps * na and abs(q[1] - ab.real) <= 2 * eps * size and abs(q[2] - nb) <= eps * nb
    assert abs(red.norm2_diff(a, b) - float(((x - y).abs() ** 2).sum())) <= eps * (na + nb)
    assert abs(red.maxabs(a) - float(x.abs().max())) <= 4 * U * float(x.abs().max())
    assert abs(red.maxangle(a) - float(torch.angle(x).abs().max())) <= 3 * 2.0 ** -22
    t = crand(3 * n, 3)
    tv = float((t.to(torch.complex128).reshape(3, n).abs() ** 2).sum(0).sqrt().sum())
    assert abs(red.tv(t) - tv) <= 8 * U * tv


def test_line_search_without_steps_is_refused():
    from ptychotomo_b200 import PtychotomoArgError
    from ptychotomo_b200.kernels import Reducer
    f, data = crand(64, 1), torch.ones(64, device="cuda")
    with pytest.raises(PtychotomoArgError):
        Reducer("cuda").ls_frames(f, f, data, 1.0, 0, [])
