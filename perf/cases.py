"""The calls of this framework whose speed matters, as a user's program makes them.

A reconstruction calls the two operators of the ADMM loop, the USFFT Radon
transform and the ptychography operator, each in both directions, on arrays
that stay on the GPU, and solves two CG subproblems per iteration with them.
The cases are those calls: single operator calls from a few slices of a
32-wide volume up to the 256-cubed benchmark geometry, the data-term gradient
in both noise models, and one whole CG subproblem of each kind.

``listed()`` holds the cases, ``draw(rng)`` gives others of the same ranges,
``prepare``/``run`` make and run one, ``work`` states what a call cannot do
without, and ``exact`` evaluates the same call in 64 bits: direct
non-uniform DFT sums at the polar points (with the angles' cosines in 64
bits) and dense 2-D FFTs of the probe-weighted patches.
"""
import math

import torch

VOXEL, ENERGY = 1e-6, 5.0                       # [cm], [keV]
WAVENUMBER = ENERGY / (6.58211928e-19 * 299792458e+2)
DELTA = 1e-5                                     # refractive index decrement of the phantom
MODELS = ("poisson", "gaussian")


# ---- cases -----------------------------------------------------------------
def listed():
    return [
        # the smallest volumes of the tests: launches and latency count
        dict(name="radon_fwd_32", op="radon_fwd", n=32, nz=9, ntheta=24, wedge=False),
        # the benchmark geometry, forward
        dict(name="radon_fwd_256", op="radon_fwd", n=256, nz=256, ntheta=384, wedge=False),
        # an 84-slice slab of the 128-wide configuration (slices not a multiple of 8 or 16)
        dict(name="radon_adj_128", op="radon_adj", n=128, nz=84, ntheta=128, wedge=False),
        # the benchmark geometry, adjoint
        dict(name="radon_adj_256", op="radon_adj", n=256, nz=256, ntheta=384, wedge=False),
        # the exact adjoint of the preconditioned CG on a 60-degree missing wedge
        dict(name="radon_adj_exact_64", op="radon_adj_exact", n=64, nz=16, ntheta=90, wedge=True),
        # the reference driver's problem at 128: 16-pixel probe, 64 x 64 detector, step 8
        dict(name="ptycho_fwd_64", op="ptycho_fwd", n=128, nz=128, ntheta=192, det=64, nprb=16, nscan=225,
             uneven=False),
        # the benchmark geometry: 13 x 13 scans of a 128-pixel probe, forward and adjoint
        dict(name="ptycho_fwd_128", op="ptycho_fwd", n=256, nz=256, ntheta=384, det=128, nprb=128, nscan=169,
             uneven=False),
        dict(name="ptycho_adj_128", op="ptycho_adj", n=256, nz=256, ntheta=384, det=128, nprb=128, nscan=169,
             uneven=False),
        # the CG gradient of the 128-wide configuration: 64-pixel probe, 7 x 7 raster, Poisson
        dict(name="ptycho_grad_64", op="ptycho_grad", n=128, nz=128, ntheta=128, det=64, nprb=64, nscan=49,
             uneven=False, model="poisson"),
        # uneven spiral scans (100 to 400 per angle, padded with the sentinel), Gaussian
        dict(name="ptycho_grad_uneven", op="ptycho_grad", n=256, nz=256, ntheta=45, det=128, nprb=128, nscan=400,
             uneven=True, model="gaussian"),
        # the tomography subproblem of the 128-wide configuration, 4 CG iterations
        dict(name="cg_tomo_128", op="cg_tomo", n=128, nz=84, ntheta=128, wedge=False, iters=4),
        # the ptychography subproblem of the reference driver's problem at 64, 4 CG iterations; Gaussian, because
        # a Poisson gradient divides by the weakest pixels' |f|^2, so a whole CG amplifies the last bit by 1e2 to 1e4
        dict(name="cg_ptycho_64", op="cg_ptycho", n=64, nz=64, ntheta=96, det=64, nprb=16, nscan=49, uneven=False,
             model="gaussian", iters=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["radon_fwd", "radon_adj", "radon_adj_exact", "ptycho_fwd", "ptycho_adj", "ptycho_grad", "cg_tomo",
                     "cg_ptycho"])
    if op.startswith("radon"):
        n = rng.choice([32, 64, 128, 256])
        return dict(op=op, n=n, nz=_log(rng, 3, 256), ntheta=_log(rng, 12, 384), wedge=rng.random() < 0.3)
    if op == "cg_tomo":
        n = rng.choice([32, 64, 128])
        return dict(op=op, n=n, nz=_log(rng, 8, n), ntheta=_log(rng, 24, 192), wedge=rng.random() < 0.3, iters=4)
    det = rng.choice([16, 32, 64, 128] if op != "cg_ptycho" else [16, 32, 64])
    nprb = det if rng.random() < 0.5 else rng.randrange(max(8, det // 4), det + 1)
    size = _log(rng, max(nprb + 8, 32), 256)
    if op == "cg_ptycho":   # a Solver's object is a compiled width of the Radon transform
        size = rng.choice([w for w in (32, 64, 128) if w >= nprb])
    c = dict(op=op, n=size, nz=max(nprb, size - rng.randrange(0, 24)), ntheta=_log(rng, 4, 384), det=det, nprb=nprb,
             nscan=_log(rng, 9, 400), uneven=rng.random() < 0.3)
    # at most the benchmark's detector pixels (an eighth of them for a whole CG)
    most = 384 * 169 * 128 * 128 // (1 if op != "cg_ptycho" else 8)
    c["ntheta"] = max(1, min(c["ntheta"], most // (c["nscan"] * det * det)))
    if op in ("ptycho_grad", "cg_ptycho"):
        c["model"] = rng.choice(MODELS) if op == "ptycho_grad" else "gaussian"
    if op == "cg_ptycho":
        c["iters"] = 4
    return c


# ---- inputs ----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _noise(g, *shape):
    return torch.complex(torch.randn(shape, generator=g, device="cuda"), torch.randn(shape, generator=g, device="cuda"))


def _theta(c):
    lo, hi = (-math.pi / 3, math.pi / 3) if c["wedge"] else (0.0, math.pi)
    return (lo + (hi - lo) * torch.arange(c["ntheta"], dtype=torch.float64) / c["ntheta"]).float().cuda()


def _blobs(g, count=12):
    """Gaussian blobs in [-1, 1]^3: centres (x, y, z), radius, -delta + i beta."""
    pos = _rand(g, count, 3, lo=-0.4, hi=0.4)
    rad = _rand(g, count, lo=0.03, hi=0.2)
    amp = torch.complex(-_rand(g, count, lo=0.1), 0.1 * _rand(g, count, lo=0.1)) * DELTA
    return pos, rad, amp


def _axis(n):
    return (torch.arange(n, device="cuda", dtype=torch.float64) - n // 2) * (2.0 / n)


def _object(c, g):
    """u [nz, n, n]: a phantom of smooth blobs with a fine texture inside them."""
    pos, rad, amp = _blobs(g)
    x, z = _axis(c["n"]), _axis(c["nz"])
    def e(t, i):
        return torch.exp(-((t[None] - pos[:, i, None]) / rad[:, None]) ** 2 / 2).to(torch.complex64)
    u = torch.einsum("b,bz,by,bx->zyx", amp.to(torch.complex64), e(z, 2), e(x, 1), e(x, 0))
    return (u * (1 + 0.1 * _noise(g, *u.shape))).contiguous()


def _projections(c, g, theta):
    """[ntheta, nz, n]: the blobs' line integrals (in pixels) with measurement noise."""
    pos, rad, amp = _blobs(g)
    x, z = _axis(c["n"]), _axis(c["nz"])
    t = theta.double()
    s = torch.cos(t)[:, None] * pos[None, :, 0] - torch.sin(t)[:, None] * pos[None, :, 1]
    ex = torch.exp(-((x[None, None] - s[:, :, None]) / rad[None, :, None]) ** 2 / 2).to(torch.complex64)
    ez = torch.exp(-((z[None] - pos[:, 2, None]) / rad[:, None]) ** 2 / 2).to(torch.complex64)
    w = (amp * rad * math.sqrt(2 * math.pi) * c["n"] / 2).to(torch.complex64)
    p = torch.einsum("b,bz,tbx->tzx", w, ez, ex)
    return (p + 0.01 * p.abs().max() * _noise(g, *p.shape)).contiguous()


def _smooth(g, *shape):
    """Smooth real fields of unit size on the last two axes."""
    k = [max(2, s // 16) for s in shape[-2:]]
    f = torch.randn((*shape[:-2], *k), generator=g, device="cuda")
    return torch.nn.functional.interpolate(f.reshape(1, -1, *k), size=shape[-2:], mode="bicubic").reshape(shape)


def _psi(c, g):
    """Transmission functions [ntheta, nz, n]: smooth phase and weak absorption, with a fine phase texture."""
    s = (c["ntheta"], c["nz"], c["n"])
    ph, ab = _smooth(g, *s), _smooth(g, *s)
    tex = torch.randn(s, generator=g, device="cuda")
    return torch.polar(torch.exp(-0.02 * ab.abs()), 0.3 * ph + 0.02 * tex)


def _probe(c, g):
    """A probe that fills the detector has a Gaussian amplitude of the usual
    width (12/64 of the probe), one that is padded to it the reference
    driver's flat top with a linear edge; both with a smooth phase."""
    P = c["nprb"]
    t = torch.arange(P, device="cuda", dtype=torch.float64) - (P - 1) / 2
    r2 = t[:, None] ** 2 + t[None] ** 2
    if P == c["det"]:
        amp = torch.exp(-r2 / (2 * (P * 12 / 64) ** 2))
    else:
        amp = ((P / 2 + 1 - r2.sqrt()) / (0.1 * P + 1)).clamp(0, 1)
    return torch.polar(amp.float(), 0.5 * _smooth(g, 1, P, P)[0]).contiguous()


def _scan(c, g):
    """[2, ntheta, nscan] positions (x, y): a jittered raster, or spirals of
    uneven length whose unused slots hold the sentinel -1."""
    nt, ns, mx, my = c["ntheta"], c["nscan"], c["n"] - c["nprb"], c["nz"] - c["nprb"]
    k = torch.arange(ns, device="cuda", dtype=torch.float64)
    if c["uneven"]:
        count = torch.floor(_rand(g, nt, 1, lo=max(1, ns // 4), hi=ns + 0.999)).clamp(max=ns)
        r, a = torch.sqrt(k / count), k * 2.39996323 + _rand(g, nt, 1, hi=2 * math.pi)
        x, y = mx / 2 * (1 + r * torch.cos(a)), my / 2 * (1 + r * torch.sin(a))
    else:
        side = math.ceil(math.sqrt(ns))
        x, y = (k % side * (mx / max(side - 1, 1))).expand(nt, ns), (k // side * (my / max(side - 1, 1))).expand(nt, ns)
    x, y = x + _rand(g, nt, ns, lo=-1.5, hi=1.5), y + _rand(g, nt, ns, lo=-1.5, hi=1.5)
    s = torch.stack([x.clamp(0, max(mx - 0.5, 0)), y.clamp(0, max(my - 0.5, 0))])
    if c["uneven"]:
        s = torch.where((k < count).expand(2, nt, ns), s, torch.full_like(s, -1.0))
    return s.float().contiguous()


# ---- the ptychography operator in plain torch ---------------------------------
class _Ptycho:
    def __init__(self, c, scan, prb, dtype):
        self.c, self.dtype = c, dtype
        corner = torch.floor(scan.double() + 0.5)
        frac = scan.double() - corner
        self.ok = (corner >= 0).all(0)
        x, y = corner.clamp(min=0).long()
        r = torch.arange(c["nprb"], device="cuda")
        self.base = (y * c["n"] + x)                                        # [nt, ns]
        self.patch = (r[:, None] * c["n"] + r[None])                        # [iy, ix]
        one = torch.ones_like(frac[0])
        self.phase = (torch.polar(one, 2 * math.pi * frac[0]) * torch.polar(one, 2 * math.pi * frac[1])).to(dtype)
        self.q = (prb.to(dtype).T / c["det"]).contiguous()                  # probe at [iy, ix], 1 / sqrt(det^2)

    def _chunks(self):
        c = self.c
        step = max(1, (1 << 26) // (c["nscan"] * c["det"] ** 2))
        return [slice(t, min(t + step, c["ntheta"])) for t in range(0, c["ntheta"], step)]

    def fwd(self, psi, out=None):
        c = self.c
        P, D, off = c["nprb"], c["det"], (c["det"] - c["nprb"]) // 2
        if out is None:
            out = torch.empty((c["ntheta"], c["nscan"], D, D), dtype=self.dtype, device="cuda")
        for t in self._chunks():
            p = psi[t].reshape(psi[t].shape[0], -1).to(self.dtype)
            idx = (self.base[t][:, :, None, None] + self.patch).reshape(p.shape[0], -1)
            w = torch.gather(p, 1, idx).reshape(-1, c["nscan"], P, P) * self.q * self.ok[t][:, :, None, None]
            f = torch.zeros((*w.shape[:2], D, D), dtype=self.dtype, device="cuda")
            f[:, :, off:off + P, off:off + P] = w.transpose(2, 3)          # the detector row is the object column
            out[t] = torch.fft.fft2(f) * self.phase[t][:, :, None, None]
        return out

    def adj(self, frames, resid=None):
        """Q* F* of frames, or of resid(frames, angles) formed angle by angle."""
        c = self.c
        P, off = c["nprb"], (c["det"] - c["nprb"]) // 2
        res = torch.zeros((c["ntheta"], c["nz"] * c["n"]), dtype=self.dtype, device="cuda")
        for t in self._chunks():
            f = frames[t].to(self.dtype) if resid is None else resid(frames[t], t)
            f = f * (self.phase[t].conj() * self.ok[t])[:, :, None, None]
            f = torch.fft.ifft2(f, norm="forward")[:, :, off:off + P, off:off + P].transpose(2, 3) * self.q.conj()
            row = torch.arange(f.shape[0], device="cuda")[:, None, None] * res.shape[1]
            part = torch.view_as_real(res[t].view(-1))
            for s in range(c["nscan"]):
                idx = (row + self.base[t][:, s, None, None] + self.patch).reshape(-1)
                part.index_add_(0, idx, torch.view_as_real(f[:, s].reshape(-1)))
        return res.reshape(c["ntheta"], c["nz"], c["n"])


def _coefs(c, prb):
    """(operator scale, count scale) of the Solver for this probe."""
    amax = float(prb.abs().max())
    return 1.0 / amax, 1.0 / (c["det"] ** 2 * amax ** 2)


def _ptycho_inputs(c, seed):
    """What the ptychography cases start from: scans, probe, psi, and for the
    ones with data the counts of another psi (1e3 photons per pixel on average)."""
    g = _gen(seed)
    d = dict(scan=_scan(c, g), prb=_probe(c, g))
    d["psi"] = _psi(c, g)
    plain = _Ptycho(c, d["scan"], d["prb"], torch.complex64)
    scale, count = _coefs(c, d["prb"])
    if c["op"] in ("ptycho_adj", "ptycho_grad"):
        d["frames"] = plain.fwd(d["psi"])
        if c["op"] == "ptycho_grad":
            d["frames"] *= scale
    if "model" in c:
        frames = plain.fwd(d["psi"] * torch.polar(torch.ones_like(d["psi"].real), 0.2 * _smooth(g, *d["psi"].shape)))
        inten = frames.abs().square_().mul_(scale * scale / count)
        del frames
        level = 1e3 / float(inten.mean())
        d["data"] = torch.poisson(inten.mul_(level), generator=g).div_(level)
    if c["op"] == "cg_ptycho":
        d["h"] = d["psi"] * torch.polar(torch.ones_like(d["psi"].real), 0.05 * _smooth(g, *d["psi"].shape))
        d["lamd"] = 0.01 * _noise(g, *d["psi"].shape)
    return d


def _tomo_inputs(c, seed):
    g = _gen(seed)
    d = dict(theta=_theta(c))
    if c["op"] == "radon_fwd":
        d["u"] = _object(c, g)
    elif c["op"] != "cg_tomo":
        d["g"] = _projections(c, g, d["theta"])
    else:
        coef = 1 / math.sqrt(c["ntheta"] * c["n"] / 2)
        p = _projections(c, g, d["theta"]) * coef
        d["K"] = 1j * torch.polar(0.9 + 0.1 * torch.rand(p.shape, generator=g, device="cuda"), 0.3 * _smooth(g, *p.shape))
        d["xi0"] = d["K"] * p
        d["init"] = 0.5 * _object(c, g)
        d["xi1"] = 0.1 * DELTA * _noise(g, 3, c["nz"], c["n"], c["n"])
    return d


def prepare(case, seed):
    from ptychotomo_b200 import Solver, ptychofft, radonusfft
    c, op = case, case["op"]
    new = dict(dtype=torch.complex64, device="cuda")
    if op.startswith("radon"):
        d = _tomo_inputs(c, seed)
        d["op"] = radonusfft(c["ntheta"], c["nz"], c["n"])
        d["op"].setobj(d["theta"])
        if op == "radon_fwd":
            d["out"] = torch.empty((c["ntheta"], c["nz"], c["n"]), **new)
        else:
            d["out"] = torch.empty((c["nz"], c["n"], c["n"]), **new)
    elif op.startswith("ptycho"):
        d = _ptycho_inputs(c, seed)
        d["op"] = ptychofft(c["ntheta"], c["nz"], c["n"], c["ntheta"], c["nscan"], c["det"], c["det"], c["nprb"])
        d["op"].setobj(d["scan"], d["prb"])
        d["scale"], d["count"] = _coefs(c, d["prb"])
        if op == "ptycho_fwd":
            d["out"] = torch.empty((c["ntheta"], c["nscan"], c["det"], c["det"]), **new)
        else:
            d["out"] = torch.empty((c["ntheta"], c["nz"], c["n"]), **new)
            del d["psi"]
    elif op == "cg_tomo":
        d = _tomo_inputs(c, seed)
        # the tomography subproblem alone: a Solver with the smallest ptychography part
        prb = torch.ones((8, 8), **new)
        d["solver"] = Solver(prb, torch.zeros((2, c["ntheta"], 1), device="cuda"), d["theta"], [8, 8], VOXEL, ENERGY,
                             c["ntheta"], c["nz"], c["n"], c["ntheta"], c["nz"])
    else:
        d = _ptycho_inputs(c, seed)
        t = torch.arange(c["ntheta"], dtype=torch.float32, device="cuda") * (math.pi / c["ntheta"])
        d["solver"] = Solver(d["prb"], d["scan"], t, [c["det"], c["det"]], VOXEL, ENERGY, c["ntheta"], c["nz"], c["n"],
                             c["ntheta"], c["nz"])
    d["case"] = c
    return d


def run(state):
    c, s = state["case"], state
    op = c["op"]
    if op == "radon_fwd":
        s["op"].fwd(s["out"], s["u"])
    elif op == "radon_adj":
        s["op"].adj(s["out"], s["g"])
    elif op == "radon_adj_exact":
        s["op"].adj_exact(s["out"], s["g"])
    elif op == "ptycho_fwd":
        s["op"].fwd(s["out"], s["psi"])
    elif op == "ptycho_adj":
        s["op"].adj(s["out"], s["frames"])
    elif op == "ptycho_grad":
        s["op"].adj_resid(s["out"], s["frames"], s["data"], s["count"], MODELS.index(c["model"]), scale=s["scale"])
    elif op == "cg_tomo":
        return s["solver"].cg_tomo(s["xi0"], s["xi1"], s["K"], s["init"], 0.5, 0.5, c["iters"])
    else:
        return s["solver"].cg_ptycho_batch(s["data"], s["psi"], s["h"], s["lamd"], 0.5, c["iters"], c["model"])
    return s["out"]


# ---- what a call cannot do without ---------------------------------------------
def _radon_flops(c):
    N = c["n"] * 3 // 2
    return c["nz"] * (10 * N * N * math.log2(N) + 5 * c["ntheta"] * N * math.log2(N))


def _ptycho_flops(c):
    D = c["det"]
    return c["ntheta"] * c["nscan"] * (10 * D * D * math.log2(D) + 6 * c["nprb"] ** 2)


def work(case):
    c, op = case, case["op"]
    vol, proj = 8 * c["nz"] * c["n"] ** 2, 8 * c["ntheta"] * c["nz"] * c["n"]
    if op.startswith("radon"):
        return {"bytes": vol + proj, "flops": _radon_flops(c)}
    if op == "cg_tomo":
        return {"bytes": 2 * proj + 5 * vol, "flops": (2 * c["iters"] + 1) * _radon_flops(c)}
    frames = c["ntheta"] * c["nscan"] * c["det"] ** 2
    if op == "cg_ptycho":
        return {"bytes": 4 * proj + 4 * frames, "flops": (2 * c["iters"] + 1) * _ptycho_flops(c)}
    return {"bytes": proj + 8 * frames + (4 * frames if op == "ptycho_grad" else 0), "flops": _ptycho_flops(c)}


# ---- the same calls in 64 bits ---------------------------------------------------
class _Radon:
    """The operators as direct sums over the N x N padded slice, N = 3n/2."""

    def __init__(self, c, theta):
        n = c["n"]
        N = n * 3 // 2
        self.c, self.N, self.c0 = c, N, N // 6
        t = torch.arange(N, device="cuda", dtype=torch.float64) - N // 2
        k = t / N
        lim = 0.5 - 1e-5
        self.x = torch.cos(theta.double())[:, None] * k
        self.y = -torch.sin(theta.double())[:, None] * k
        self.x, self.y = (torch.where(v >= 0.5, torch.full_like(v, lim), v) for v in (self.x, self.y))
        self.t = t
        self.idx = torch.clamp(torch.arange(N, device="cuda"), self.c0, 5 * N // 6 - 1) - self.c0
        q = (t / N).float()
        self.mask = (4 * q[None] * q[None] + 4 * q[:, None] * q[:, None] < 1 - 1.0 / N).double()
        self.s1 = 1.0 - 2.0 * ((torch.arange(N, device="cuda", dtype=torch.float64) + 1) % 2)

    def _waves(self, a, sign):
        ph = sign * 2 * math.pi * self.t[None]
        one = torch.ones((), dtype=torch.float64, device="cuda")
        ex = torch.polar(one.expand(self.N, self.N), ph * self.x[a][:, None])
        ey = torch.polar(one.expand(self.N, self.N), ph * self.y[a][:, None])
        return ex, ey                                                        # [k, t]

    def fwd(self, f):
        c, N = self.c, self.N
        fp = (f.to(torch.complex128)[:, self.idx][:, :, self.idx] * self.mask).reshape(-1, N)
        g = torch.empty((c["ntheta"], c["nz"], N), dtype=torch.complex128, device="cuda")
        for a in range(c["ntheta"]):
            ex, ey = self._waves(a, -1)
            rows = (fp @ ex.T).reshape(c["nz"], N, N)                        # [z, y, k]
            g[a] = torch.einsum("zyk,ky->zk", rows, ey) / N
        g = torch.fft.ifft(g * self.s1, norm="forward") * self.s1
        return g[:, :, self.c0:self.c0 + c["n"]]

    def adj(self, g, exact=False):
        c, N, n = self.c, self.N, self.c["n"]
        g = g.to(torch.complex128)
        gl = torch.zeros((c["ntheta"], c["nz"], N), dtype=torch.complex128, device="cuda")
        if exact:
            gl[:, :, self.c0:self.c0 + n] = g
        else:
            gl = g[:, :, self.idx]
        gl = torch.fft.fft(gl * self.s1) * self.s1 / N
        w = slice(0, N) if exact else slice(self.c0, self.c0 + n)
        size = N if exact else n
        f = torch.zeros((c["nz"] * size, size), dtype=torch.complex128, device="cuda")
        for a in range(c["ntheta"]):
            ex, ey = self._waves(a, +1)
            f.addmm_((gl[a][:, None, :] * ey.T[None, w]).reshape(-1, N), ex[:, w])
        f = f.reshape(c["nz"], size, size) * self.mask[w, w]
        if not exact:
            return f
        fold = torch.zeros((n, N), dtype=torch.complex128, device="cuda")
        fold[self.idx, torch.arange(N, device="cuda")] = 1.0
        return fold @ f @ fold.T


def _diff(u):
    s = 2 / math.sqrt(3)
    r = torch.zeros((3, *u.shape), dtype=u.dtype, device="cuda")
    r[0, :, :, :-1] = s * (u[:, :, 1:] - u[:, :, :-1])
    r[1, :, :-1] = s * (u[:, 1:] - u[:, :-1])
    r[2, :-1] = s * (u[1:] - u[:-1])
    return r


def _diff_adj(g):
    r = g.sum(0)
    r[:, :, 1:] -= g[0, :, :, :-1]
    r[:, 1:] -= g[1, :, :-1]
    r[1:] -= g[2, :-1]
    return -2 / math.sqrt(3) * r


def _dot(a, b):
    return complex(torch.vdot(a.reshape(-1), b.reshape(-1)))


def _norm2(a):
    return _dot(a, a).real


def _halve(gamma, decrease):
    while decrease(gamma) < 0 and gamma > 1e-12:
        gamma *= 0.5
    return 0 if gamma <= 1e-12 else gamma


def _cg_tomo(c, d):
    op, rho, tau = _Radon(c, d["theta"]), 0.5, 0.5
    coef = 1 / math.sqrt(c["ntheta"] * c["n"] / 2)
    K, u = d["K"].to(torch.complex128), d["init"].to(torch.complex128)
    a = K * (coef * op.fwd(u)) - d["xi0"].to(torch.complex128)
    b = _diff(u) - d["xi1"].to(torch.complex128)
    gamma, dr, g0 = 2.0, None, None
    for _ in range(c["iters"]):
        grad = rho * coef * op.adj(K.conj() * a) + tau * _diff_adj(b)
        dr = -grad if dr is None else -grad + _norm2(grad) / (_dot(dr, grad) - _dot(dr, g0)) * dr
        g0 = grad
        fd, gd = K * (coef * op.fwd(dr)), _diff(dr)
        c1 = rho * _dot(a, fd).real + tau * _dot(b, gd).real
        c2 = rho * _norm2(fd) + tau * _norm2(gd)
        gamma = _halve(gamma, lambda s: -(2 * s * c1 + s * s * c2))
        u, a, b = u + gamma * dr, a + gamma * fd, b + gamma * gd
        if gamma == 0:
            break
    return u


def _residual(f, D, model):
    if model == "poisson":
        return f - D * f / (f.abs().square() + 1e-32)
    return f - torch.sqrt(D) * torch.polar(torch.ones_like(D), f.angle())


def _cg_ptycho(c, d):
    op, rho = _Ptycho(c, d["scan"], d["prb"], torch.complex128), 0.5
    scale, count = _coefs(c, d["prb"])
    D, h, lamd = d["data"].double() * count, d["h"].to(torch.complex128), d["lamd"].to(torch.complex128)
    psi = d["psi"].to(torch.complex128)
    gamma, dr, g0 = 2.0, None, None

    def term(y):
        a = y.abs()
        if c["model"] == "poisson":
            return a.square() - 2 * D * torch.log(a.clamp(min=1e-32))
        return (a - torch.sqrt(D)).square()

    f = scale * op.fwd(psi)
    for _ in range(c["iters"]):
        w = h - psi + lamd / rho
        grad = scale * op.adj(_residual(f, D, c["model"])) - rho * w
        dr = -grad if dr is None else -grad + _norm2(grad) / (_dot(dr, grad) - _dot(dr, g0)) * dr
        g0 = grad
        fd = scale * op.fwd(dr)
        wd, d2, t0 = _dot(w, dr).real, _norm2(dr), term(f)
        gamma = _halve(gamma, lambda s: float((t0 - term(f + s * fd)).sum()) + rho * (2 * s * wd - s * s * d2))
        psi, f = psi + gamma * dr, f + gamma * fd
        if gamma == 0:
            break
    return psi


def exact(case, seed):
    c, op = case, case["op"]
    if op.startswith("radon"):
        d = _tomo_inputs(c, seed)
        r = _Radon(c, d["theta"])
        return r.fwd(d["u"]) if op == "radon_fwd" else r.adj(d["g"], exact=op == "radon_adj_exact")
    if op == "cg_tomo":
        return _cg_tomo(c, _tomo_inputs(c, seed))
    d = _ptycho_inputs(c, seed)
    if op == "cg_ptycho":
        return _cg_ptycho(c, d)
    p = _Ptycho(c, d["scan"], d["prb"], torch.complex128)
    if op == "ptycho_fwd":
        return p.fwd(d["psi"])
    if op == "ptycho_adj":
        return p.adj(d["frames"])
    scale, count = _coefs(c, d["prb"])
    return scale * p.adj(d["frames"],
                         lambda f, t: _residual(f.to(torch.complex128), d["data"][t].double() * count, c["model"]))
