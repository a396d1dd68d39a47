"""The ptycho forward on either side of the number of frames at which its kernel
changes (16 x 16 to 64 x 64 frames), against the oracle, and with the sub-pixel
model against the same frames in the other kernel.

Tolerance 2e-6: two FFT passes of det <= 64 points round by at most 12 x 2^-24 =
7e-7 relative to the frame."""
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


@pytest.mark.parametrize("det,P,per_sm", [(16, 16, 12), (16, 15, 16), (16, 4, 16), (32, 32, 2), (32, 17, 5), (32, 1, 5),
                                          (64, 64, 1), (64, 63, 2), (64, 30, 2)])
def test_forward_around_the_change_of_kernel(det, P, per_sm):
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(100 * det + P)
    most = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    n, nz = P + 21, P + 30
    prb, psi = crand(rng, (P, P)), crand(rng, (1, nz, n))
    scan = np.stack([rng.uniform(0, n - P, (1, most + 1)), rng.uniform(0, nz - P, (1, most + 1))]).astype(np.float32)
    scan[:, 0, [1, most - 1]] = -1
    sub = {}
    for ns in (1, most, most + 1):
        s = scan[:, :, :ns]
        op = ptychofft(1, nz, n, 1, ns, det, det, P)
        op.setobj(T(s), T(prb))
        orc = PtychoFFT(1, nz, n, 1, ns, det, det, P)
        orc.setobj(s, prb)
        g = torch.full((1, ns, det, det), float("nan"), dtype=torch.complex64, device="cuda")
        op.fwd(g, T(psi), scale=0.5)
        assert rel(g.cpu().numpy(), 0.5 * orc.fwd(psi)) <= 2e-6      # skipped scans: zero frames
        op.set_subpixel(4)
        sub[ns] = torch.full_like(g, float("nan"))
        op.fwd(sub[ns], T(psi))
    a, b = sub[most][0].cpu().numpy(), sub[most + 1][0, :most].cpu().numpy()
    assert rel(a, b) <= 2e-6
