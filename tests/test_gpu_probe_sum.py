"""The probe gradient of parts of the angles, added in FP64: what one operator
over all angles gives, to the bit (one frame per partial sum; the FP64 sums
differ by 1e-16, so the rounded ones differ for one value in 1e8)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("det,P", [(16, 16), (32, 21), (64, 64), (128, 100)])
@pytest.mark.parametrize("model", [0, 1])
def test_parts_of_the_angles_add_up(det, P, model):
    from ptychotomo_b200 import ptychofft
    rng = np.random.default_rng(det + P)
    nt, ns, n, nz = 8, 9, P + 12, P + 7
    crand = lambda *s: torch.from_numpy((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()  # noqa: E731
    scan = torch.from_numpy(np.stack([rng.uniform(0, n - P, (nt, ns)), rng.uniform(0, nz - P, (nt, ns))]).astype(np.float32)).cuda()
    prb, psi, frames = crand(P, P), crand(nt, nz, n), crand(nt, ns, det, det)
    data = torch.from_numpy(rng.poisson(2.0, (nt, ns, det, det)).astype(np.float32)).cuda()

    def gradient(ids, name, dtype):
        op = ptychofft(ids.stop - ids.start, nz, n, ids.stop - ids.start, ns, det, det, P)
        op.setobj(scan[:, ids].contiguous(), prb)
        g = torch.full((P, P), float("nan"), dtype=dtype, device="cuda")
        getattr(op, name)(g, psi[ids].contiguous(), frames[ids].contiguous(), data[ids].contiguous(), 0.7, model, scale=0.5)
        return g

    whole = gradient(slice(0, nt), "adj_probe_resid", torch.complex64)
    whole64 = gradient(slice(0, nt), "adj_probe_resid64", torch.complex128)
    assert torch.equal(whole64.to(torch.complex64), whole)
    parts = sum(gradient(s, "adj_probe_resid64", torch.complex128) for s in (slice(0, 3), slice(3, 4), slice(4, nt)))
    assert torch.equal(parts.to(torch.complex64), whole)
