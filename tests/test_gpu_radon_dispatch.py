"""The radon forward's default at the sizes on either side of the limits between
its gathers (polar points in flight), against every variant: the
same bits, whatever the default is."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,nt", [(8, 3, 5), (8, 32, 384), (8, 32, 385), (16, 33, 96), (16, 25, 192), (16, 25, 193), (32, 32, 96), (32, 32, 97), (32, 8, 384), (32, 9, 193),
                                     (64, 3, 12), (64, 25, 48), (64, 25, 49)])
def test_default_forward_has_the_bits_of_every_variant(n, nz, nt):
    from ptychotomo_b200 import radonusfft
    rng = np.random.default_rng(n + nz + nt)
    op = radonusfft(nt, nz, n)
    op.setobj(torch.from_numpy(rng.uniform(-np.pi, np.pi, nt).astype(np.float32)).cuda())
    f = torch.from_numpy((rng.standard_normal((nz, n, n)) + 1j * rng.standard_normal((nz, n, n))).astype(np.complex64)).cuda()
    new = lambda: torch.full((nt, nz, n), float("nan"), dtype=torch.complex64, device="cuda")  # noqa: E731
    ref = new()
    op.fwd(ref, f)
    assert torch.isfinite(torch.view_as_real(ref)).all()
    for streams in (1, 2, 4):
        for gather in (0, 1, 2):
            op.set_variant(streams, gather)
            out = new()
            op.fwd(out, f)
            assert torch.equal(out, ref), (streams, gather)
    assert op.status() == (0, True)
