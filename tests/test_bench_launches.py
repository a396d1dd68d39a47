"""bench.py's count of kernel launches per step (CPU)."""
from types import SimpleNamespace

import pytest

import bench


@pytest.mark.parametrize("n,nz,ntheta,tuned,parts,launches", [
    (256, 256, 384, None, 3, 4 * 16 + 6),
    (256, 256, 384, {"radon_fwd_streams": 4, "radon_gather": "TMA smem tiles"}, 1, 4 * 32 + 5),
    (64, 40, 96, None, 1, 4 * 3 + 5),
    (64, 40, 96, {"radon_fwd_streams": 2, "radon_gather": "L1"}, 1, 3 * 3 + 5),
    (64, 40, 48, None, 1, 3 * 3 + 5), (128, 40, 12, None, 1, 4 * 3 + 5),
    (32, 32, 96, None, 1, 3 * 2 + 5),                                                   # gather and lines in one launch
    (32, 32, 97, None, 1, 4 * 2 + 5),
    (16, 32, 192, None, 1, 3 * 2 + 5), (16, 32, 193, None, 1, 4 * 2 + 5), (8, 8, 1536, None, 1, 3 * 1 + 5),
    (32, 32, 97, {"radon_fwd_streams": 1, "radon_gather": "L1"}, 1, 3 * 1 + 5)])
def test_launches_per_step(n, nz, ntheta, tuned, parts, launches):
    ops = SimpleNamespace(c=dict(n=n, nz=nz, ntheta=ntheta), tuned=tuned, ptycho=SimpleNamespace(parts=parts))
    assert bench.Ops.launches_per_step(ops) == launches
