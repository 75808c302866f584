"""P1's plane sums (p1_plane_kernel, p1_finish_kernel) where their split can go
wrong: extents of one, extents around and above the 16 sites a CTA holds at a
time, fewer and more planes than 16. Against the oracle. Needs a GPU.

Tolerances relative to P1's largest element, those of the other 2+2 tests:
FP64 1e-13, FP32 1e-6."""
import numpy as np
import pytest

import support as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

LATTICES = [(1, 1, 1, 2), (1, 2, 17, 1), (2, 1, 1, 33), (5, 7, 3, 2), (17, 1, 16, 15), (3, 18, 2, 17)]


@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
@pytest.mark.parametrize("lat", LATTICES, ids=lambda v: "x".join(map(str, v)))
def test_p1_planes(lat, fp32):
    import hlbl_gb300 as hg

    fwd = S.random_block(lat, 77)
    gsw = [L // 2 for L in lat]
    targets = [[0, 0, 0, 0]]
    want, _ = S.oracle_pieces_2p2(fwd, gsw, targets, 0.3, lat)
    with hg.Contractor(lat) as c:
        r = c.pieces_2p2(torch.from_numpy(fwd).cuda(), gsw, targets, 0.3, hg.FP32 if fp32 else hg.FP64)
    got = np.asarray(r.p1).reshape(want.shape)
    assert np.max(np.abs(got - want)) <= (1e-6 if fp32 else 1e-13) * np.max(np.abs(want))
