"""The FP64 passes at the edges of their tiles (8 sites in pass 1, 4 and 32 in
pass 2, runs along z that cross them, more tiles than thread blocks, the flush of
the compensated sums), and the launcher of pass 2 on sums that are not the gamma
images of one dz. Against the CPU oracle at the FP64 bar, 1e-12 of the pair's
(flavour's) sum. Needs a GPU."""
import numpy as np
import pytest

import support as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
TOL64 = 1e-12


@pytest.fixture(scope="module")
def hg():
    import hlbl_gb300

    return hlbl_gb300


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("lat", [(1, 1, 1, 1), (1, 1, 1, 5), (3, 5, 1, 7), (2, 3, 3, 2), (5, 2, 3, 40), (8, 9, 8, 11)])
def test_kernel_sum_at_tile_edges(hg, lat):
    x, y = S.gaussian_block(lat, 31), S.gaussian_block(lat, 32)
    gsx, yv = tuple((2 * r + 1) % lat[r] for r in range(4)), (1, -2, 3, -1)
    want = S.oracle_kernel_sum(x, y, gsx, yv, 0.4, lat)
    with hg.Contractor(lat) as c:
        got = c.kernel_sum(dev(x), dev(y), gsx, yv, 0.4, hg.FP64)
    assert S.pair_rel_err(got, want) <= TOL64


@pytest.mark.parametrize("kind", ["images", "one entry changed", "any numbers"])
@pytest.mark.parametrize("lat", [(3, 5, 1, 7), (7, 9, 8, 5)])
def test_launchers_at_tile_edges_and_with_any_sums(hg, lat, kind):
    x, y = S.gaussian_block(lat, 41), S.gaussian_block(lat, 42)
    gsx, yv, xu, f = (1, 2, 0, 3), (-1, 2, 5, 1), 0.3, 1
    dzu, dzsu = S.oracle_dz(x, y, f, gsx, lat)
    gu, gs = S.oracle_gammas(dzu, dzsu)
    rng = np.random.default_rng(5)
    if kind == "one entry changed":
        gs[-1] *= 1.5
    elif kind == "any numbers":
        gu, gs = rng.normal(size=gu.size), rng.normal(size=gs.size)
    want = S.oracle_4pt(gu, gs, x, y, f, gsx, xu, yv, lat)
    z = (0, 0, 0, 0)
    with hg.Contractor(lat) as c:
        d_x, d_y = dev(x), dev(y)
        du = torch.zeros(1728, dtype=torch.float64, device="cuda")
        ds = torch.zeros(1152, dtype=torch.float64, device="cuda")
        c.cu_dzu_dzsu(du, ds, d_x, d_y, f, z, gsx, lat, lat)
        ks = torch.full((1,), 2.5, dtype=torch.float64, device="cuda")
        c.cu_4pt_contraction(ks, dev(gu), dev(gs), d_x, d_y, f, z, gsx, xu, yv, lat, lat)
        c.check()
    scale = max(np.abs(dzu).max(), np.abs(dzsu).max())
    assert np.abs(du.cpu().numpy() - dzu).max() <= TOL64 * scale
    assert np.abs(ds.cpu().numpy() - dzsu).max() <= TOL64 * scale
    assert abs(float(ks[0]) - 2.5 - want) <= TOL64 * (abs(want) + 2.5)
