"""The FP64 pass 2 by digit products (p2_dig.cu) where it can go wrong: around
the volume from which a batch of pairs takes it, ragged tiles of 32 and groups of 4
sites, more sites than a batch, one and two flavours, blocks of widely different scale (per
site, per row and per block), zero blocks and values that are not finite.
Against the CPU oracle at the FP64 bar, 1e-12 of the pair's sum. Needs a GPU."""
import numpy as np
import pytest

import support as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
TOL64 = 1e-12


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def run(lat, x, y, gsx, yv, xu=0.4):
    import hlbl_gb300 as hg

    with hg.Contractor(lat) as c:
        return np.array(c.kernel_sum(dev(x), dev(y), gsx, yv, xu, hg.FP64))


@pytest.mark.parametrize("lat", [(1, 1, 1, 127), (1, 2, 4, 16), (1, 1, 3, 43), (3, 1, 1, 53), (10, 11, 9, 13)])
def test_sizes(lat):
    x, y = S.gaussian_block(lat, 51), S.random_block(lat, 52)
    gsx, yv = tuple((2 * r + 1) % lat[r] for r in range(4)), (1, -2, 3, -1)
    assert S.pair_rel_err(run(lat, x, y, gsx, yv), S.oracle_kernel_sum(x, y, gsx, yv, 0.4, lat)) <= TOL64


@pytest.mark.parametrize("kind", ["sites", "rows", "blocks"])
def test_scales(kind):
    lat = (3, 4, 5, 6)
    shape = (2, 12, S.volume(lat), 24)
    x, y = S.gaussian_block(lat, 61).reshape(shape), S.gaussian_block(lat, 62).reshape(shape)
    rng = np.random.default_rng(8)
    if kind == "sites":
        x, y = (b * np.ldexp(1.0, rng.integers(-80, 1, size=shape[2]))[None, None, :, None] for b in (x, y))
    elif kind == "rows":
        x, y = (b * np.ldexp(1.0, rng.integers(-30, 1, size=shape[:2]))[:, :, None, None] for b in (x, y))
    else:
        x, y = x * 2.0**-200, y * 2.0**150
    x, y, gsx, yv = x.ravel(), y.ravel(), (2, 1, 0, 3), (1, 2, -2, 1)
    assert S.pair_rel_err(run(lat, x, y, gsx, yv), S.oracle_kernel_sum(x, y, gsx, yv, 0.4, lat)) <= TOL64


@pytest.mark.parametrize("value", [0.0, np.nan, np.inf])
def test_zero_and_not_finite(value):
    lat, gsx, yv = (3, 4, 5, 6), (2, 1, 0, 3), (1, 2, -2, 1)
    x, y = S.gaussian_block(lat, 71), S.gaussian_block(lat, 72)
    if value == 0.0:
        x[:] = 0.0
        assert np.all(run(lat, x, y, gsx, yv) == 0.0)
    else:
        y[7 * 24 + 5] = value  # flavour 0 of y: both passes of both flavours' sums read it
        assert not np.any(np.isfinite(run(lat, x, y, gsx, yv)))


@pytest.mark.parametrize("lat", [(4, 4, 4, 7), (4, 8, 4, 4), (5, 7, 5, 3)])
def test_several_pairs_in_a_batch(lat):
    """448, 512 and 525 sites: both sides of the volume from which a batch of pairs
    goes through digit products; repeated calls are bit-identical."""
    import hlbl_gb300 as hg

    n = 3
    y, xs = S.gaussian_block(lat, 81), [S.random_block(lat, 82 + i) for i in range(n)]
    gsxs, yvs = [(i, 1, 2, 0) for i in range(n)], [(1, i, -1, 2) for i in range(n)]
    with hg.Contractor(lat) as c:
        out = torch.zeros(2, n, 2, dtype=torch.float64, device="cuda")
        d_y, d_xs = dev(y), [dev(x) for x in xs]
        for rep in range(2):
            c.kernel_sums_batched(d_y, d_xs, gsxs, yvs, 0.4, out[rep], hg.FP64)
        torch.cuda.synchronize()
        c.check()
        out = out.cpu().numpy()
    assert np.array_equal(out[0], out[1])
    for i in range(n):
        assert S.pair_rel_err(out[0, i], S.oracle_kernel_sum(xs[i], y, gsxs[i], yvs[i], 0.4, lat)) <= TOL64


def test_capture_without_the_work_buffer():
    """A capture on a context that has no work buffer yet takes the kernel that
    needs none; afterwards the eager call and a new capture take digit products."""
    import hlbl_gb300 as hg

    lat, gsx, yv = (3, 4, 5, 6), (2, 1, 0, 3), (1, 2, -2, 1)
    x, y = S.gaussian_block(lat, 91), S.gaussian_block(lat, 92)
    want = S.oracle_kernel_sum(x, y, gsx, yv, 0.4, lat)
    with hg.Contractor(lat) as c:
        d_x, d_y = dev(x), dev(y)
        out = torch.zeros(3, 2, dtype=torch.float64, device="cuda")
        c.reserve(1)
        graphs = []
        for i in (0, 2):
            c.graph_begin()
            c.kernel_sum_async(d_x, d_y, gsx, yv, 0.4, out[i], hg.FP64)
            graphs.append(c.graph_end())
            if i == 0:
                c.kernel_sum_async(d_x, d_y, gsx, yv, 0.4, out[1], hg.FP64)
        for g in graphs:
            g.launch()
        torch.cuda.synchronize()
        c.check()
        got = out.cpu().numpy()
        for g in graphs:
            g.close()
    for i in range(3):
        assert S.pair_rel_err(got[i], want) <= TOL64
    assert np.array_equal(got[1], got[2])


def test_launcher_in_a_capture_without_the_work_buffer():
    """There the launcher of pass 2 takes the kernels that need no buffer, also
    with sums that are not the gamma images of one dz."""
    import hlbl_gb300 as hg

    lat, gsx, yv, f = (3, 4, 5, 6), (2, 1, 0, 3), (1, 2, -2, 1), 1
    x, y = S.gaussian_block(lat, 93), S.gaussian_block(lat, 94)
    rng = np.random.default_rng(9)
    images = S.oracle_gammas(*S.oracle_dz(x, y, f, gsx, lat))
    z = (0, 0, 0, 0)
    for gu, gs in (images, (rng.normal(size=6912), rng.normal(size=4608))):
        want = S.oracle_4pt(gu, gs, x, y, f, gsx, 0.4, yv, lat)
        with hg.Contractor(lat) as c:
            d_x, d_y, d_gu, d_gs = dev(x), dev(y), dev(gu), dev(gs)
            ks = torch.zeros(1, dtype=torch.float64, device="cuda")
            c.reserve(1)
            c.graph_begin()
            c.cu_4pt_contraction(ks, d_gu, d_gs, d_x, d_y, f, z, gsx, 0.4, yv, lat, lat)
            g = c.graph_end()
            g.launch()
            torch.cuda.synchronize()
            c.check()
            g.close()
        assert abs(float(ks[0]) - want) <= TOL64 * abs(want)


def test_graph_outlives_a_larger_launcher_geometry():
    """A launcher on a larger lattice than the context's makes the work buffer grow;
    a graph captured before keeps its own and gives the same sums."""
    import hlbl_gb300 as hg

    lat, gsx, yv = (3, 4, 5, 6), (2, 1, 0, 3), (1, 2, -2, 1)
    big, f, z = (7, 9, 8, 5), 0, (0, 0, 0, 0)
    x, y = S.gaussian_block(lat, 95), S.gaussian_block(lat, 96)
    bx, by = S.gaussian_block(big, 97), S.gaussian_block(big, 98)
    gu, gs = S.oracle_gammas(*S.oracle_dz(bx, by, f, gsx, big))
    with hg.Contractor(lat) as c:
        d_x, d_y, d_bx, d_by, d_gu, d_gs = (dev(a) for a in (x, y, bx, by, gu, gs))
        out = torch.zeros(2, 2, dtype=torch.float64, device="cuda")
        ks = torch.zeros(1, dtype=torch.float64, device="cuda")
        c.kernel_sum_async(d_x, d_y, gsx, yv, 0.4, out[0], hg.FP64)
        c.graph_begin()
        c.kernel_sum_async(d_x, d_y, gsx, yv, 0.4, out[1], hg.FP64)
        g = c.graph_end()
        c.cu_4pt_contraction(ks, d_gu, d_gs, d_bx, d_by, f, z, gsx, 0.4, yv, big, big)
        g.launch()
        torch.cuda.synchronize()
        c.check()
        got, launched = out.cpu().numpy(), float(ks[0])
        g.close()
    assert np.array_equal(got[0], got[1])
    assert S.pair_rel_err(got[0], S.oracle_kernel_sum(x, y, gsx, yv, 0.4, lat)) <= TOL64
    want = S.oracle_4pt(gu, gs, bx, by, f, gsx, 0.4, yv, big)
    assert abs(launched - want) <= TOL64 * abs(want)
