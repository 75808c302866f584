"""The FP64 pass 2 by digit products (p2_dig.cu) where it can go wrong: around
the volume from which it is taken, ragged tiles of 32 and groups of 4 sites, more
sites than a batch, one and two flavours, blocks of widely different scale (per
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
