"""FP32 kernel sums of FP64 blocks at the sizes where their launch can go wrong:
several pairs over odd and flat lattices (the tiles of all pairs come from one
counter, their sums are added in a fixed order), pair groups, both operand types,
many evaluations near the origin in every pair (listed, then evaluated in FP64),
and a captured call. Against the CPU oracle at the FP32 path's bar (1e-4 of a
pair's scale, the path's other tests'); repeated calls are bit-identical. Needs a
GPU."""
import numpy as np
import pytest

import support as S

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
TOL32 = 1e-4


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def problem(lat, n, seed):
    y = S.gaussian_block(lat, seed)
    xs = [S.random_block(lat, seed + 1 + i) for i in range(n)]
    gsxs = [tuple((i + 2 * r) % lat[r] for r in range(4)) for i in range(n)]
    yvs = [tuple((-1) ** r * (i + r) for r in range(4)) for i in range(n)]
    return y, xs, gsxs, yvs


@pytest.mark.parametrize("fp16", [True, False], ids=["fp16", "tf32"])
@pytest.mark.parametrize("lat,n,group", [((3, 5, 7, 9), 5, 0), ((1, 1, 1, 33), 3, 2), ((2, 1, 17, 1), 4, 1), ((4, 4, 4, 2), 16, 0)])
def test_pairs_of_blocks(lat, n, group, fp16):
    import hlbl_gb300 as hg

    y, xs, gsxs, yvs = problem(lat, n, 80)
    with hg.Contractor(lat) as c:
        c.set_tc_fp16(fp16)
        c.set_batch_group(group)
        out = torch.zeros(2, n, 2, dtype=torch.float64, device="cuda")
        d_y, d_xs = dev(y), [dev(x) for x in xs]
        for rep in range(2):
            c.kernel_sums_batched(d_y, d_xs, gsxs, yvs, 0.4, out[rep], hg.FP32)
        torch.cuda.synchronize()
        c.check()
        out = out.cpu().numpy()
    assert np.array_equal(out[0], out[1])
    for i in range(n):
        assert S.pair_rel_err(out[0, i], S.oracle_kernel_sum(xs[i], y, gsxs[i], yvs[i], 0.4, lat)) <= TOL32


@pytest.mark.parametrize("xunit", [0.02, 0.06])
def test_many_evaluations_near_the_origin(xunit):
    import hlbl_gb300 as hg

    lat, n = (4, 5, 3, 6), 3
    y, xs, gsxs, yvs = problem(lat, n, 90)
    with hg.Contractor(lat) as c:
        out = torch.zeros(n, 2, dtype=torch.float64, device="cuda")
        c.kernel_sums_batched(dev(y), [dev(x) for x in xs], gsxs, yvs, xunit, out, hg.FP32)
        torch.cuda.synchronize()
        out = out.cpu().numpy()
    for i in range(n):
        assert S.pair_rel_err(out[i], S.oracle_kernel_sum(xs[i], y, gsxs[i], yvs[i], xunit, lat)) <= TOL32


def test_captured_call_equals_the_eager_one():
    import hlbl_gb300 as hg

    lat, n = (3, 5, 7, 9), 4
    y, xs, gsxs, yvs = problem(lat, n, 95)
    with hg.Contractor(lat) as c:
        d_y, d_xs = dev(y), [dev(x) for x in xs]
        out, eager = (torch.zeros(n, 2, dtype=torch.float64, device="cuda") for _ in range(2))
        c.reserve(n)
        c.graph_begin()
        c.kernel_sums_batched(d_y, d_xs, gsxs, yvs, 0.4, out, hg.FP32)
        g = c.graph_end()
        g.launch()
        c.kernel_sums_batched(d_y, d_xs, gsxs, yvs, 0.4, eager, hg.FP32)
        torch.cuda.synchronize()
        c.check()
        assert torch.equal(out, eager)
        g.close()
