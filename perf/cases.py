"""What a user of this library has it do, as cases that can be timed and checked.

The library's work is the connected kernel sum of pairs of point sources and the
2+2 pieces of single sources. A driver solves a source, stores its propagator
block, and contracts it with the sources in range; so most cases are one such
step, on the lattices of the benchmark configurations (16 x 8^3, 24 x 12^3,
32 x 16^3, 48 x 24^3) and on ragged ones. Blocks are i.i.d. complex Gaussian FP64
fields, as in the benchmark.

Results of the FP32-product paths are returned as FP32: their buffers are FP64
because the sums over sites are, but each result carries single precision.
"""
import numpy as np
import torch

import hlbl_gb300 as hg

LAMBDA = 0.4
XUNIT = hg.xunit(105.658, 0.1)  # the benchmark's lattice spacing, 0.1 fm
DENSE_SEED = 20261204
H = (1, -1, 1, -1)  # the direction and stride of the benchmark's schedule
STRIDE = 2


def listed():
    def case(name, kind, lat, n):
        return {"name": name, "kind": kind, "t": lat[0], "x": lat[1], "y": lat[2], "z": lat[3], "n": n}

    return [
        # the driver's step on FP32 tile copies: a new block is converted and
        # contracted with its partners. The smallest benchmark lattice (launches
        # count), the headline one (autotuned, as the benchmark runs it), and one
        # whose extents are no power of two and whose volume ends inside a tile
        case("step_f32_L8", "step_f32", (16, 8, 8, 8), 4),
        case("step_f32_L24", "step_f32_tuned", (48, 24, 24, 24), 3),
        case("step_f32_ragged", "step_f32", (25, 14, 19, 22), 5),
        # one window of the driver as a recorded graph, replayed: two sources
        # of four partners each, blocks resident
        case("window_graph_f32_L12", "graph_f32", (24, 12, 12, 12), 4),
        # pairs on FP64 blocks with FP32 products: batched per source, and the
        # reference's blocking call for one pair
        case("pairs_blocks_f32_L16", "pairs_blocks_f32", (32, 16, 16, 16), 4),
        case("pair_f32_L12", "pair_f32", (24, 12, 12, 12), 1),
        # the reference's call in its own precision: the parity configuration and
        # the headline lattice (the longest pass)
        case("pair_f64_L8", "pair_f64", (16, 8, 8, 8), 1),
        case("pair_f64_L24", "pair_f64", (48, 24, 24, 24), 1),
        # the vendored launchers that the reference's own host code links with:
        # one flavour's pass 1, gamma insertion and pass 2, in FP64
        case("launchers_f64_L12", "launchers_f64", (24, 12, 12, 12), 1),
        # a QED kernel of no known structure, through the generic coefficient path
        case("step_dense_f32_L16", "step_dense_f32", (32, 16, 16, 16), 3),
        # the 2+2 pieces of a source: 16 targets from its FP32 copy, and the
        # reference's blocking FP64 call
        case("pieces_f32_L24", "pieces_f32", (48, 24, 24, 24), 16),
        case("pieces_f64_L12", "pieces_f64", (24, 12, 12, 12), 8),
    ]


# how many sites (times partners or targets) a drawn case of a kind may have
_RANGE = {
    "step_f32": (8192, 663552, 5), "step_f32_tuned": (65536, 663552, 3), "graph_f32": (8192, 82944, 4),
    "pairs_blocks_f32": (8192, 262144, 4), "pair_f32": (8192, 663552, 1), "pair_f64": (8192, 331776, 1),
    "launchers_f64": (8192, 331776, 1), "step_dense_f32": (8192, 262144, 4), "pieces_f32": (8192, 663552, 16),
    "pieces_f64": (8192, 82944, 8),
}


def draw(rng):
    kind = rng.choice(sorted(_RANGE))
    lo, hi, most = _RANGE[kind]
    volume = lo * (hi / lo) ** rng.random()
    while True:
        side = volume / 2
        x, y, z = (max(4, round(side ** 0.25 * rng.uniform(0.75, 1.35))) for _ in range(3))
        t = max(4, round(volume / (x * y * z)))
        if t <= 96 and lo // 2 <= t * x * y * z <= hi:
            return {"kind": kind, "t": t, "x": x, "y": y, "z": z, "n": rng.randint(1, most)}


def _lattice(case):
    return case["t"], case["x"], case["y"], case["z"]


def _block(lat, gen):
    v = lat[0] * lat[1] * lat[2] * lat[3]
    return torch.randn(2 * 12 * v * 24, dtype=torch.float64, device="cuda", generator=gen)


def _pairs(lat, seed, n):
    """The new source's site, and its partners' sites and distances y - x."""
    y = tuple((3 + 5 * r + seed) % lat[r] for r in range(4))
    ds = [tuple(STRIDE * (i + 1) * h for h in H) for i in range(n)]
    gsx = [tuple((y[r] - d[r]) % lat[r] for r in range(4)) for d in ds]
    return y, gsx, ds


def _targets(lat, seed, n):
    """The 2+2 targets: sites at several distances from the source."""
    g = np.random.RandomState(seed % (1 << 31))
    return [tuple(int(v) for v in (g.randint(0, L) for L in lat)) for _ in range(n)]


def _inputs(case, seed):
    """The blocks of a case (new source first) from the seed alone."""
    lat, kind, n = _lattice(case), case["kind"], case["n"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    count = 1 if kind.startswith("pieces") else 2 + n if kind == "graph_f32" else 1 + n
    return [_block(lat, gen) for _ in range(count)]


def prepare(case, seed):
    lat, kind, n = _lattice(case), case["kind"], case["n"]
    blocks = _inputs(case, seed)
    c = hg.Contractor(lat)
    y, gsx, yv = _pairs(lat, seed, n)
    s = {"kind": kind, "c": c, "lat": lat, "y": y, "gsx": gsx, "yv": yv,
         "out": torch.zeros(n, 2, dtype=torch.float64, device="cuda")}

    def copy(block=None):
        d = torch.zeros(c.f32_block_length, dtype=torch.float32, device="cuda")
        if block is not None:
            c.f32_tile_copy(block, d)
        return d

    torch.cuda.synchronize()  # the blocks are there before the library's stream reads them
    if kind in ("step_f32", "step_f32_tuned", "step_dense_f32"):
        s["block"] = blocks[0]
        s["copy"] = copy()
        s["partners"] = [copy(b) for b in blocks[1:]]
        if kind == "step_dense_f32":
            c.set_qed_kernel(hg.QED_DENSE, DENSE_SEED)
        if kind == "step_f32_tuned":
            c.f32_tile_copy(s["block"], s["copy"])
            c.autotune_f32(s["copy"], s["partners"], gsx, yv, XUNIT, s["out"])
    elif kind == "graph_f32":
        copies = [copy(b) for b in blocks]
        s["copies"] = copies
        s["out"] = torch.zeros(2, n, 2, dtype=torch.float64, device="cuda")
        c.reserve(16)
        c.graph_begin()
        for k in range(2):
            c.kernel_sums_batched_f32(copies[k], copies[2:], gsx, yv, XUNIT, s["out"][k])
        s["graph"] = c.graph_end()
    elif kind in ("pairs_blocks_f32", "pair_f32", "pair_f64", "launchers_f64"):
        s["block"], s["partners"] = blocks[0], blocks[1:]
        if kind == "launchers_f64":
            def zeros(k):
                return torch.zeros(k, dtype=torch.float64, device="cuda")
            s["dz"], s["g_dzu"], s["g_dzsu"], s["sum"] = zeros(2880), zeros(6912), zeros(4608), zeros(1)
    else:
        s["targets"] = _targets(lat, seed, n)
        if kind == "pieces_f32":
            s["copy"] = copy(blocks[0])
            s["p1"] = torch.zeros(64 * c.lmax, dtype=torch.float64, device="cuda")
            s["p234"] = torch.zeros(n * 320, dtype=torch.float64, device="cuda")
            c.reserve_2p2()
        else:
            s["block"] = blocks[0]
    torch.cuda.synchronize()
    return s


def run(s):
    c, kind = s["c"], s["kind"]
    if kind in ("step_f32", "step_f32_tuned", "step_dense_f32"):
        c.f32_tile_copy(s["block"], s["copy"])
        c.kernel_sums_batched_f32(s["copy"], s["partners"], s["gsx"], s["yv"], XUNIT, s["out"])
        return {"sums": s["out"].to(torch.float32)}
    if kind == "graph_f32":
        s["graph"].launch()
        return {"sums": s["out"].to(torch.float32)}
    if kind == "pairs_blocks_f32":
        c.kernel_sums_batched(s["block"], s["partners"], s["gsx"], s["yv"], XUNIT, s["out"], hg.FP32)
        return {"sums": s["out"].to(torch.float32)}
    if kind in ("pair_f32", "pair_f64"):
        f32 = kind == "pair_f32"
        got = c.kernel_sum(s["partners"][0], s["block"], s["gsx"][0], s["yv"][0], XUNIT, hg.FP32 if f32 else hg.FP64)
        return {"sums": np.array(got, dtype=np.float32 if f32 else np.float64)}
    if kind == "launchers_f64":
        lat, here = s["lat"], (0, 0, 0, 0)
        s["dz"].zero_()
        s["sum"].zero_()
        dzu, dzsu = s["dz"][:1728], s["dz"][1728:]
        c.cu_dzu_dzsu(dzu, dzsu, s["partners"][0], s["block"], 0, here, s["gsx"][0], lat, lat)
        c.insert_gammas(dzu, dzsu, s["g_dzu"], s["g_dzsu"])
        c.cu_4pt_contraction(s["sum"], s["g_dzu"], s["g_dzsu"], s["partners"][0], s["block"], 0, here, s["gsx"][0],
                             XUNIT, s["yv"][0], lat, lat)
        return {"dz": s["dz"], "g_dzu": s["g_dzu"], "g_dzsu": s["g_dzsu"], "sum": s["sum"]}
    if kind == "pieces_f32":
        c.pieces_2p2_f32(s["copy"], s["y"], s["targets"], XUNIT, s["p1"], s["p234"])
        return {"p1": s["p1"].to(torch.float32), "p234": s["p234"].to(torch.float32)}
    got = c.pieces_2p2(s["block"], s["y"], s["targets"], XUNIT, hg.FP64)
    return {"p1": got.p1, "p234": got.p234}


def work(case):
    lat, kind, n = _lattice(case), case["kind"], case["n"]
    v = lat[0] * lat[1] * lat[2] * lat[3]
    b64, b32 = 4608 * v, 2304 * v
    # per site of one flavour: the 8 spin-block products of 144 (ia, ib), their
    # sums with the weights, the contraction of the four D_mu with the ten sums
    # (four chirality blocks of 4 x 4 spin components, nine colour pairs), the
    # dot with the 640 coefficients
    flavour = 2 * (144 * (96 + 16) + 4 * 160 * 72 + 640)
    weight = 16 * 20  # one QED evaluation: 16 nodes
    pair = v * (2 * flavour + 3 * weight)
    if kind in ("step_f32", "step_f32_tuned", "step_dense_f32"):
        return {"bytes": b64 + b32 + n * b32, "flops": n * pair}
    if kind == "graph_f32":
        return {"bytes": (2 + n) * b32, "flops": 2 * n * pair}
    if kind in ("pairs_blocks_f32", "pair_f32", "pair_f64"):
        return {"bytes": (1 + n) * b64, "flops": n * pair}
    if kind == "launchers_f64":
        return {"bytes": 2 * b64, "flops": v * (flavour + 3 * weight)}
    block = b32 if kind == "pieces_f32" else b64
    return {"bytes": block, "flops": v * (2 * 64 * 36 + n * 4 * (weight + 400))}


# ---- the same results in 64 bits, in plain torch ---------------------------------
_SRC = ((2, 3, 0, 1), (3, 2, 1, 0), (3, 2, 1, 0), (2, 3, 0, 1), None, (0, 1, 2, 3))
_PH = ((2, 2, 2, 2), (3, 3, 1, 1), (2, 0, 0, 2), (3, 1, 1, 3), None, (0, 0, 2, 2))
_COMB = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))
_SITES = 32768  # sites at a time


def _gamma(g, dev):
    m = torch.zeros(4, 4, dtype=torch.complex128)
    for s in range(4):
        m[s, _SRC[g][s]] = 1j ** _PH[g][s]
    return torch.kron(m, torch.eye(3, dtype=torch.complex128)).to(dev)


def _map(x, L):
    return torch.where(x >= L // 2, x - L, x).to(torch.float64)


def _map_zerohalf(x, L):
    return torch.where(x > L // 2, x - L, torch.where(x < L // 2, x, torch.zeros_like(x))).to(torch.float64)


def _rel(lat, origin, lo, hi, dev):
    """Positions of sites [lo, hi) relative to `origin`, in [0, L)."""
    i = torch.arange(lo, hi, device=dev)
    out = []
    for r in (3, 2, 1, 0):
        out.append((i % lat[r] - origin[r]) % lat[r])
        i = i // lat[r]
    return torch.stack(out[::-1], 1)


def _each(f, x, lat):
    return torch.stack([f(x[:, r], lat[r]) for r in range(4)], 1)


_NODES = np.polynomial.legendre.leggauss(16)


def _standin(a, b):
    """The stand-in QED tensor [n][6][4][4][4] at the argument pairs (a, b)."""
    dev, n = a.device, a.shape[0]
    X, Y = a.norm(dim=1), b.norm(dim=1)
    den = X * Y
    c = torch.where(den > 0, (a * b).sum(1) / torch.where(den > 0, den, torch.ones_like(den)), torch.zeros_like(den)).clamp(-1, 1)
    w = torch.zeros(6, n, dtype=torch.float64, device=dev)
    for node, weight in zip(*_NODES):
        u = 0.5 * (1 + node)
        v = 1 - u
        r2 = (u * u * X * X + v * v * Y * Y - 2 * u * v * X * Y * c).clamp(min=0)
        g = 0.5 * weight / (1 + r2)
        r = torch.sqrt(r2 + LAMBDA ** 2)
        first, step = torch.exp(-0.6 * r), torch.exp(-0.2 * r)
        for j, h in enumerate((1, u, v, u * v, u * u, v * v)):
            w[j] += g * h * first
            first = first * step
    d, s = a - b, a + b
    k = torch.zeros(n, 6, 4, 4, 4, dtype=torch.float64, device=dev)
    for q, (rho, sig) in enumerate(_COMB):
        for p, m, sign in ((rho, sig, 1.0), (sig, rho, -1.0)):
            k[:, q, p, m, :] += sign * w[0, :, None] * a
            k[:, q, p, :, m] += sign * w[1, :, None] * b
            k[:, q, :, p, m] += sign * w[2, :, None] * d
            k[:, q, m] += sign * (w[4] * a[:, p])[:, None, None] * b[:, :, None] * b[:, None, :]
            k[:, q, :, :, m] += sign * (w[5] * b[:, p])[:, None, None] * a[:, :, None] * a[:, None, :]
        for m in range(4):
            k[:, q, m, m] += (w[3] * (a[:, rho] * b[:, sig] - a[:, sig] * b[:, rho]))[:, None] * s
    return k


def _dense_table(seed):
    i = np.arange(13 * 384, dtype=np.uint64)
    with np.errstate(over="ignore"):
        x = np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + i + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        x = x ^ (x >> np.uint64(31))
    return ((x >> np.uint64(11)).astype(np.float64) / 9007199254740992.0 * 2 - 1).reshape(13, 384)


def _dense(a, b, table=[]):
    """The dense test tensor [n][6][4][4][4]."""
    if not table:
        table.append(torch.from_numpy(_dense_table(DENSE_SEED)))
    g = 1 / (1 + (a * a).sum(1) + (b * b).sum(1) + 0.5 * ((a - b) ** 2).sum(1))
    phi = torch.cat([torch.ones_like(a[:, :1]), a, b, a * b], 1) * g[:, None]
    return (phi @ table[0].to(a.device)).reshape(-1, 6, 4, 4, 4)


def _rows(block, lat, f, lo, hi):
    """A flavour's 12 rows of sites [lo, hi): complex [sites][12 rows][12]."""
    v = lat[0] * lat[1] * lat[2] * lat[3]
    x = block.view(2, 12, v, 12, 2)[f, :, lo:hi].permute(1, 0, 2, 3).contiguous()
    return torch.view_as_complex(x)


def _exact_dz(x, y, f, gsx, lat):
    """Pass 1: dzu [6][12][12] and dzsu [4][12][12]."""
    v, dev = lat[0] * lat[1] * lat[2] * lat[3], x.device
    g5 = [_gamma(5, dev) @ _gamma(s, dev) for s in range(4)]
    acc = torch.zeros(5, 4, 12, 12, dtype=torch.complex128, device=dev)
    for lo in range(0, v, _SITES):
        hi = min(v, lo + _SITES)
        z = _each(_map_zerohalf, _rel(lat, gsx, lo, hi, dev), lat).to(torch.complex128)
        a, b = _rows(x, lat, f, lo, hi), _rows(y, lat, 1 - f, lo, hi).conj()
        b = b.permute(1, 0, 2).reshape(12, -1)  # [ib][site, i]
        for s in range(4):
            ga = a @ g5[s].T
            for w in range(5):
                gw = ga if w == 4 else ga * z[:, w, None, None]
                acc[w, s] += (b @ gw.permute(0, 2, 1).reshape(-1, 12)).T
    dzu = torch.stack([acc[r, s] - acc[s, r] for r, s in _COMB])
    return dzu, acc[4]


def _insert(dz, dev):
    """gamma_mu gamma_5 on the last index: [j][mu][12][12]."""
    g = torch.stack([_gamma(m, dev) @ _gamma(5, dev) for m in range(4)])
    return torch.einsum("mcb,jab->jmac", g, dz)


def _exact_pass2(x, y, f, g, gsx, yv, lat, tensor):
    v, dev = lat[0] * lat[1] * lat[2] * lat[3], x.device
    gg5 = torch.stack([_gamma(m, dev) @ _gamma(5, dev) for m in range(4)])
    g5 = [_gamma(5, dev) @ _gamma(s, dev) for s in range(4)]
    # F[mu][j, nu, lam] = Re sum_pq D_mu[p][q] M[j, nu, lam][q][p]
    m = torch.einsum("lcq,jncp->jnlpq", gg5, g).reshape(160, 144)
    m = torch.stack([m.real, -m.imag], -1).reshape(160, 288).T.contiguous()
    ym = torch.tensor([[(lambda t, L: t - L if t >= L // 2 else t)(yv[r] % lat[r], lat[r]) for r in range(4)]],
                      dtype=torch.float64, device=dev) * XUNIT
    total = torch.zeros((), dtype=torch.float64, device=dev)
    for lo in range(0, v, _SITES):
        hi = min(v, lo + _SITES)
        rel = _rel(lat, gsx, lo, hi, dev)
        S, Y = _rows(x, lat, 1 - f, lo, hi), _rows(y, lat, f, lo, hi)
        gs = torch.cat([S @ g5[u].T for u in range(4)], 1).conj()  # [site][mu, q][i]
        D = -(Y @ gs.transpose(1, 2)).reshape(hi - lo, 12, 4, 12).transpose(1, 2)
        F = torch.view_as_real(D.contiguous()).reshape(-1, 288) @ m
        F = F.reshape(hi - lo, 4, 10, 4, 4)
        xm = _each(_map, rel, lat) * XUNIT
        xmy = _each(_map, torch.stack([(rel[:, r] - yv[r]) % lat[r] for r in range(4)], 1), lat) * XUNIT
        zh = _each(_map_zerohalf, rel, lat)
        yy = ym.expand(hi - lo, 4)
        k3 = tensor(xm, xmy).permute(0, 1, 4, 3, 2)  # [k][lam][nu][mu] as [k][mu][nu][lam]
        cf = tensor(xm, yy) + tensor(yy, xm).transpose(2, 3) - k3
        total -= torch.einsum("skmnl,smknl->", cf, F[:, :, :6])
        for q, (r, s) in enumerate(_COMB):
            G = zh[:, r, None, None, None] * F[:, :, 6 + s] - zh[:, s, None, None, None] * F[:, :, 6 + r]
            total -= (k3[:, q] * G).sum()
    return total


def _exact_sum(x, y, gsx, yv, lat, tensor):
    out = []
    for f in range(2):
        g = _insert(torch.cat(_exact_dz(x, y, f, gsx, lat)), x.device)
        out.append(_exact_pass2(x, y, f, g, gsx, yv, lat, tensor))
    return torch.stack(out)


def _exact_pieces(block, gsw, targets, lat):
    v, dev = lat[0] * lat[1] * lat[2] * lat[3], block.device
    g5 = [_gamma(5, dev) @ _gamma(s, dev) for s in range(4)]
    gg5 = [_gamma(s, dev) @ _gamma(5, dev) for s in range(4)]
    lmax, n = max(lat), len(targets)
    p1 = torch.zeros(4, 16, lmax, dtype=torch.float64, device=dev)
    p234 = torch.zeros(n, 5, 4, 4, 4, dtype=torch.float64, device=dev)
    for lo in range(0, v, _SITES):
        hi = min(v, lo + _SITES)
        u, d = _rows(block, lat, 0, lo, hi), _rows(block, lat, 1, lo, hi).conj()
        pi = torch.zeros(hi - lo, 4, 4, dtype=torch.float64, device=dev)
        for mu in range(4):
            w = (u @ g5[mu].T) @ d.transpose(1, 2)  # w[ia][ib] = <d_ib, g5 g_mu u_ia>
            for nu in range(4):
                pi[:, mu, nu] = torch.einsum("sab,ab->s", w, gg5[nu]).real
        x = _rel(lat, gsw, lo, hi, dev)
        for r in range(4):
            p1[r].index_add_(1, x[:, r], pi.reshape(-1, 16).T.contiguous())
        xv = _each(_map, x, lat)
        xm, xn = xv * XUNIT, _each(_map, torch.stack([(-x[:, r]) % lat[r] for r in range(4)], 1), lat) * XUNIT
        for t, target in enumerate(targets):
            y = torch.tensor([[(target[r] - gsw[r]) % lat[r] for r in range(4)]], device=dev)
            yn = torch.stack([(-y[:, r]) % lat[r] for r in range(4)], 1)
            ym, yn = (_each(_map, q, lat).mul(XUNIT).expand(hi - lo, 4) for q in (y, yn))
            diff = torch.stack([(x[:, r] - y[:, r]) % lat[r] for r in range(4)], 1)
            back = torch.stack([(y[:, r] - x[:, r]) % lat[r] for r in range(4)], 1)
            xy, yx = (_each(_map, q, lat) * XUNIT for q in (diff, back))
            v0 = torch.einsum("skmnl,sml->skn", _standin(xm, ym), pi)
            v1 = torch.einsum("sknml,sml->skn", _standin(ym, xm), pi)
            v3 = torch.einsum("skmln,sml->skn", _standin(xy, yn), pi)
            v4 = torch.einsum("sknlm,sml->skn", _standin(yx, xn), pi)
            for q, (r, s) in enumerate(_COMB):
                for slot, val in enumerate((v0, v1, v3, v4)):
                    p234[t, slot, r, s] += val[:, q].sum(0)
                p234[t, 4, r, s] += (xv[:, r, None] * v4[:, q]).sum(0)
                p234[t, 4, s, r] -= (xv[:, s, None] * v4[:, q]).sum(0)
    return p1.reshape(-1), p234.reshape(-1)


def exact(case, seed):
    lat, kind, n = _lattice(case), case["kind"], case["n"]
    volume = lat[0] * lat[1] * lat[2] * lat[3]
    if kind.startswith("pieces"):
        if volume * n > 3_000_000:
            return None  # minutes in plain 64-bit torch
        p1, p234 = _exact_pieces(_inputs(case, seed)[0], _pairs(lat, seed, n)[0], _targets(lat, seed, n), lat)
        return {"p1": p1, "p234": p234}
    blocks = _inputs(case, seed)
    _, gsx, yv = _pairs(lat, seed, n)
    if kind == "launchers_f64":
        dzu, dzsu = _exact_dz(blocks[1], blocks[0], 0, gsx[0], lat)
        g = _insert(torch.cat([dzu, dzsu]), dzu.device)
        total = _exact_pass2(blocks[1], blocks[0], 0, g, gsx[0], yv[0], lat, _standin)
        real = [torch.view_as_real(q.contiguous()).reshape(-1) for q in (torch.cat([dzu, dzsu]), g[:6], g[6:])]
        return {"dz": real[0], "g_dzu": real[1], "g_dzsu": real[2], "sum": total.reshape(1)}
    tensor = _dense if kind == "step_dense_f32" else _standin
    ys, xs = (blocks[:2], blocks[2:]) if kind == "graph_f32" else (blocks[:1], blocks[1:])
    sums = torch.stack([torch.stack([_exact_sum(x, y, gsx[i], yv[i], lat, tensor) for i, x in enumerate(xs)]) for y in ys])
    if kind != "graph_f32":
        sums = sums[0]
    return {"sums": sums.reshape(2) if kind in ("pair_f32", "pair_f64") else sums}
