"""The block-diagonal form of pass 2's contraction (hlbl_gb300/csrc/quat_basis.cuh),
restated in numpy from its header's formulas, against the direct trace
Re Tr(D M) with the gamma matrices of the oracle: every (nu, lam), random
complex D and dz, to FP64 rounding (sums of 288 products of order one)."""
import numpy as np

import support as S


def _gamma_g5(mu):
    out = np.zeros((12, 12), complex)
    for i in range(12):
        v, w, g = np.zeros(24), np.zeros(24), np.zeros(24)
        v[2 * i] = 1.0
        S.oracle().oracle_apply_gamma(5, S.vp(v), S.vp(w))
        S.oracle().oracle_apply_gamma(mu, S.vp(w), S.vp(g))
        out[:, i] = g[0::2] + 1j * g[1::2]
    return out


def _components(x):
    return [x[0, 0] + x[1, 1], -1j * (x[0, 1] + x[1, 0]), x[0, 1] - x[1, 0], -1j * (x[0, 0] - x[1, 1])]


def _signs(gg5):
    """t of the block (0, 0): the spin factors of unit components."""
    unit = [np.eye(2), 1j * np.array([[0, 1], [1, 0]]), np.array([[0, 1], [-1, 0]]), 1j * np.diag([1, -1])]
    t = np.zeros((4, 4, 4, 4))
    for a in range(4):
        for b in range(4):
            D, Z = np.zeros((12, 12), complex), np.zeros((12, 12), complex)
            D[0:6:3, 0:6:3], Z[6:12:3, 6:12:3] = unit[b], unit[a]
            for nu in range(4):
                for lam in range(4):
                    t[nu, lam, a, b] = np.real(np.sum(D * (gg5[lam].T @ (Z @ gg5[nu].T)).T)) / 2
    return t


def test_block_diagonal_form_equals_the_trace():
    gg5 = [_gamma_g5(m) for m in range(4)]
    rng = np.random.default_rng(3)
    D, dz = (rng.normal(size=(12, 12)) + 1j * rng.normal(size=(12, 12)) for _ in range(2))
    direct = np.array([[np.real(np.sum(D * (gg5[lam].T @ (dz @ gg5[nu].T)).T)) for lam in range(4)] for nu in range(4)])
    t00, s = _signs(gg5), np.array([1, -1, -1, -1])
    assert set(np.unique(np.round(t00, 12))) == {-1.0, 0.0, 1.0}
    for nu, lam, a, b in np.argwhere(np.abs(t00) > 0.5):
        assert nu ^ lam ^ a ^ b == 0
    blocks = np.zeros((4, 4))
    for cp in range(2):
        for cq in range(2):
            t = t00 * (-1) ** (cp + cq) * (s[:, None, None, None] if cp else 1) * (s[None, :, None, None] if cq else 1)
            q = np.zeros((4, 4))
            for kp in range(3):
                for kq in range(3):
                    X = D[6 * cp + kp:6 * cp + 6:3, 6 * cq + kq:6 * cq + 6:3]
                    Z = dz[6 * (1 - cq) + kq:6 * (1 - cq) + 6:3, 6 * (1 - cp) + kp:6 * (1 - cp) + 6:3]
                    q += np.real(np.outer(_components(Z), _components(X))) / 2
            blocks += np.einsum("nlab,ab->nl", t, q)
    assert np.abs(blocks - direct).max() <= 288 * 4 * 2.2e-16 * np.abs(direct).max()
