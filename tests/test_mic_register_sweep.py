"""The lane schedule of the block-MIC(0) sweeps in k_pcg_update (vare_gb300/csrc/projection.cu,
mic_sweeps), restated lane by lane in numpy: rotated registers, three shuffles per step, the
scaled unknowns w = M y with squared pivots. Checked against the sweeps in their plain
wavefront form (float64; the bound is the float32 rounding of 44 chained steps of
non-negative couplings: 64 ulp of the largest value)."""
import numpy as np
import pytest

F = np.float32


def plain(r, M):
    """y_c = (r_c + sum M_n y_n) M_c, then z_c = (y_c + M_c sum z_n) M_c, cells [k, j, i]."""
    y = np.zeros((8, 8, 8))
    z = np.zeros((8, 8, 8))
    cells = [(k, j, i) for k in range(8) for j in range(8) for i in range(8)]
    for k, j, i in cells:
        t = r[k, j, i]
        for kk, jj, ii in ((k, j, i - 1), (k, j - 1, i), (k - 1, j, i)):
            if min(kk, jj, ii) >= 0:
                t += M[kk, jj, ii] * y[kk, jj, ii]
        y[k, j, i] = t * M[k, j, i]
    for k, j, i in reversed(cells):
        t = sum(z[n] for n in ((k, j, i + 1), (k, j + 1, i), (k + 1, j, i)) if max(n) <= 7)
        z[k, j, i] = (y[k, j, i] + M[k, j, i] * t) * M[k, j, i]
    return z


def lanes(r, M):
    L = np.arange(32)
    j, kq = L & 7, L >> 3
    sA = j + 2 * kq
    rho = (sA + 1) & 7
    M2 = np.zeros((8, 8, 8), F)  # as k_mic_factor stores it
    for k in range(8):
        for jj in range(8):
            for i in range(8):
                M2[k, jj, (i + jj + k + 1) & 7] = F(M[k, jj, i]) * F(M[k, jj, i])
    mA, mB = M2[2 * kq, j], M2[2 * kq + 1, j]

    def rotate(v, rho):
        v = v.copy()
        for b in (1, 2, 4):
            on = (rho & b) != 0
            v = np.where(on[:, None], np.roll(v, b, axis=1), v)
        return v

    rA, rB = rotate(r[2 * kq, j].astype(F), rho), rotate(r[2 * kq + 1, j].astype(F), rho)
    up = lambda v, n: np.concatenate([v[:n], v[:-n]])  # noqa: E731
    down = lambda v, n: np.concatenate([v[n:], v[-n:]])  # noqa: E731
    ym, yp, zm, zp = ((c).astype(F) for c in (j > 0, j < 7, kq > 0, kq < 3))
    live = 0xFF << (sA + 1)
    zero = np.zeros(32, F)
    wA, wB, rz = zero, zero, zero
    for u in range(1, 23):
        a, b = (live >> u) & 1 != 0, (live >> (u - 1)) & 1 != 0
        sA_, sB_, sz = up(wA, 1), up(wB, 1), up(wB, 8)
        p, q = u & 7, (u - 1) & 7
        tA = zm * sz + (ym * sA_ + (rA[:, p] + wA))
        tB = ym * sB_ + ((rB[:, q] + wB) + wA)
        wA, wB = np.where(a, mA[:, p] * tA, F(0)), np.where(b, mB[:, p] * tB, F(0))
        rz = rz + wA * tA + wB * tB
        rA[:, p], rB[:, q] = np.where(a, wA, rA[:, p]), np.where(b, wB, rB[:, q])
    zA, zB = zero, zero
    for u in range(22, 0, -1):
        a, b = (live >> u) & 1 != 0, (live >> (u - 1)) & 1 != 0
        yA, yB, n = down(zA, 1), down(zB, 1), down(zA, 8)
        p, q = u & 7, (u - 1) & 7
        sumA, sumB = yp * yA + (zA + zB), zp * n + (yp * yB + zB)
        zA = np.where(a, mA[:, p] * sumA + rA[:, p], F(0))
        zB = np.where(b, mB[:, p] * sumB + rB[:, q], F(0))
        rA[:, p], rB[:, q] = np.where(a, zA, rA[:, p]), np.where(b, zB, rB[:, q])
    z = np.zeros((8, 8, 8), F)
    back = (8 - rho) & 7
    z[2 * kq, j], z[2 * kq + 1, j] = rotate(rA, back), rotate(rB, back)
    return z, rz.sum(dtype=np.float64)


@pytest.mark.parametrize("holes", [0.0, 0.3, 1.0])
def test_register_sweep_schedule(holes):
    rng = np.random.default_rng(17)
    M = rng.uniform(0.35, 0.55, (8, 8, 8)) * (rng.random((8, 8, 8)) >= holes)
    M = M.astype(F).astype(np.float64)
    r = (rng.standard_normal((8, 8, 8)) * (M > 0)).astype(F)
    ref = plain(r.astype(np.float64), M)
    z, rz = lanes(r, M)
    tol = 64 * 2.0 ** -24 * max(np.abs(ref).max(), 1e-30)
    assert np.abs(z - ref).max() <= tol
    assert abs(rz - (r * ref).sum()) <= 64 * 2.0 ** -24 * max(np.abs(r * ref).sum(), 1e-30)
    assert not z[M == 0].any()
