"""Redistancing (rows of half tiles, vare_gb300/csrc/surface.cu) from fields that the caller sets,
bit for bit against the same step on dense numpy arrays, the sign of zeros included: values of
both signs, +0 and -0, denormals, infinities and NaN, large magnitudes; one step and two;
ragged grids; with the water tank's faces and without. The step is the reference's with the term
whose factor max(sign, 0) or min(sign, 0) is zero counted as a signed zero, also where its
square root overflows (the reference forms 0 * infinity there)."""
import numpy as np
import pytest

from test_gpu_post import pair, real_cells
from vare_gb300 import scenes

pytestmark = pytest.mark.gpu


F = np.float32


def _nbr(a, ax, d):
    out = np.full_like(a, F(10))
    src, dst = [slice(None)] * 3, [slice(None)] * 3
    src[2 - ax], dst[2 - ax] = (slice(1, None), slice(None, -1)) if d > 0 else (slice(None, -1), slice(1, None))
    out[tuple(dst)] = a[tuple(src)]
    return out


def _step(v, tank, wall):
    """one step over the dense grid [z, y, x]"""
    zero, one = F(0), F(1)
    a = b = None
    for ax in range(3):
        lo, hi = _nbr(v, ax, -1), _nbr(v, ax, 1)
        n = v.shape[2 - ax]
        idx = np.broadcast_to(np.arange(n).reshape([-1 if k == 2 - ax else 1 for k in range(3)]), v.shape)
        if tank:
            ll = (np.broadcast_to(np.arange(v.shape[1], dtype=F).reshape(1, -1, 1), v.shape) + F(0.5)) - F(wall)
            n0 = np.where(idx == 0, ll - one if ax == 1 else ll, lo)
            n1 = np.where(idx == n - 1, ll + one if ax == 1 else ll, hi)
        else:
            n0, n1 = np.where(idx == 0, F(2) * v - hi, lo), np.where(idx == n - 1, F(2) * v - lo, hi)
        d0, d1 = v - n0, n1 - v
        mx, mn = (lambda d: np.where(d > 0, d, zero)), (lambda d: np.where(d < 0, d, zero))
        ta, tb = (mx(d0) * mx(d0), mn(d1) * mn(d1)), (mn(d0) * mn(d0), mx(d1) * mx(d1))
        a = (ta[0] if a is None else a + ta[0]) + ta[1]
        b = (tb[0] if b is None else b + tb[0]) + tb[1]
    sign = v / np.sqrt(v * v + one)
    zp, zn = np.where(a < 1, F(-0.0), zero), np.where(b < 1, F(-0.0), zero)
    t1 = np.where(sign > 0, F(0.3) * sign * (np.sqrt(a) - one), zp)
    t2 = np.where(sign < 0, F(0.3) * sign * (np.sqrt(b) - one), zn)
    return ((v - t1) - t2).astype(F)


@pytest.mark.parametrize("n,tank", [(20, False), (20, True), (32, False), (44, True)])
@pytest.mark.parametrize("iters", [1, 2])
def test_redistance_values(gpu, oracle_lib, n, tank, iters):
    B = oracle_lib
    sc = scenes.dam_break(n, (0.5, 0.4), seed=3, ppc=1)
    sim, ora = pair(gpu, B, sc, tank, redist_iteration=iters)
    sim.run_stage(gpu.STAGE_REBUILD)
    tiles, fi = sim.tiles(), sim.frame_info()
    real = real_cells(tiles, fi["nx"], fi["ny"], fi["nz"])
    rng = np.random.default_rng(n)
    surf = rng.uniform(-3, 3, len(real)).astype(np.float32)
    odd = np.array([0.0, -0.0, 1e-42, -1e-42, np.inf, -np.inf, np.nan, 1e30, -1e30, 1.0, -1.0], np.float32)
    pick = rng.random(len(surf)) < 0.3
    surf[pick] = rng.choice(odd, pick.sum(), p=np.array([8, 8, 1, 1, .2, .2, .2, .4, .4, 2, 2]) / 23.4)
    flat = rng.random(len(surf)) < 0.2  # equal neighbours: differences of 0, sums of 0 or 1
    surf[flat] = np.round(surf[flat])
    sim.set_field(gpu.FIELD_SURF, surf)
    sim.run_post_stage(gpu.POST_REDISTANCE)
    nx, ny, nz = fi["nx"], fi["ny"], fi["nz"]
    dense = np.full((nz + 8, ny + 8, nx + 8), F(10))
    active = np.zeros(dense.shape, bool)
    for (i, j, k), c in zip(tiles, surf.reshape(-1, 8, 8, 8)):
        dense[8 * k:8 * k + 8, 8 * j:8 * j + 8, 8 * i:8 * i + 8] = c
        active[8 * k:8 * k + 8, 8 * j:8 * j + 8, 8 * i:8 * i + 8] = True
    dense, active = dense[:nz, :ny, :nx].copy(), active[:nz, :ny, :nx]
    wall = fi["voxel_wall"]
    with np.errstate(all="ignore"):
        for _ in range(iters):
            dense = np.where(active, _step(dense, tank, wall), F(10))
    full = np.full((fi["tz"] * 8, fi["ty"] * 8, fi["tx"] * 8), F(0))
    full[:nz, :ny, :nx] = dense
    want = np.concatenate([full[8 * k:8 * k + 8, 8 * j:8 * j + 8, 8 * i:8 * i + 8].reshape(-1) for i, j, k in tiles])[real]
    got = sim.field(gpu.FIELD_SURF)[real]
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.int32), want[~nan].view(np.int32))
