"""The right-hand side, the stencil codes and the velocity update (warps over half tiles,
vare_gb300/csrc/projection.cu) against the same formulas on dense numpy arrays, bit for bit (FP32,
same operation order), with flags that the caller has set at random: fluid next to inactive tiles,
at the grid's faces, in ragged edge tiles; a neighbour tile missing on any side."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu
AIR, SOLID, WALL, FLUID, MASKED = 0, 1, 2, 4, 255
F = np.float32


def _dense(tiles, shape, field, fill):
    nz, ny, nx = shape
    out = np.full((nz + 8, ny + 8, nx + 8), fill, field.dtype)
    for (i, j, k), v in zip(tiles, field.reshape(len(tiles), 8, 8, 8)):
        out[8 * k:8 * k + 8, 8 * j:8 * j + 8, 8 * i:8 * i + 8] = v
    return out[:nz, :ny, :nx]


def _shift(a, ax, d, fill):
    """a's neighbour in direction d (+1 / -1) of axis ax (0 x, 1 y, 2 z), fill beyond the grid"""
    n = 2 - ax
    out = np.full_like(a, fill)
    src, dst = [slice(None)] * 3, [slice(None)] * 3
    src[n], dst[n] = (slice(1, None), slice(None, -1)) if d > 0 else (slice(None, -1), slice(1, None))
    out[tuple(dst)] = a[tuple(src)]
    return out


def _edges(shape, ax):
    idx = np.arange(shape[2 - ax]).reshape([-1 if a == 2 - ax else 1 for a in range(3)])
    return np.broadcast_to(idx == 0, shape), np.broadcast_to(idx == shape[2 - ax] - 1, shape)


@pytest.mark.parametrize("n,fluid,seed", [((24, 24, 24), 0.9, 1), ((20, 28, 36), 0.6, 2), ((40, 12, 24), 1.0, 3),
                                          ((36, 36, 20), 0.3, 4)])
def test_row_stencils(gpu, n, fluid, seed):
    rng = np.random.default_rng(seed)
    sim = flip.FlipSim(n, (0, 0, 0), tuple(F(v) for v in n), flip.default_params(wall_level=5.0, voxel_size=1.0, dt=1e-2))
    nx, ny, nz = (sim.frame_info()[k] for k in ("nx", "ny", "nz"))
    assert (nx, ny, nz) == n
    # particles in one corner: some tiles stay inactive in the larger grids
    pos = rng.uniform(0.5, 9.0, (400, 3)).astype(F)
    sim.set_particles(pos, np.zeros_like(pos), space=flip.SPACE_VOXEL)
    sim.run_stage(flip.STAGE_REBUILD)
    sim.run_stage(flip.STAGE_P2G)
    tiles = sim.tiles()
    shape = (nz, ny, nx)
    flag = sim.field(flip.FIELD_FLAG)
    inside = flag != MASKED
    flag = np.where(inside, np.where(rng.random(flag.shape) < fluid, FLUID, rng.choice([AIR, AIR, SOLID], flag.shape)), MASKED).astype(np.uint8)
    vel = (rng.uniform(-1, 1, (len(flag), 3)) * inside[:, None]).astype(F)
    pres = np.where(flag == FLUID, rng.uniform(-1, 1, len(flag)), 0).astype(F)
    sim.set_field(flip.FIELD_FLAG, flag)
    sim.set_field(flip.FIELD_VELO, vel)
    sim.run_stage(flip.STAGE_BUILD_SYSTEM)
    rhs, code = sim.field(flip.FIELD_RHS), sim.field(flip.FIELD_CODE)
    sim.set_field(flip.FIELD_PRES, pres)
    sim.run_stage(flip.STAGE_UPDATE_VELOCITY)
    comp, pout = sim.field(flip.FIELD_COMP), sim.field(flip.FIELD_PRES)
    sim.close()

    fl = _dense(tiles, shape, flag, AIR)
    active = _dense(tiles, shape, np.ones(len(flag), np.uint8), 0) > 0
    y = np.broadcast_to(np.arange(ny, dtype=F).reshape(1, -1, 1), shape)
    low = y + F(0.5) <= F(5.0) + F(1.0)
    isf = fl == FLUID

    def types(ax, wall):
        e0, e1 = _edges(shape, ax)
        return np.where(e0, wall, _shift(fl, ax, -1, AIR)), np.where(e1, wall, _shift(fl, ax, 1, AIR)), e0, e1

    # right-hand side and codes
    d = []
    diag, mask = np.full(shape, 6), np.zeros(shape, int)
    for ax in range(3):
        t0, t1, e0, e1 = types(ax, np.where(low, WALL, AIR))
        v = _dense(tiles, shape, np.ascontiguousarray(vel[:, ax]), F(0))
        lo, hi = _shift(v, ax, -1, F(0)), _shift(v, ax, 1, F(0))
        n0, n1 = np.where(e0, F(2) * v - hi, lo), np.where(e1, F(2) * v - lo, hi)
        a = np.where(t0 == AIR, F(2) * v - n1, np.where(t0 == WALL, np.abs(v), n0))
        b = np.where(t1 == AIR, F(2) * v - n0, np.where(t1 == WALL, -np.abs(v), n1))
        d.append((b - a) * F(0.5))
        for q, t in ((0, t0), (1, t1)):
            diag = diag + (t == AIR) - ((t == SOLID) | (t == WALL))
            mask = mask | ((t == FLUID).astype(int) << (2 * ax + q))
    want = np.where(isf, -((d[0] + d[1]) + d[2]), F(0))
    np.testing.assert_array_equal(_dense(tiles, shape, rhs, F(0))[active], want[active])
    wcode = np.where(isf, 0x8000 | (diag << 8) | mask, 0).astype(np.uint16)
    np.testing.assert_array_equal(_dense(tiles, shape, code, 0)[active], wcode[active])

    # air cells' mean pressure, then the gradient
    p = _dense(tiles, shape, pres, F(0))
    press, cnt = np.zeros(shape, F), np.zeros(shape, np.int32)
    for ax in range(3):
        for s in (-1, 1):
            f = _shift(isf, ax, s, False)
            press = np.where(f, press + _shift(p, ax, s, F(0)), press).astype(F)
            cnt += f
    mean = np.divide(press, cnt.astype(F), out=np.zeros(shape, F), where=cnt > 0)
    pa = np.where(isf, p, np.where(fl == AIR, mean, F(0))).astype(F)
    np.testing.assert_array_equal(_dense(tiles, shape, pout, F(0))[active], pa[active])
    for ax in range(3):
        t0, t1, e0, e1 = types(ax, np.where(low, SOLID, AIR))
        v = _dense(tiles, shape, np.ascontiguousarray(vel[:, ax]), F(0))
        lo, hi = _shift(pa, ax, -1, F(0)), _shift(pa, ax, 1, F(0))
        n0, n1 = np.where(e0, F(2) * pa - hi, lo), np.where(e1, F(2) * pa - lo, hi)
        a = np.where(t0 == SOLID, F(2) * pa - n1, np.where(t0 == AIR, -n0, n0))
        b = np.where(t1 == SOLID, F(2) * pa - n0, np.where(t1 == AIR, -n1, n1))
        want = np.where(isf, v - (b - a) * F(0.5), v)
        np.testing.assert_array_equal(_dense(tiles, shape, np.ascontiguousarray(comp[:, ax]), F(0))[active], want[active])
