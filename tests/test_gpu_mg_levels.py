"""Cell types and stencil codes of every coarse multigrid level (vare_gb300/csrc/multigrid.cu) against the
rules on dense numpy arrays, exactly: a coarse cell is air when a child inside the domain is, else
fluid when one is, else solid; cells of inactive tiles are air; a fluid cell's code has its fluid
neighbours' bits and 6 + #air - #others, with the wall rule at the domain's faces. Flags at random,
ragged extents, hierarchies from three levels to dense levels of more than 2048 cells."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu
AIR, SOLID, WALL, FLUID, MASKED = 0, 1, 2, 4, 255


def _scatter(tiles, E, values, shape, fill):
    """Tile after tile (x fastest) -> dense (z, y, x); cells beyond `shape` are cut off."""
    t = -(-np.array(shape) // E) if E > 1 else np.array(shape)
    out = np.full(tuple(t * E), fill, values.dtype)
    for (i, j, k), v in zip(tiles, values.reshape(len(tiles), E, E, E)):
        out[E * k:E * k + E, E * j:E * j + E, E * i:E * i + E] = v
    return out[:shape[0], :shape[1], :shape[2]]


def _coarsen(t):
    pad = [(0, n % 2) for n in t.shape]
    t = np.pad(t, pad, constant_values=MASKED)  # children beyond the domain are none
    c = t.reshape(t.shape[0] // 2, 2, t.shape[1] // 2, 2, t.shape[2] // 2, 2)
    air, fluid = (c == AIR).any((1, 3, 5)), (c == FLUID).any((1, 3, 5))
    return np.where(air, AIR, np.where(fluid, FLUID, SOLID)).astype(np.uint8)


def _codes(t, level, voxel_wall):
    j = np.arange(t.shape[1], dtype=np.float32) * np.float32(2 ** level)
    wall = np.where(j + np.float32(0.5) <= np.float32(voxel_wall) + np.float32(1), WALL, AIR).reshape(1, -1, 1)
    wall = np.broadcast_to(wall, t.shape)
    diag, mask = np.full(t.shape, 6), np.zeros(t.shape, int)
    for ax in range(3):  # x, y, z
        n = 2 - ax
        for side, d in ((0, 1), (1, -1)):
            nb = np.roll(t, d, axis=n)
            edge = [slice(None)] * 3
            edge[n] = 0 if side == 0 else -1
            nb[tuple(edge)] = wall[tuple(edge)]
            diag += np.where(nb == AIR, 1, np.where(nb == FLUID, 0, -1))
            mask |= (nb == FLUID).astype(int) << (2 * ax + side)
    return np.where(t == FLUID, 0x8000 | (diag << 8) | mask, 0).astype(np.uint16)


@pytest.mark.parametrize("n,box,share", [((24, 24, 24), 10.0, 0.98), ((20, 28, 12), 18.0, 0.999), ((64, 40, 100), 34.0, 0.999),
                                         ((100, 60, 76), 55.0, 1.0), ((224, 208, 216), 60.0, 0.9999)])
def test_levels(gpu, n, box, share):
    rng = np.random.default_rng(sum(n))
    sim = flip.FlipSim(n, (0, 0, 0), tuple(np.float32(v) for v in n),
                       flip.default_params(wall_level=9.0, voxel_size=1.0, dt=1e-2, solver=flip.SOLVER_MIXED))
    hi = np.minimum(box, np.array(n) - 0.5)
    pos = rng.uniform(0.5, hi, (int(2 * np.prod(hi)), 3)).astype(np.float32)
    if max(n) > 200:  # a second pool, across the far corner
        pos = np.concatenate([pos, rng.uniform(np.array(n) - 20.5, np.array(n) - 0.5, (20000, 3)).astype(np.float32)])
    sim.set_particles(pos, np.zeros_like(pos), space=flip.SPACE_VOXEL)
    sim.run_stage(flip.STAGE_REBUILD)
    sim.run_stage(flip.STAGE_P2G)
    flag = sim.field(flip.FIELD_FLAG)
    real = flag != MASKED
    fluid = (flag == FLUID) | (rng.random(len(flag)) < 0.3)  # the pool, and some of the cells around it
    rare = rng.choice([AIR, SOLID, SOLID], len(flag))
    flag = np.where(real, np.where(fluid & (rng.random(len(flag)) < share), FLUID, np.where(fluid, rare, flag)), MASKED).astype(np.uint8)
    solid = (rng.random(len(flag) // 8) < 0.02).repeat(8) & real  # x-rows of solid cells
    flag[solid] = SOLID
    sim.set_field(flip.FIELD_FLAG, flag)
    sim.run_stage(flip.STAGE_BUILD_SYSTEM)
    tiles = np.asarray(sim.tiles()).reshape(-1, 3)
    want = _scatter(tiles, 8, flag, n[::-1], AIR)
    level, seen = 0, []
    while True:
        try:
            E, (nx, ny, nz), types, codes = sim.mg_level(level)
        except flip.BoraError:
            break
        if level:
            want = _coarsen(want)
        shape = want.shape
        assert shape == (nz, ny, nx)
        wcode = _codes(want, level, 9.0)
        if E:
            active = _scatter(tiles, E, np.ones(len(types), bool), shape, False)
            np.testing.assert_array_equal(_scatter(tiles, E, codes, shape, 0)[active], wcode[active])
            got = _scatter(tiles, E, types, shape, AIR)
            np.testing.assert_array_equal(got, want)
        else:
            np.testing.assert_array_equal(types.reshape(shape), want)
            np.testing.assert_array_equal(codes.reshape(shape), wcode)
        seen.append((E, len(types), int((want == FLUID).sum())))
        level += 1
    sim.close()
    print(n, seen)
    assert level >= 3 and seen[-1][1] <= 512 and seen[2][2] > 0
    if max(n) > 200:
        assert any(e == 0 and c > 2048 for e, c, _ in seen)
