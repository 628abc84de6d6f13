"""The resident plain PCG (vare_gb300/csrc/projection.cu, k_pcg_resident: one warp per solver tile,
blocks that meet twice per iteration) against the per-phase form, which a proj_iteration past
2^24 selects: tile counts around a block's warps, around the change to eight warps per block and
at the form's limit, with and without coupling between tiles. Both forms stop at 1e-9 relative
and the pressures agree to 1e-6 of the largest (a residual of 1e-9 ||b|| leaves an error of at
most cond(A) 1e-9; droplets and these dam breaks have cond(A) below 1e3 per free surface)."""
import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu


def _pressure(res, pos, vel, dt, proj_iteration):
    n = res[0]
    sim = flip.FlipSim(res, (0, 0, 0), tuple(r / n for r in res),
                       flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=dt, solver=flip.SOLVER_PLAIN,
                                           proj_iteration=proj_iteration, tolerance=1e-9, max_refinements=30))
    sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
    for st in (flip.STAGE_REBUILD, flip.STAGE_P2G, flip.STAGE_BUILD_SYSTEM):
        sim.run_stage(st)
    assert sim.run_stage(flip.STAGE_SOLVE) == 0
    launches = sim.stats()["kernel_launches"]
    again = sim.field(flip.FIELD_PRES)
    assert sim.run_stage(flip.STAGE_SOLVE) == 0  # the same words and tags after a first solve
    out = sim.field(flip.FIELD_PRES), sim.field(flip.FIELD_CODE), sim.stats(), launches
    np.testing.assert_array_equal(out[0], again)
    sim.close()
    return out


def _compare(res, pos, vel, dt, tiles=None, resident=True):
    a = _pressure(res, pos, vel, dt, 10000)
    b = _pressure(res, pos, vel, dt, (1 << 24) + 1)
    n = int(((a[1] & 0x8000) != 0).reshape(-1, 512).any(axis=1).sum())
    if tiles is not None:
        assert n == tiles
    # a pass is one launch in the resident form, two per iteration otherwise
    assert a[3] < b[3] if resident else a[3] == b[3]
    assert a[2]["converged"] and b[2]["converged"]
    assert np.abs(a[0]).max() > 0
    assert np.abs(a[0] - b[0]).max() <= 1e-6 * np.abs(b[0]).max()


@pytest.mark.parametrize("tiles", [1, 3, 4, 5, 255, 256, 257, 608, 609])
def test_tile_counts(gpu, tiles):
    """Droplets, one tile each."""
    rng = np.random.default_rng(tiles)
    c = 16 * np.stack(np.meshgrid(*[np.arange(9)] * 3, indexing="ij"), -1).reshape(-1, 3)[:tiles] + 12
    pos = (c[:, None, :] + rng.uniform(-1.5, 1.5, (tiles, 30, 3))).reshape(-1, 3).astype(np.float32)
    vel = rng.uniform(-20, 20, pos.shape).astype(np.float32)
    _compare((160, 160, 160), pos, vel, 1e-3, tiles, resident=tiles <= 608)


@pytest.mark.parametrize("n", [20, 44, 76])
def test_coupled_tiles(gpu, n):
    sc = scenes.small(n, seed=n)
    rng = np.random.default_rng(n)
    x = sc.pos / n * np.pi
    vel = np.stack([np.sin(x[:, 0]) * np.cos(x[:, 1]), -np.cos(x[:, 0]) * np.sin(x[:, 1]), 0 * x[:, 2]], 1) * 50
    vel = (vel * rng.uniform(0.9, 1.1, vel.shape)).astype(np.float32)
    _compare(sc.res, sc.pos, vel, sc.dt)
