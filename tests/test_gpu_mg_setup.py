"""The multigrid hierarchy's set-up (cell types and stencil codes, vare_gb300/csrc/multigrid.cu): the
same pool of fluid, away from the walls, in grids whose hierarchies have from three levels to
dense levels of more than 2048 cells (types formed by one CTA, or over the grid). The levels are
aligned with the grid's origin, so the pool's cells have the same types in every grid but for the
coarsest levels: the solver converges in the same number of iterations within two."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu


def _iterations(n):
    rng = np.random.default_rng(2)
    pos = rng.uniform((14.0, 13.0, 12.0), (50.0, 30.0, 51.0), (200000, 3)).astype(np.float32)
    vel = np.stack([np.sin(0.2 * pos[:, 1]), np.cos(0.1 * pos[:, 0]), np.sin(0.15 * pos[:, 2])], 1).astype(np.float32)
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1),
                       flip.default_params(wall_level=-1.0, voxel_size=1.0 / n, dt=1e-3, solver=flip.SOLVER_MIXED))
    sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
    for st in range(4):
        sim.run_stage(st)
    st = sim.stats()
    pres, tiles = sim.field(flip.FIELD_PRES), sim.tiles()
    sim.close()
    assert st["converged"] == 1 and st["residual_rel"] < 1e-6
    return st["solver_iterations"], pres, tiles


@pytest.mark.parametrize("n", [64, 76, 160, 512, 600])
def test_same_pool(gpu, n):
    it, pres, tiles = _iterations(n)
    it0, pres0, tiles0 = _iterations(128)
    assert abs(it - it0) <= 2
    np.testing.assert_array_equal(tiles, tiles0)
    # two solutions within the solver's tolerance of the same one
    assert np.abs(pres - pres0).max() <= 1e-4 * np.abs(pres0).max()
