"""The solver's tile table (the active tiles that hold a fluid cell, vare_gb300/csrc/projection.cu):
built from the flags that the right-hand-side kernel leaves, or from stencil codes that the
caller has set - both must give the same bits - at tile counts around a thread's 16 flags and
past the table kernel's one round (16384 tiles), with tiles that hold no fluid in between."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu


def _droplets(tiles_per_axis, spacing, seed):
    """Clusters of particles on a lattice of tile centres, falling at different speeds."""
    rng = np.random.default_rng(seed)
    n = 8 * spacing * tiles_per_axis + 16
    c = 8 * spacing * np.stack(np.meshgrid(*[np.arange(tiles_per_axis)] * 3, indexing="ij"), -1).reshape(-1, 3) + 12
    pos = (c[:, None, :] + rng.uniform(-1.5, 1.5, (len(c), 12, 3))).reshape(-1, 3).astype(np.float32)
    vel = rng.uniform(-20, 20, pos.shape).astype(np.float32)
    return n, pos, vel


def _solve(n, pos, vel, solver, set_codes):
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1),
                       flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=1e-3, solver=solver, proj_iteration=2000))
    sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
    for st in (flip.STAGE_REBUILD, flip.STAGE_P2G, flip.STAGE_BUILD_SYSTEM):
        sim.run_stage(st)
    code = sim.field(flip.FIELD_CODE)
    if set_codes:
        sim.set_field(flip.FIELD_CODE, code)
    status = sim.run_stage(flip.STAGE_SOLVE)
    out = sim.field(flip.FIELD_PRES), code, sim.field(flip.FIELD_RHS), sim.stats(), status
    sim.close()
    return out


@pytest.mark.parametrize("solver", [flip.SOLVER_PLAIN, flip.SOLVER_MIXED])
@pytest.mark.parametrize("tiles_per_axis,spacing", [(1, 4), (2, 4), (2, 1), (9, 3)])
def test_solve_tiles(gpu, tiles_per_axis, spacing, solver):
    n, pos, vel = _droplets(tiles_per_axis, spacing, 11)
    pres, code, rhs, st, status = _solve(n, pos, vel, solver, False)
    fluid = (code & 0x8000) != 0
    per_tile = fluid.reshape(-1, 512).any(axis=1)
    if spacing > 2:
        assert 0 < per_tile.sum() < len(per_tile)
    if tiles_per_axis == 9:
        assert len(per_tile) > 16384
    assert status == 0 and st["converged"] == 1 and st["residual_rel"] < 1e-6
    assert np.abs(rhs[fluid]).max() > 0 and np.isfinite(pres).all()
    assert not pres[~fluid].any()
    again = _solve(n, pos, vel, solver, True)
    np.testing.assert_array_equal(again[0], pres)
    assert again[3]["solver_iterations"] == st["solver_iterations"]
