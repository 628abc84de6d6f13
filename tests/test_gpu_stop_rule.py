"""The stop rule of the plain form's inner PCG, one refinement pass: with persistent = 0 every
check_every-th iteration is tested and one more follows a test that holds, in the resident form
(small systems) as in the per-phase form, which a proj_iteration past 2^24 selects; with persistent = 1
every iteration is tested and the pass ends at once."""
import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu
PER_PHASE = (1 << 24) + 1


def _iterations(sc, vel, proj_iteration, persistent, check):
    sim = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_PLAIN, proj_iteration=proj_iteration, persistent=persistent,
                                  check_every=check, max_refinements=1, tolerance=1e-9)
    sim.set_particles(sc.pos, vel, space=flip.SPACE_VOXEL)
    for st in (flip.STAGE_REBUILD, flip.STAGE_P2G, flip.STAGE_BUILD_SYSTEM, flip.STAGE_SOLVE):
        assert sim.run_stage(st) >= 0
    st = sim.stats()
    sim.close()
    assert st["refinements"] == 1
    return st["solver_iterations"]


@pytest.mark.parametrize("n", [20, 44, 70])  # four and eight warps per block
def test_stop_rule(gpu, n):
    sc = scenes.small(n, seed=n)
    x = sc.pos / n * np.pi
    vel = (np.stack([np.sin(x[:, 0]) * np.cos(x[:, 1]), -np.cos(x[:, 0]) * np.sin(x[:, 1]), 0 * x[:, 2]], 1) * 50).astype(np.float32)
    first = _iterations(sc, vel, 10000, 1, 1)  # the iteration that reaches the target
    assert first > 5
    for form in (10000, PER_PHASE):
        reached = _iterations(sc, vel, form, 0, 1) - 1
        assert abs(reached - first) <= (0 if form == 10000 else 1)  # the forms' sums are rounded differently
        for check in (2, 7, 10 * first):
            assert _iterations(sc, vel, form, 0, check) == -(-reached // check) * check + 1
        assert _iterations(sc, vel, form, 1, 7) in ((first,) if form == 10000 else (first - 1, first, first + 1))
    for limit in (1, first - 1, first):  # a pass never runs past proj_iteration
        assert _iterations(sc, vel, limit, 0, 1) == limit
        assert _iterations(sc, vel, limit, 1, 1) == limit
