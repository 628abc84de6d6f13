"""Vector fields read and written through the solver's x as staging (bora_flip_get_field, set_field):
no device memory is allocated for it, and every cell makes the round trip, at cell counts that take
one piece (the particles' staging) and two (the solver's x holds two thirds of the cells at its full size)."""
import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ppc", [(128, 1), (100, 1), (100, 8)])
def test_no_allocation(gpu, n, ppc):
    import torch
    sc = scenes.dam_break(n, ppc=ppc)
    sim = flip.FlipSim.from_scene(sc)
    sim.run_stage(flip.STAGE_REBUILD)
    sim.run_stage(flip.STAGE_P2G)
    ncell = 512 * len(sim.tiles())
    assert ncell * 12 > 4 << 20  # an allocation for a whole field would show
    sim.field(flip.FIELD_FLAG)
    free = torch.cuda.mem_get_info()[0]
    rng = np.random.default_rng(n)
    v = rng.standard_normal((ncell, 3)).astype(np.float32)
    w = rng.standard_normal((ncell, 3)).astype(np.float32)
    sim.set_field(flip.FIELD_VELO, v)
    sim.set_field(flip.FIELD_COMP, w)
    np.testing.assert_array_equal(sim.field(flip.FIELD_VELO), v)
    np.testing.assert_array_equal(sim.field(flip.FIELD_COMP), w)
    assert free - torch.cuda.mem_get_info()[0] < 1 << 20
    sim.close()


def test_shrunk_system(gpu):
    """A later, smaller system fits the staging in one piece."""
    rng = np.random.default_rng(1)
    sim = flip.FlipSim((96, 96, 96), (0, 0, 0), (1, 1, 1), flip.default_params(wall_level=2.0, voxel_size=1 / 96, dt=1e-4))
    for hi in (90.0, 10.0):
        pos = rng.uniform(2.0, hi, (20000, 3)).astype(np.float32)
        sim.set_particles(pos, np.zeros_like(pos), space=flip.SPACE_VOXEL)
        sim.run_stage(flip.STAGE_REBUILD)
        sim.run_stage(flip.STAGE_P2G)
        v = rng.standard_normal((512 * len(sim.tiles()), 3)).astype(np.float32)
        sim.set_field(flip.FIELD_VELO, v)
        np.testing.assert_array_equal(sim.field(flip.FIELD_VELO), v)
    sim.close()
