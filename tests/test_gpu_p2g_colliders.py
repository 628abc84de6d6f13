"""P2G's tile test against box colliders (vare_gb300/csrc/p2g.cu): a tile far from every box skips
the collider samples. Flags and velocities are the same, bit for bit, as with the boxes given
as a sampled field, which no tile skips - for boxes whose faces lie around tile edges, a
box thinner than a cell, one that reaches out of the grid and two of different velocity."""
import numpy as np
import pytest

from test_gpu_parity import _sampled_boxes
from vare_gb300 import flip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxes", [
    [((e, 15.2, 8.0), (e + w, 24.6, 33.0), (3.0, -1.0, 2.0))] for e in (15.4, 16.0, 23.5, 24.6) for w in (0.6, 8.3)
] + [[((-5.0, -2.0, -3.0), (7.4, 8.5, 60.0), (0.0, 4.0, 0.0)), ((31.5, 31.5, 31.5), (40.5, 32.5, 33.5), (1.0, 1.0, 1.0))]])
def test_far_tiles(gpu, boxes):
    n = 48
    rng = np.random.default_rng(4)
    pos = rng.uniform(1.0, n - 1.0, (60000, 3)).astype(np.float32)
    pos = pos[(pos[:, 1] < 30.0) | (pos[:, 0] > 36.0)]  # cells without particles too
    vel = rng.uniform(-5.0, 5.0, pos.shape).astype(np.float32)

    def p2g(field):
        sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1), flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=1e-2))
        if field:
            fi = sim.frame_info()
            sim.set_collider_field(*_sampled_boxes(boxes, 3.0, fi["nx"], fi["ny"], fi["nz"]))
        else:
            sim.set_colliders(boxes, 3.0)
        sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
        sim.run_stage(flip.STAGE_REBUILD)
        sim.run_stage(flip.STAGE_P2G)
        out = sim.field(flip.FIELD_FLAG), sim.field(flip.FIELD_VELO), sim.field(flip.FIELD_MASS)
        sim.close()
        return out

    a, b = p2g(False), p2g(True)
    for u, v, name in zip(a, b, ("flag", "velo", "mass")):
        np.testing.assert_array_equal(u, v, err_msg=name)
    assert len(np.unique(a[0])) >= 2
