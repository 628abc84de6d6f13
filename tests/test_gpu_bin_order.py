"""The order of the particles inside a dual cell (k_order_bins, vare_gb300/csrc/grid_build.cu): by
source index, for bins around the sizes where the sort changes (16 in a lane's registers, 32, 64
and 128 by the warp, more by insertion), alone and next to each other."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(2, 15, 16, 17, 18, 27), (31, 32, 33, 1, 63, 64, 65), (127, 128, 129, 96, 97, 300), (20,) * 40])
def test_bins_in_source_order(gpu, counts):
    n = 32
    rng = np.random.default_rng(sum(counts))
    cells = rng.permutation(np.stack(np.meshgrid(*[np.arange(4, 14)] * 3, indexing="ij"), -1).reshape(-1, 3))[:len(counts)]
    if counts[0] == 20:  # a warp's neighbours along x
        cells = np.stack([np.arange(len(counts)) % 20 + 4, np.arange(len(counts)) // 20 + 5, np.full(len(counts), 6)], 1)
    cell = np.repeat(np.arange(len(counts)), counts)
    pos = (cells[cell] + 0.5 + rng.uniform(0.05, 0.95, (len(cell), 3))).astype(np.float32)
    order = rng.permutation(len(cell))
    pos, cell = pos[order], cell[order]
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1), flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=1e-6))
    sim.set_particles(pos, np.zeros_like(pos), space=flip.SPACE_VOXEL)
    sim.run_stage(flip.STAGE_REBUILD)
    sim.run_stage(flip.STAGE_P2G)
    sim.run_stage(flip.STAGE_UPDATE_PARTICLES, 1e-6)
    ids = sim.particles()[3]  # written in the sorted order; an id is a source index
    sim.close()
    assert sorted(ids) == list(range(len(cell)))
    c = cell[ids]
    runs = np.flatnonzero(np.diff(c)) + 1
    assert len(runs) == len(counts) - 1  # one contiguous run per dual cell
    for run in np.split(ids, runs):
        assert (np.diff(run) > 0).all()
