"""Bins of more than 128 particles (dense emissions), ordered by the warp in pieces that are merged
(k_order_bins, vare_gb300/csrc/grid_build.cu): by source index at the sizes around a piece, a merge and
the largest bin that is ordered, alone and with 32 such bins next to each other."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(129,), (255, 256, 257), (383, 384, 385, 130), (511, 512, 513, 7, 20), (1000, 1024, 1025),
                                    (2047, 2049, 128, 4095, 4096), (200,) * 32])
def test_dense_bins(gpu, counts):
    n = 48
    rng = np.random.default_rng(sum(counts))
    cells = np.stack([np.arange(len(counts)) + 8, np.full(len(counts), 9), np.full(len(counts), 10)], 1)  # a warp's neighbours in x
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
    runs = np.flatnonzero(np.diff(cell[ids])) + 1
    assert len(runs) == len(counts) - 1  # one contiguous run per dual cell
    for run in np.split(ids, runs):
        assert (np.diff(run) > 0).all()
