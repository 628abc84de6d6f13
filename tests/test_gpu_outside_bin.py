"""The sort's last bin, the particles outside the grid (vare_gb300/csrc/flip_api.cu, rebuild_sort;
k_order_bins): it ends at the number of live particles, whatever an earlier, larger system has left
in the bins' offsets behind it. The earlier system has the same low-corner tiles with more particles
in them, in reverse source order, and further tiles; the later one's outside particles are put back
onto the face by the wall rule, so that every particle survives the step."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outside", [1, 3, 16, 17, 40, 200])
@pytest.mark.parametrize("earlier", [12, 100, 400])
def test_outside_bin(gpu, outside, earlier):
    n = 64
    rng = np.random.default_rng(outside + earlier)
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1), flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=1e-6))
    # particle i in one cell after the other of the first tile, the last index in the first cell
    c = np.arange(earlier)[::-1] * 300 // earlier
    low = np.stack([c % 7, c // 7 % 7, c // 49], 1) + 0.6
    far = rng.uniform(40, 60, (50, 3))
    a = np.concatenate([low, far]).astype(np.float32)
    inside = np.array([[1.6, 1.6, 1.6], [3.2, 4.1, 2.7], [5.9, 0.7, 6.2]])
    out = rng.uniform(0.5, 6.0, (outside, 3))
    out[:, 0] = -rng.uniform(0.1, 2.0, outside)
    b = np.concatenate([inside, out]).astype(np.float32)
    for pos in (a, b):
        sim.set_particles(pos, np.zeros_like(pos), space=flip.SPACE_VOXEL)
        sim.run_stage(flip.STAGE_REBUILD)
        sim.run_stage(flip.STAGE_P2G)
    sim.run_stage(flip.STAGE_UPDATE_PARTICLES, 1e-6)
    ids = sim.particles()[3]  # in the sorted order
    sim.close()
    first = len(a)  # ids go on over the particles that were replaced
    first = 0 if ids.min() < first else first
    assert sorted(ids - first) == list(range(len(b)))
    assert (np.diff(ids[3:]) > 0).all()  # the outside bin by source index
