"""Cells of an edge tile beyond the grid (extents that are not multiples of 8) in the right-hand side,
the stencil codes, the air pressure and the velocity update (vare_gb300/csrc/projection.cu): they count
as air with pressure 0 whatever flags, velocities and pressures the caller has set there, and change
nothing inside the grid."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu
MASKED, FLUID = 255, 4


@pytest.mark.parametrize("n", [(20, 28, 12), (12, 24, 20), (24, 20, 16), (20, 20, 20)])
def test_padded_cells(gpu, n):
    rng = np.random.default_rng(sum(n))
    sim = flip.FlipSim(n, (0, 0, 0), tuple(np.float32(v) for v in n), flip.default_params(wall_level=5.0, voxel_size=1.0, dt=1e-2))
    pos = rng.uniform(0.5, np.array(n) - 0.5, (2000, 3)).astype(np.float32)
    sim.set_particles(pos, np.zeros_like(pos), space=flip.SPACE_VOXEL)
    sim.run_stage(flip.STAGE_REBUILD)
    sim.run_stage(flip.STAGE_P2G)
    flag0 = sim.field(flip.FIELD_FLAG)
    pad = flag0 == MASKED
    assert 0 < pad.sum() < len(pad)
    flag0 = np.where(pad, MASKED, np.where(rng.random(len(pad)) < 0.7, FLUID, 0)).astype(np.uint8)
    vel0 = np.where(pad[:, None], 0, rng.uniform(-1, 1, (len(pad), 3))).astype(np.float32)
    pres0 = np.where(flag0 == FLUID, rng.uniform(-1, 1, len(pad)), 0).astype(np.float32)
    out = []
    for flags in (None, np.full(len(pad), FLUID), rng.choice([0, 1, 2, FLUID], len(pad))):
        flag, vel, pres = flag0.copy(), vel0.copy(), pres0.copy()
        if flags is not None:
            flag[pad] = flags[pad]
            vel[pad] = rng.uniform(1, 2, (pad.sum(), 3))
            pres[pad] = rng.uniform(1, 2, pad.sum())
        sim.set_field(flip.FIELD_FLAG, flag)
        sim.set_field(flip.FIELD_VELO, vel)
        sim.run_stage(flip.STAGE_BUILD_SYSTEM)
        sim.set_field(flip.FIELD_PRES, pres)
        rhs, code = sim.field(flip.FIELD_RHS), sim.field(flip.FIELD_CODE)
        sim.run_stage(flip.STAGE_UPDATE_VELOCITY)
        comp, p = sim.field(flip.FIELD_COMP), sim.field(flip.FIELD_PRES)
        assert not rhs[pad].any() and not code[pad].any() and not p[pad].any()
        np.testing.assert_array_equal(comp[pad], vel[pad])
        out.append((rhs[~pad], code[~pad], comp[~pad], p[~pad]))
    sim.close()
    for a in out[1:]:
        for x, y in zip(out[0], a):
            np.testing.assert_array_equal(x, y)
