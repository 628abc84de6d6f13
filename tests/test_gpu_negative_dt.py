"""G2P (vare_gb300/csrc/g2p.cu) with a negative time step, which no entry point refuses: the substep
count 1 + trunc(1.5 |v| dt) is then 1, 0 or negative, the substep loop runs once or not at all, and
the table of dt / iter must not be read with such a count. Bit for bit against the oracle from the
oracle's fields; all three kernels, in both loops that advance particles."""
import numpy as np
import pytest

from test_gpu_parity import by_id, tight
from vare_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed", [10.0, 100.0, 5000.0])
@pytest.mark.parametrize("rk2,tank", [(0, 0), (0, 1), (1, 0)])
def test_negative_dt(gpu, oracle_lib, rk2, tank, speed):
    B = oracle_lib
    sc = scenes.small(20, dt=1.0 / 60.0)
    rng = np.random.default_rng(3)
    sc.vel = rng.uniform(-speed, speed, sc.pos.shape).astype(np.float32)
    sim = gpu.FlipSim.from_scene(sc, **tight(advection=gpu.ADVECT_RK2 if rk2 else gpu.ADVECT_EULER, enable_water_tank=tank,
                                             damping_band=6.0))
    ora = B.Oracle(sc, block=8, solver="fp64", tol=1e-13, threads=1, advection=rk2, tank=bool(tank), damping_band=6.0)
    ora.set_particles(sc.pos, sc.vel)
    sim.run_stage(gpu.STAGE_REBUILD)
    sim.run_stage(gpu.STAGE_P2G)
    ora.rebuild(); ora.p2g(); ora.mark(); ora.build_system(); ora.solve(); ora.update_velocity()
    for f in (B.FIELD_VELO, B.FIELD_COMP, B.FIELD_SURF):
        sim.set_field(f, ora.field(f))
    sim.run_stage(gpu.STAGE_UPDATE_PARTICLES, -sc.dt)
    ora.update_particles(-sc.dt)
    ora.compact()
    g, o = by_id(*sim.particles()), by_id(*ora.particles())
    assert 0 < len(o[3])
    for a, b, name in zip(g, o, ("pos", "vel", "adj", "ids")):
        np.testing.assert_array_equal(a, b, err_msg=name)
