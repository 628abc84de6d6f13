"""G2P's kernels (vare_gb300/csrc/g2p.cu) from the oracle's fields, bit for bit: the common case, the
water tank and colliders with Euler advection, RK2; particles that meet a collider (a loop of
their own) next to particles that do not; one substep to more than the table of dt / iter holds
(32); particles killed at the domain's edge."""
import ctypes

import numpy as np
import pytest

from test_gpu_parity import by_id, colliders_for, tight
from vare_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("substeps,speed", [(1, 10.0), (31, 1500.0), (60, 4000.0)])
@pytest.mark.parametrize("rk2,tank,colliders", [(0, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1), (1, 1, 0)])
def test_g2p_modes(gpu, oracle_lib, rk2, tank, colliders, substeps, speed):
    B = oracle_lib
    sc = scenes.small(20, dt=1.0 / 60.0)
    if colliders:
        sc.colliders = colliders_for(20)
    rng = np.random.default_rng(5)
    sc.vel = rng.uniform(-speed, speed, sc.pos.shape).astype(np.float32)
    sim = gpu.FlipSim.from_scene(sc, **tight(advection=gpu.ADVECT_RK2 if rk2 else gpu.ADVECT_EULER, max_substeps=substeps,
                                             enable_water_tank=tank, damping_band=6.0))
    ora = B.Oracle(sc, block=8, solver="fp64", tol=1e-13, threads=1, advection=rk2, tank=bool(tank), damping_band=6.0)
    ora.lib.ora_destroy(ora.h)
    ora.cfg.maxsubsteps = substeps
    ora.h = ora.lib.ora_create(ctypes.byref(ora.cfg))
    if colliders:
        ora.set_colliders(sc.colliders, sc.collider_band)
    ora.set_particles(sc.pos, sc.vel)
    sim.run_stage(gpu.STAGE_REBUILD)
    sim.run_stage(gpu.STAGE_P2G)
    ora.rebuild(); ora.p2g(); ora.mark(); ora.build_system(); ora.solve(); ora.update_velocity()
    for f in (B.FIELD_VELO, B.FIELD_COMP, B.FIELD_SURF):
        sim.set_field(f, ora.field(f))
    sim.run_stage(gpu.STAGE_UPDATE_PARTICLES, sc.dt)
    ora.update_particles(sc.dt)
    ora.compact()
    g, o = by_id(*sim.particles()), by_id(*ora.particles())
    assert 0 < len(o[3])
    for a, b, name in zip(g, o, ("pos", "vel", "adj", "ids")):
        np.testing.assert_array_equal(a, b, err_msg=name)
