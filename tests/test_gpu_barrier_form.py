"""k_pcg_persistent (vare_gb300/csrc/projection.cu), the one-launch plain PCG with grid barriers: it runs
with persistent = 1 on systems past the resident form's size, and on smaller ones with a
proj_iteration past 2^24, which the resident form does not take. Which form ran is read from the
launches of the update class: one per refinement pass here, one per iteration and pass in the
per-phase form. Against that form, the FP64 oracle, itself, and with every barrier wait running out."""
import time

import numpy as np
import pytest

from oracle import parity
from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu
PAST = (1 << 24) + 1
UPDATE = flip.KERNEL_CLASSES.index("pcg_update")


def _step(sc, steps, **params):
    sim = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_PLAIN, **params)
    for k in range(steps):
        sim.set_profiling(1 << UPDATE if k == steps - 1 else 0)
        assert sim.step(sc.dt) == 0
    n, st = sim.kernel_times()[1][UPDATE], sim.stats()
    pos, vel, _, ids = sim.particles()
    pres = sim.field(flip.FIELD_PRES)
    sim.close()
    o = np.argsort(ids)
    if params["persistent"]:
        assert n == st["refinements"] > 0
    else:
        assert n == st["refinements"] + st["solver_iterations"]
    assert st["converged"]
    return pos[o], vel[o], pres


@pytest.mark.parametrize("n,proj_iteration", [(24, PAST), (48, PAST), (112, 10000), (112, PAST)])
def test_agrees_with_per_phase(gpu, n, proj_iteration):
    sc = scenes.small(n)
    a = _step(sc, 2, persistent=1, proj_iteration=proj_iteration)
    b = _step(sc, 2, persistent=0, proj_iteration=PAST)
    for x, y, tol in zip(a, b, (1e-6, 1e-5, 1e-5)):
        assert parity.rel_err(x, y) < tol


def test_matches_fp64_oracle(gpu, oracle_lib):
    sc = scenes.small(24)
    ora0 = oracle_lib.Oracle(sc, block=8, solver="fp64", tol=1e-13)
    for _ in range(2):
        ora0.step(sc.dt)
    pos, vel, _, ids = ora0.particles()
    o = np.argsort(ids)
    state = parity.with_state(sc, pos[o], vel[o])
    ora = parity.oracle_step(state)
    dev = parity.device_step(flip, state, solver=flip.SOLVER_PLAIN, persistent=1, proj_iteration=PAST)
    e = parity.compare(dev, ora)
    assert e["same_tiles"] and e["same_particles"] and e["converged"]
    assert e["pressure"] <= 1e-5 and e["grid_velocity"] <= 1e-5 and e["particle_velocity"] <= 1e-5


def test_deterministic(gpu):
    sc = scenes.small(40)
    for x, y in zip(_step(sc, 2, persistent=1, proj_iteration=PAST), _step(sc, 2, persistent=1, proj_iteration=PAST)):
        assert np.array_equal(x, y)


def test_barrier_wait_runs_out(gpu):
    """A barrier that waits for one block more than the launch has (BORA_FAULT_BARRIER): the kernel
    returns within its limit, the step reports it, and the handle steps normally afterwards."""
    sc = scenes.small(32)
    sim = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_PLAIN, persistent=1, proj_iteration=PAST)
    assert sim.step(sc.dt) == 0  # from rest
    sim.set_fault(flip.FAULT_BARRIER)
    t0 = time.perf_counter()
    with pytest.raises(flip.BoraError) as e:
        sim.step(sc.dt)
    assert e.value.status == -5 and time.perf_counter() - t0 < 10.0  # BORA_ERR_INTERNAL
    sim.set_fault(flip.FAULT_NONE)
    sim.set_particles(sc.pos, sc.vel, space=flip.SPACE_VOXEL)
    sim.set_profiling(1 << UPDATE)
    for _ in range(2):
        assert sim.step(sc.dt) == 0
    assert sim.stats()["converged"] and 0 < sim.kernel_times()[1][UPDATE] < sim.stats()["solver_iterations"]
    sim.close()
