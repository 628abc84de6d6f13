"""Timing the one-launch plain PCG (class pcg_pass of bora_flip_set_profiling): one bracket per
refinement pass, and the timed run gives the bits of the untimed one; a system past the form's size
has no such launch."""
import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu
PASS = flip.KERNEL_CLASSES.index("pcg_pass")


def test_pass_class(gpu):
    sc = scenes.small(32, seed=3)
    sims = [flip.FlipSim.from_scene(sc, solver=flip.SOLVER_PLAIN) for _ in range(2)]
    for sim in sims:
        assert sim.step(sc.dt) == 0
    everything_else = sum(1 << c for c in range(len(flip.KERNEL_CLASSES)) if flip.KERNEL_CLASSES[c] not in ("pcg_direction", "pcg_update"))
    sims[0].set_profiling(everything_else)
    for sim in sims:
        assert sim.step(sc.dt) == 0
    ms, n = sims[0].kernel_times()
    assert n[PASS] == sims[0].stats()["refinements"] > 0 and ms[PASS] > 0.0
    for x, y in zip(sims[0].particles(), sims[1].particles()):
        np.testing.assert_array_equal(x, y)
    for sim in sims:
        sim.close()


def test_per_phase_has_no_pass(gpu):
    sc = scenes.small(24, seed=3)
    sim = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_PLAIN, proj_iteration=(1 << 24) + 1)
    sim.set_profiling(1 << PASS)
    for _ in range(2):
        assert sim.step(sc.dt) == 0
    assert sim.kernel_times()[1][PASS] == 0 and sim.stats()["solver_iterations"] > 0
    sim.close()
