"""The V-cycle's coarse levels (vare_gb300/csrc/mg_mid.cu) in their forms: one CTA or a cluster
(up to and past 2048 level-3 cells), one or two coarsest cells per thread (a coarsest level
of more than 256 cells below few tiles), batches that hold both. Every form is the same
arithmetic: a simulation gives the same bits alone and in the mix. Its own step outside a
batch has a shallower hierarchy where it is small (the coarsest level is level 2 or 3, run by
the same kernel): the iteration count is within two."""
import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu


def _particles(sim):
    pos, vel, _, ids = sim.particles()
    o = np.argsort(ids)
    return pos[o], vel[o]


@pytest.mark.parametrize("sizes", [(24, 120), (96, 152, 40), (128, 168)])
def test_coarse_forms(gpu, sizes):
    scs = [scenes.small(n, seed=n) for n in sizes]
    # a thin layer in a wide box: few tiles over a coarsest level of 8^3 cells
    scs.append(scenes.dam_break(128, (0.2, 0.1), seed=9))
    dt = scs[0].dt
    mix = [flip.FlipSim.from_scene(sc, solver=flip.SOLVER_MIXED) for sc in scs]
    for _ in range(2):
        assert flip.step_batch(mix, dt) == [0] * len(mix)
    tiles = [m.stats()["active_tiles"] for m in mix]
    if 168 in sizes:
        assert min(tiles) <= 256 and max(tiles) > 2048, tiles
    for sc, m in zip(scs, mix):
        alone = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_MIXED)
        single = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_MIXED)
        for _ in range(2):
            assert flip.step_batch([alone], dt) == [0]
            assert single.step(dt) == 0
        for a, b in zip(_particles(m), _particles(alone)):
            np.testing.assert_array_equal(a, b)
        sm, sa, ss = m.stats(), alone.stats(), single.stats()
        assert sm["converged"] == 1 and sm["residual_rel"] < 1e-6
        assert sm["solver_iterations"] == sa["solver_iterations"]
        assert abs(sm["solver_iterations"] - ss["solver_iterations"]) <= 2
        if ss["active_tiles"] > 512:
            for a, b in zip(_particles(single), _particles(m)):
                np.testing.assert_array_equal(a, b)
        alone.close()
        single.close()
    for m in mix:
        m.close()
