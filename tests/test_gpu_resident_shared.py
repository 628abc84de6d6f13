"""The resident plain PCG (k_pcg_resident, vare_gb300/csrc/projection.cu) where its launches share
something: several simulations stepped at the same time from threads of their own (cooperative grids
next to each other and to other kernels), and one simulation's words whose tags start over (a launch
takes 2 max_inner + 2 of the 2^32 tags, so 128 launches at the largest proj_iteration that the form
takes). The same bits as alone, and as with few tags."""
import threading

import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu


def _run(sc, steps, **params):
    sim = flip.FlipSim.from_scene(sc, solver=flip.SOLVER_PLAIN, **params)
    passes = 0
    for _ in range(steps):
        assert sim.step(sc.dt) == 0
        passes += sim.stats()["refinements"]
    out = sim.particles()
    sim.close()
    return out, passes


def test_threads(gpu):
    sizes = [24, 64, 80, 40, 88, 64]  # 5 to 64 blocks each, four and eight warps a block
    scs = [scenes.small(n, seed=n + k) for k, n in enumerate(sizes)]
    alone = [_run(sc, 4)[0] for sc in scs]
    got, errors = [None] * len(scs), []

    def work(k):
        try:
            got[k] = _run(scs[k], 4)[0]
        except Exception as e:  # reported below
            errors.append((sizes[k], e))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(scs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, b in zip(alone, got):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)


def test_tags_start_over(gpu):
    sc = scenes.small(20, seed=5)
    a, passes = _run(sc, 80, proj_iteration=1 << 24)
    assert passes > 140
    b, _ = _run(sc, 80, proj_iteration=10000)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
