"""Stencil codes and right-hand sides that the caller sets between the system's build and the solve
(vare_gb300/csrc/flip_api.cu, stage_solve): the solver's tiles, and the plain form's pivots, follow
the codes. An active tile without fluid gets one isolated fluid cell (six air neighbours, diagonal
12, so its pressure is b / 12), alone in its tile, in a grid whose other tiles keep their fluid."""
import numpy as np
import pytest

from vare_gb300 import flip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [flip.SOLVER_PLAIN, flip.SOLVER_MIXED])
@pytest.mark.parametrize("proj_iteration", [2000, (1 << 24) + 1])  # the plain form's resident and per-phase kernels
@pytest.mark.parametrize("cells", [(0,), (511, 77, 256)])
def test_codes_of_an_empty_tile(gpu, solver, proj_iteration, cells):
    n = 48
    rng = np.random.default_rng(4)
    pos = rng.uniform(9.0, 23.0, (20000, 3)).astype(np.float32)
    vel = rng.uniform(-20, 20, pos.shape).astype(np.float32)
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1),
                       flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=1e-3, solver=solver,
                                           proj_iteration=proj_iteration, tolerance=1e-9, max_refinements=30))
    sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
    for st in (flip.STAGE_REBUILD, flip.STAGE_P2G, flip.STAGE_BUILD_SYSTEM):
        sim.run_stage(st)
    code, rhs = sim.field(flip.FIELD_CODE), sim.field(flip.FIELD_RHS)
    assert sim.run_stage(flip.STAGE_SOLVE) == 0
    before = sim.field(flip.FIELD_PRES)
    empty = np.flatnonzero(~((code & 0x8000) != 0).reshape(-1, 512).any(axis=1))
    assert len(empty) > 3
    tiles = empty[[0, len(empty) // 2, -1]]
    at = np.array([t * 512 + c for t in tiles for c in cells])
    code[at] = 0x8000 | (12 << 8)
    b = np.abs(rhs).max() * np.linspace(0.3, 1.0, len(at)).astype(np.float32)
    rhs[at] = b
    sim.set_field(flip.FIELD_CODE, code)
    sim.set_field(flip.FIELD_RHS, rhs)
    assert sim.run_stage(flip.STAGE_SOLVE) == 0
    st, pres = sim.stats(), sim.field(flip.FIELD_PRES)
    sim.close()
    assert st["converged"] == 1 and np.isfinite(pres).all()
    # a residual of 1e-9 ||b|| leaves at most cond(A) 1e-9 of the largest pressure; cond(A) < 1e3 here
    scale = np.abs(before).max()
    assert np.abs(pres[at] - b / 12).max() <= 1e-6 * max(scale, b.max())
    others = np.ones(len(pres), bool)
    others[at] = False
    assert np.abs(pres[others] - before[others]).max() <= 1e-6 * scale


@pytest.mark.parametrize("solver", [flip.SOLVER_PLAIN, flip.SOLVER_MIXED])
@pytest.mark.parametrize("face", range(6))
def test_neighbour_without_fluid(gpu, face, solver):
    """A code that names a fluid neighbour across a tile's face: in an active tile without fluid the
    neighbour counts as 0; in an inactive tile the code is inconsistent and the solve says so."""
    n = 64
    rng = np.random.default_rng(4)
    pos = rng.uniform(24.5, 39.5, (20000, 3)).astype(np.float32)
    vel = rng.uniform(-20, 20, pos.shape).astype(np.float32)
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1),
                       flip.default_params(wall_level=2.0, voxel_size=1.0 / n, dt=1e-3, solver=solver, proj_iteration=2000))
    sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
    for st in (flip.STAGE_REBUILD, flip.STAGE_P2G, flip.STAGE_BUILD_SYSTEM):
        sim.run_stage(st)
    code, rhs = sim.field(flip.FIELD_CODE), sim.field(flip.FIELD_RHS)
    tiles = {tuple(t): s for s, t in enumerate(np.asarray(sim.tiles()).reshape(-1, 3))}
    fluid = ((code & 0x8000) != 0).reshape(-1, 512).any(axis=1)
    ax, d = face // 2, 1 if face & 1 else -1
    step = np.eye(3, dtype=int)[ax] * d
    cell = (7 if d > 0 else 0) * 8 ** ax + 3 * sum(8 ** a for a in range(3) if a != ax)
    empty = [(t, s) for t, s in tiles.items() if not fluid[s]]
    inner = [s for t, s in empty if tuple(np.add(t, step)) in tiles and not fluid[tiles[tuple(np.add(t, step))]]]
    outer = [s for t, s in empty if tuple(np.add(t, step)) not in tiles]
    assert inner and outer
    for s, ok in ((inner[0], True), (outer[0], False)):
        c, b = code.copy(), rhs.copy()
        c[512 * s + cell] = 0x8000 | (12 << 8) | (1 << face)
        b[512 * s + cell] = np.abs(rhs).max()
        sim.set_field(flip.FIELD_CODE, c)
        sim.set_field(flip.FIELD_RHS, b)
        if ok:
            assert sim.run_stage(flip.STAGE_SOLVE) == 0
            p = sim.field(flip.FIELD_PRES)[512 * s + cell]
            assert abs(p - b.max() / 12) <= 1e-4 * b.max()
        else:
            with pytest.raises(flip.BoraError) as e:
                sim.run_stage(flip.STAGE_SOLVE)
            assert e.value.status == -5  # BORA_ERR_INTERNAL
    sim.close()
