"""The plain form's block-MIC(0) factor and sweeps and the direction's operator on the device
(vare_gb300/csrc/projection.cu), seen through one PCG iteration from zero: the pressure is then
alpha z with z = M^-1 b and alpha = b.z / z.Az. Both forms: the resident kernel's rolled sweeps
(four and eight warps per block), the per-phase kernels' unrolled ones. Against plain loops over the
cells of every tile, the factor in FP32 by the same operations, the sweeps in FP64.

All of M^-1 is >= 0, and each of the 2 * 22 steps rounds at most three times, so a cell of z is off by
at most 3 * 44 * 2^-24 (M^-1 |b|), and alpha and the two roundings that follow add less than 20 * 2^-24
of it: 1e-5 bounds both."""
import numpy as np
import pytest

from vare_gb300 import flip, scenes

pytestmark = pytest.mark.gpu
DIRECTION = flip.KERNEL_CLASSES.index("pcg_direction")


def _planes():
    c = np.arange(512)
    s = (c & 7) + ((c >> 3) & 7) + (c >> 6)
    return [c[s == p] for p in range(22)]


def _nbr(c, ax, d):
    """The cell next to c in its tile, or None where that is another tile."""
    x = ((c & 7), ((c >> 3) & 7), (c >> 6))[ax] + d
    return c + d * 8 ** ax if 0 <= x < 8 else None


def _factor(code):
    """FP32, the device's operations; squared pivots, (tiles, 512)."""
    F = np.float32
    m = np.zeros(code.shape, F)
    diag = ((code >> 8) & 15).astype(F)
    for c in np.concatenate(_planes()):
        e, e2 = diag[:, c].copy(), np.zeros(len(code), F)
        for ax in range(3):
            n = _nbr(c, ax, -1)
            if n is None:
                continue
            on = (code[:, c] >> (2 * ax)) & 1 != 0
            ab = np.zeros(len(code), F)
            for o in range(3):
                if o != ax and _nbr(n, o, 1) is not None:
                    ab += ((code[:, n] >> (2 * o + 1)) & 1).astype(F)
            M = m[:, n] * m[:, n]
            e = np.where(on, e - M, e)
            e2 = np.where(on, e2 + ab * M, e2)
        e = e - F(0.97) * e2
        e = np.where(e < diag[:, c] * F(0.25), diag[:, c], e)
        m[:, c] = np.where(code[:, c] & 0x8000 != 0, F(1) / np.sqrt(e + F(1e-30)), F(0))
    return (m * m).astype(np.float64)


def _sweeps(m2, r):
    w = np.zeros(r.shape)
    for c in np.concatenate(_planes()):
        t = r[:, c].copy()
        for ax in range(3):
            n = _nbr(c, ax, -1)
            if n is not None:
                t += w[:, n]
        w[:, c] = m2[:, c] * t
    z = w
    for c in np.concatenate(_planes())[::-1]:
        t = np.zeros(len(r))
        for ax in range(3):
            n = _nbr(c, ax, 1)
            if n is not None:
                t += z[:, n]
        z[:, c] += m2[:, c] * t
    return z


def _apply(tiles, code, z, shape):
    def dense(v):
        out = np.zeros(shape, v.dtype)
        for (i, j, k), t in zip(tiles, v.reshape(-1, 8, 8, 8)):
            out[8 * k:8 * k + 8, 8 * j:8 * j + 8, 8 * i:8 * i + 8] = t
        return out
    c, d = dense(code), dense(z)
    q = ((c >> 8) & 15) * d
    for ax in range(3):
        for b, s in ((0, 1), (1, -1)):
            q -= np.where((c >> (2 * ax + b)) & 1, np.roll(d, s, axis=2 - ax), 0.0)
    return np.stack([q[8 * k:8 * k + 8, 8 * j:8 * j + 8, 8 * i:8 * i + 8].ravel() for i, j, k in tiles])


def _scene(n, kind):
    rng = np.random.default_rng(n)
    if kind == "droplets":  # single tiles, single cells and cells at a tile's corners among them
        c = 16 * np.stack(np.meshgrid(*[np.arange(n // 16)] * 3, indexing="ij"), -1).reshape(-1, 3) + 12
        w = rng.choice([0.3, 1.5, 5.0], len(c))
        pos = (c[:, None, :] + rng.uniform(-1, 1, (len(c), 30, 3)) * w[:, None, None]).reshape(-1, 3)
    else:
        pos = scenes.small(n, seed=n).pos
    pos = np.clip(pos, 0.1, n - 0.1).astype(np.float32)
    return pos, rng.uniform(-20, 20, pos.shape).astype(np.float32)


@pytest.mark.parametrize("per_phase", [False, True])
@pytest.mark.parametrize("n,kind", [(24, "dam"), (44, "dam"), (80, "dam"), (48, "droplets"), (88, "droplets")])
def test_one_iteration(gpu, n, kind, per_phase):
    pos, vel = _scene(n, kind)
    sim = flip.FlipSim((n, n, n), (0, 0, 0), (1, 1, 1),
                       flip.default_params(wall_level=0.4, voxel_size=1.0 / n, dt=1e-3, solver=flip.SOLVER_PLAIN,
                                           proj_iteration=1, max_refinements=1, tolerance=1e-12, div_tolerance=1e-12))
    sim.set_particles(pos, vel, space=flip.SPACE_VOXEL)
    if per_phase:
        sim.set_profiling(1 << DIRECTION)
    for st in (flip.STAGE_REBUILD, flip.STAGE_P2G, flip.STAGE_BUILD_SYSTEM, flip.STAGE_SOLVE):
        sim.run_stage(st)
    assert sim.stats()["solver_iterations"] == 1
    assert sim.kernel_times()[1][DIRECTION] == per_phase
    tiles = np.asarray(sim.tiles()).reshape(-1, 3)
    code = sim.field(flip.FIELD_CODE).reshape(-1, 512).astype(np.int64)
    b = sim.field(flip.FIELD_RHS).reshape(-1, 512).astype(np.float64)
    p = sim.field(flip.FIELD_PRES).reshape(-1, 512).astype(np.float64)
    t = sim.frame_info()
    sim.close()
    m2 = _factor(code)
    z = _sweeps(m2, b)
    q = _apply(tiles, code, z, (8 * t["tz"], 8 * t["ty"], 8 * t["tx"]))
    alpha = (b * z).sum() / (z * q).sum()
    bound = 1e-5 * abs(alpha) * _sweeps(m2, np.abs(b))
    assert np.abs(p).max() > 0
    assert (np.abs(p - alpha * z) <= bound).all()
