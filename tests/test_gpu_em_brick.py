"""The brick pass of the mixed EM step (em_brick_kernel) against the FP64 mode on
the same particles: charge and edge currents after one step, where the pass can
go wrong: boxes smaller than a brick's window and not a multiple of it, every
cell crowded past one 1024-particle batch and past one 7168-particle segment,
speeds near a cell per step (most moves change their cell, many leave the
window or the box), particles that drifted since the last sort."""
import numpy as np
import pytest

from fopis_b200 import RootGrid, _abi

from helpers import em_config, random_particles

pytestmark = pytest.mark.gpu

CURRENTS = (_abi.FIELD_JX, _abi.FIELD_JY, _abi.FIELD_JZ)


def run(n, boundary, precision, per_cell, speed, steps, crowd):
    cfg = em_config(n=n, boundary=boundary, precision=precision, density=1e8)   # so thin that the particles coast
    p = cfg.params
    g = RootGrid(cfg)
    hi = [p.nx - 1 if p.boundary[2 * a] != b"P"[0] else p.nx for a in range(3)]
    crowded = 0
    for s in range(2):
        r = random_particles(int(np.prod(hi)) * per_cell, (0, 0, 0), [1.0] * 3 if crowd else hi, speed, 50 + s, s)
        for k in ("vx", "vy", "vz"):
            r[k] = np.clip(r[k], -0.95, 0.95).astype(np.float32)
        for k in "xyz":   # both modes start from the same single-precision offsets
            f = np.floor(r[k])
            r[k] = f + np.minimum((r[k] - f).astype(np.float32), np.float32(1.0 - 2.0 ** -24)).astype(np.float64)
        cells = np.floor(np.stack([r[k] for k in "xyz"], 1)).astype(int)
        crowded = max(crowded, np.unique(cells, axis=0, return_counts=True)[1].max())
        g.load_particles(s, r)
    g.initialize()
    for _ in range(steps):
        assert g.mainLoopEM(1) == 0
    out = [g.get_field(w) for w in CURRENTS] + [g.getRho(s) for s in range(2)]
    count = [len(g.getParticles(s)) for s in range(2)]
    g.close()
    return out, count, crowded, abs(p.species[0].charge * p.species[0].size)


@pytest.mark.parametrize("n,boundary,per_cell,speed,steps,crowd", [
    (5, "PPPPPP", 6, 0.3, 1, False), (9, "DDDDDD", 8, 0.05, 1, False), (13, "PPDDPP", 4, 0.6, 1, False),
    (18, "DDDDDD", 3, 0.3, 3, False), (11, "PPPPPP", 12, 0.2, 1, True)])
def test_currents_and_charge_match_fp64(gpu_available, n, boundary, per_cell, speed, steps, crowd):
    mixed, cm, crowded, unit = run(n, boundary, _abi.MIXED, per_cell, speed, steps, crowd)
    fp64, c64, _, _ = run(n, boundary, _abi.FP64, per_cell, speed, steps, crowd)
    assert cm == c64
    # One particle's weight on a node: three offsets rounded to 2^-18 and moved in FP32 (2^-24 a step each). Its term on
    # an edge, both halves: FP32 factors and positions, 8 roundings of 2^-24 of at most one crossing, and the unit of the
    # sums. At most 8 (4, two species) times the fullest cell's particles meet at a node (an edge); moves of up to a
    # cell a step can pile neighbours up, so twice that.
    node = 2 * 8 * crowded * unit * (3 * 2.0 ** -18 + 3 * steps * 2.0 ** -24)
    edge = 2 * 8 * crowded * unit * (8 + 3 * steps) * 2.0 ** -24
    for q, (a, b) in enumerate(zip(mixed, fp64)):
        assert np.max(np.abs(a - b)) <= (edge if q < 3 else node), (q, np.max(np.abs(a - b)), edge, node)
        assert np.max(np.abs(b)) > 100 * (edge if q < 3 else node) / crowded   # the bounds mean something
