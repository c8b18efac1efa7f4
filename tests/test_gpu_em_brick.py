"""The brick pass of the mixed EM step (em_brick_kernel) against the FP64 mode on
the same particles: charge and edge currents after one step, where the pass can
go wrong: boxes smaller than a brick's window and not a multiple of it, every
cell crowded past one 1024-particle batch and past one 7168-particle segment,
speeds near a cell per step (most moves change their cell, many leave the
window or the box), particles that drifted since the last sort. The charge also
bit for bit against the fixed-point replay of the particles the step left, and
in a crowded cell the currents' totals, to less than one particle's share."""
import numpy as np
import pytest

import oracle as orc
from fopis_b200 import RootGrid, _abi

from helpers import em_config, random_particles

pytestmark = pytest.mark.gpu

CURRENTS = (_abi.FIELD_JX, _abi.FIELD_JY, _abi.FIELD_JZ)


def start(n, boundary, precision, per_cell, speed, lo, hi):
    """A grid with the given particles, the same in both modes, and the number of those in the fullest cell."""
    cfg = em_config(n=n, boundary=boundary, precision=precision, density=1e8)   # so thin that the particles coast
    p = cfg.params
    g = RootGrid(cfg)
    if hi is None:
        hi = [p.nx - 1 if p.boundary[2 * a] != b"P"[0] else p.nx for a in range(3)]
    count = int(np.prod([p.nx - 1 if p.boundary[2 * a] != b"P"[0] else p.nx for a in range(3)])) * per_cell
    crowded = 0
    for s in range(2):
        r = random_particles(count, lo, hi, speed, 50 + s, s)
        for k in ("vx", "vy", "vz"):
            r[k] = np.clip(r[k], -0.95, 0.95).astype(np.float32)
        for k in "xyz":   # both modes start from the same single-precision offsets
            f = np.floor(r[k])
            r[k] = f + np.minimum((r[k] - f).astype(np.float32), np.float32(1.0 - 2.0 ** -24)).astype(np.float64)
        cells = np.floor(np.stack([r[k] for k in "xyz"], 1)).astype(int)
        crowded = max(crowded, np.unique(cells, axis=0, return_counts=True)[1].max())
        g.load_particles(s, r)
    g.initialize()
    return g, crowded, abs(p.species[0].charge * p.species[0].size), count


def run(n, boundary, precision, per_cell, speed, steps, crowd):
    g, crowded, unit, _ = start(n, boundary, precision, per_cell, speed, (0, 0, 0), [1.0] * 3 if crowd else None)
    for _ in range(steps):
        assert g.mainLoopEM(1) == 0
    out = [g.get_field(w) for w in CURRENTS] + [g.getRho(s) for s in range(2)]
    count = [len(g.getParticles(s)) for s in range(2)]
    g.close()
    return out, count, crowded, unit


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


@pytest.mark.parametrize("n,boundary,per_cell,speed,steps,lo,hi", [
    (5, "PPPPPP", 6, 0.3, 1, (0, 0, 0), None), (9, "DDDDDD", 8, 0.05, 1, (0, 0, 0), None),
    (13, "PPDDPP", 4, 0.6, 1, (0, 0, 0), None), (18, "DDDDDD", 3, 0.3, 3, (0, 0, 0), None),
    (11, "PPPPPP", 12, 0.2, 1, (0, 0, 0), (1, 1, 1)), (13, "DDDDDD", 5, 0.3, 2, (3, 7, 8), (4, 8, 9)),
    (4, "PPPPPP", 12, 0.3, 14, (0, 0, 0), None), (9, "PPPPPP", 6, 0.6, 20, (0, 0, 0), None)])
def test_charge_matches_replay(gpu_available, n, boundary, per_cell, speed, steps, lo, hi):
    """The last two: particles that leave their brick's window and come back into it, around the box, between sorts."""
    g, _, _, _ = start(n, boundary, _abi.MIXED, per_cell, speed, lo, hi)
    for _ in range(steps):
        assert g.mainLoopEM(1) == 0
    p = g.cfg.params
    for s in range(2):
        cell, f = g.getParticlesRaw(s)
        W = orc.fixed_deposit(p, cell, f[0], f[1], f[2])
        assert np.array_equal(g.getRho(s), W.astype(np.float64) * (p.species[s].charge * p.species[s].size * 2.0 ** -51))
    g.close()


@pytest.mark.parametrize("per_cell", [1, 5, 9])
def test_crowded_current_totals(gpu_available, per_cell):
    """1728, 8640 and 15552 particles of a species in one cell: batches of 1024 and segments of 7168 with remainders.
    The edges of a direction add up to the sum of the particles' velocities."""
    total, vmax = [], 0.0
    for precision in (_abi.MIXED, _abi.FP64):
        g, crowded, unit, count = start(13, "DDDDDD", precision, per_cell, 0.2, (5, 6, 7), (6, 7, 8))
        assert crowded == count
        assert g.mainLoopEM(1) == 0
        total.append([g.get_field(w).sum() for w in CURRENTS])
        g.close()
    # a move's terms of one direction: four or, where it changes its cell, two times four, each the product of FP32
    # factors (6 roundings of 2^-24 of its share of at most one crossing) rounded to the unit of 2^-24 (half of it)
    bound = 2 * count * unit * (6 + 4) * 2.0 ** -24
    assert np.max(np.abs(np.subtract(*total))) <= bound
    assert bound < 0.1 * unit   # less than half the share of a typical particle, 0.2 of a crossing
