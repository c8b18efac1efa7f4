"""The per-brick body marks that let the brick passes skip the body test: two
bodies added one after the other (each marks the bricks anew), particles that
cross into them from every side, and the absorbed counts of one step against the
cell lists of the bodies. Electrons and ions coincide and the bodies are
uncharged, so nothing but the move acts; offsets are odd multiples of 1/128 and
velocities multiples of 1/64, so the moves are exact and end inside a cell."""
import numpy as np
import pytest

from fopis_b200 import PARTICLE_DTYPE, RootGrid, config
from fopis_b200.config import SpeciesInfo, make_params, objects_from_boxes, plasma_units

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxyz,first,second", [
    ((33, 30, 35), ((-12, -3, -2), (-9, 3, 4)), ((5, 4, -7), (8, 7, -4))),
    ((18, 19, 41), ((2, -1, -16), (5, 2, -11)), ((-6, -6, 9), (-2, -3, 17)))])
def test_absorbed_counts(gpu_available, nxyz, first, second):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, 8), SpeciesInfo("Ion", "ambient", 100.0, 1.0, 1e7, 1.0, 8)]
    p, norm = make_params(nxyz, "DDDDDD", dx, dt, sp, sort_interval=1000000)
    objs = [objects_from_boxes([b], nxyz) for b in (first, second)]
    owner = np.full([n + 2 for n in nxyz], -1)
    for o, obj in enumerate(objs):
        owner[tuple(np.asarray(obj.cells).T)] = o
    rng = np.random.default_rng(5)
    n = 60000
    x = np.stack([rng.integers(0, m - 1, n) + (2 * rng.integers(0, 64, n) + 1) / 128.0 for m in nxyz], 1)
    v = rng.integers(-48, 49, (n, 3)) / 64.0
    outside = owner[tuple(np.floor(x).astype(int).T + 1)] < 0
    x, v = x[outside], v[outside]
    end = x + v
    inside = np.all((end >= 0) & (end < np.array(nxyz) - 1), 1)
    hit = owner[tuple(np.floor(end[inside]).astype(int).T + 1)]
    g = RootGrid(config.SimConfig(params=p, norm=norm, species=sp, objects=objs))
    for o in range(2):
        g.initializeObjectsCmatrix(o)
    for s in range(2):
        r = np.zeros(len(x), PARTICLE_DTYPE)
        for a, k in enumerate("xyz"):
            r[k], r["v" + k] = x[:, a], v[:, a]
        r["typeId"], r["isValid"] = s, 1
        g.load_particles(s, r)
    g.initialize()
    assert g.mainLoopES(1) == 0
    for o in range(2):
        assert np.sum(hit == o) > 10
        current = g.getObject(o)[2]
        for s in range(2):
            assert round(current[s] / (p.species[s].charge * p.species[s].size)) == np.sum(hit == o)
    g.close()
