"""Charge of the fused step, bit for bit against the fixed-point replay of the
particles it left: the smallest periodic boxes, where folds join nodes that lie
next to each other, periodic and held axes together, and a hot plasma of which much
has left its bricks since the last sort."""
import numpy as np
import pytest

import oracle as orc
from fopis_b200 import RootGrid, config
from fopis_b200.config import SpeciesInfo, make_params, plasma_units

from helpers import random_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxyz,boundary,per_cell,speed,steps", [
    ((3, 4, 5), "PPPPPP", 9, 0.05, 1), ((3, 9, 4), "PPDDPP", 6, 0.1, 2), ((6, 3, 3), "DDPPPP", 6, 0.1, 1),
    ((20, 18, 22), "PPPPPP", 24, 0.5, 6), ((21, 20, 19), "DDPPDD", 40, 0.6, 4)])
def test_rho_matches_replay(gpu_available, nxyz, boundary, per_cell, speed, steps):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, per_cell),
          SpeciesInfo("Ion", "ambient", 100.0, 1.0, 1e7, 1.0, per_cell)]
    p, norm = make_params(nxyz, boundary, dx, dt, sp, tol=1e-10, sort_interval=1000000)
    g = RootGrid(config.SimConfig(params=p, norm=norm, species=sp))
    hi = [n if boundary[2 * a] == "P" else n - 1 for a, n in enumerate(nxyz)]
    for s in range(2):
        g.load_particles(s, random_particles(int(np.prod(hi)) * per_cell, (0, 0, 0), hi, speed, 70 + s, s))
    g.initialize()
    assert g.mainLoopES(steps) == 0
    for s in range(2):
        cell, f = g.getParticlesRaw(s)
        W = orc.fixed_deposit(p, cell, f[0], f[1], f[2])
        q = p.species[s].charge * p.species[s].size
        assert np.array_equal(g.getRho(s), W.astype(np.float64) * (q * 2.0 ** -51))
    # the total adds the species' products with one fused rounding less: an ulp of either term
    a, b = g.getRho(0), g.getRho(1)
    assert np.all(np.abs(g.getRho() - (a + b)) <= 2.0 ** -52 * (np.abs(a) + np.abs(b)))
    g.close()
