"""Coordinates that the mixed mode's single-precision offsets round up to the
length of a periodic axis: they are at its start, in cell 1 with offset 0, and not
in a cell beyond the arrays. Loaded records, generated plasma (seeds whose draws
hold such a coordinate, found by drawing on the CPU) and injected particles."""
import numpy as np
import pytest

import oracle as orc
from fopis_b200 import PARTICLE_DTYPE, FopisError, RootGrid, _abi, config
from fopis_b200.config import SpeciesInfo, make_params, plasma_units

pytestmark = pytest.mark.gpu


def grid(nxyz, boundary, ppc, seed=1, drift=(0.0, 0.0, 0.0)):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, ppc, drift),
          SpeciesInfo("Ion", "ambient", 100.0, 1.0, 1e7, 1.0, ppc, drift)]
    p, norm = make_params(nxyz, boundary, dx, dt, sp, seed=seed)
    return RootGrid(config.SimConfig(params=p, norm=norm, species=sp)), p


def check(g, p, s, nxyz, count=None):
    cell, f = g.getParticlesRaw(s)
    ijk = np.stack([(cell >> 20) & 1023, (cell >> 10) & 1023, cell & 1023], 1)
    assert count is None or len(cell) == count
    assert np.all(ijk >= 0) and np.all(ijk <= np.array(nxyz))   # cell n is the last of either kind of axis
    W = orc.fixed_deposit(p, cell, f[0], f[1], f[2])
    assert np.array_equal(g.getRho(s), W.astype(np.float64) * (p.species[s].charge * p.species[s].size * 2.0 ** -51))
    return ijk, f


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_loaded_record(gpu_available, axis):
    nxyz = (12, 9, 10)
    g, p = grid(nxyz, "PPPPPP", 1)
    r = np.zeros(2, PARTICLE_DTYPE)
    for k in "xyz":
        r[k] = 4.25
    r["xyz"[axis]] = [nxyz[axis] - 1e-9, nxyz[axis] - 2.0 ** -24]   # rounds up; the largest offset that does not
    r["isValid"] = 1
    g.load_particles(0, r)
    g.initialize()
    ijk, f = check(g, p, 0, nxyz, 2)
    assert sorted(zip(ijk[:, axis], f[axis])) == [(1, 0.0), (nxyz[axis], 1.0 - 2.0 ** -24)]
    r["xyz"[axis]] = nxyz[axis]   # beyond the box: refused as before
    with pytest.raises(FopisError) as e:
        g.load_particles(0, r)
        g.initialize()
    assert e.value.code == _abi.ERR_DEVICE
    g.close()


@pytest.mark.parametrize("seed,axis", [(8911, 1), (31017, 0), (32709, 1)])
def test_generated_plasma(gpu_available, seed, axis):
    nxyz = (16, 16, 16)
    g, p = grid(nxyz, "PPPPPP", 4, seed)
    g.generate_ambient()
    g.initialize()
    ijk, f = check(g, p, 0, nxyz, 4 * 16 ** 3)
    assert np.sum((ijk[:, axis] == 1) & (f[axis] == 0.0)) >= 1
    g.close()


def test_injected_particle(gpu_available):
    nxyz = (97, 61, 45)
    g, p = grid(nxyz, "PPDDNN", 20, 171718608, (300.0, 0.0, 50.0))   # drawn in step 291
    g.initialize()
    assert g.mainLoopES(293) == 0
    check(g, p, 0, nxyz)
    g.close()
