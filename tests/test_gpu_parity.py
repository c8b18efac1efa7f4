"""GPU parity: libfopis_gpu.so through its C ABI against the FP64 oracle.

Tolerances: particle positions and velocities within 1e-5
relative after a step; rho bit-exact against the fixed-point replay of the
same split-precision particles; phi within 1e-7 relative of the converged FP64
solve (solver tolerance 1e-10 here; the 1e-8 default is checked separately);
spacecraft potential within 1 %.
"""
import numpy as np
import pytest

import oracle as orc
from fopis_b200 import RootGrid, _abi, config
from fopis_b200.config import SpeciesInfo, make_params, plasma_units

from helpers import as_f32_state, match, random_particles, rel_err

pytestmark = pytest.mark.gpu


def periodic_cfg(n=16, ppc=4, tol=1e-10):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, ppc),
          SpeciesInfo("Ion", "ambient", 100.0, 1.0, 1e7, 1.0, ppc)]
    p, norm = make_params((n, n, n), "PPPPPP", dx, dt, sp, tol=tol, sort_interval=1000000)
    return config.SimConfig(params=p, norm=norm, species=sp)


def dirichlet_cfg(n=33, ppc=4, tol=1e-10, boundary="DDDDDD"):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, ppc),
          SpeciesInfo("Ion", "ambient", 100.0, 1.0, 1e7, 1.0, ppc)]
    p, norm = make_params((n, n, n), boundary, dx, dt, sp, tol=tol, sort_interval=1000000)
    return config.SimConfig(params=p, norm=norm, species=sp)


def load_both(cfg, parts):
    g = RootGrid(cfg)
    o = orc.Oracle(cfg.params, cfg.objects)
    o.set_solver(1, exact_tol=1e-13)
    for s, recs in enumerate(parts):
        g.load_particles(s, recs)
        o.load_particles(s, as_f32_state(recs))   # the oracle starts from the GPU's split-precision state
    return g, o


def unknown_slices(p):
    sl = []
    for n, b in zip((p.nx, p.ny, p.nz), (p.boundary[0:1], p.boundary[2:3], p.boundary[4:5])):
        sl.append(slice(1, n + 1) if b == b"P" else slice(2, n))
    return tuple(sl)


def demean(a, sl):
    v = a[sl]
    return v - v.mean()


def check_rho_bit_exact(g, cfg):
    for s in range(cfg.params.nspecies):
        cell, f = g.getParticlesRaw(s)
        W = orc.fixed_deposit(cfg.params, cell, f[0], f[1], f[2])
        q = cfg.params.species[s].charge * cfg.params.species[s].size
        expect = W.astype(np.float64) * (q * 2.0 ** -51)
        got = g.getRho(s)
        assert np.array_equal(got, expect), f"species {s}: rho not bit-exact"


def test_initialize_periodic_rho_phi_e(gpu_available):
    cfg = periodic_cfg()
    n = 16 ** 3 * 4
    parts = [random_particles(n, (-1, -1, -1), (16, 16, 16), 0.1, 100 + s, s) for s in range(2)]
    g, o = load_both(cfg, parts)
    assert g.initialize() == 0
    o.initialize()
    check_rho_bit_exact(g, cfg)
    for s in range(2):
        assert rel_err(g.getRho(s), o.field(16 + s)) < 3e-5
    sl = unknown_slices(cfg.params)
    pg, po = g.getPhi(), o.field(0)
    # the rho the GPU solved differs from the oracle's by the 2^-17 weight rounding,
    # so compare phi on the GPU's own rho via the oracle's exact solve
    o2 = orc.Oracle(cfg.params)
    o2.set_solver(1, exact_tol=1e-13)
    o2.set_field(1, g.getRho())
    o2.solve()
    assert rel_err(demean(pg, sl), demean(o2.field(0), sl)) < 1e-7
    assert rel_err(demean(pg, sl), demean(po, sl)) < 1e-3
    # nodal E from the same phi
    o2.update_efield()
    for a, e in enumerate(g.getEref()):
        assert rel_err(e, o2.field(2 + a)) < 1e-6


def test_push_phases_match_oracle(gpu_available):
    cfg = periodic_cfg()
    n = 16 ** 3 * 4
    parts = [random_particles(n, (-1, -1, -1), (16, 16, 16), 0.1, 200 + s, s) for s in range(2)]
    g, o = load_both(cfg, parts)
    g.initialize()
    o.initialize()
    # identical phi on both sides, then E
    o.set_field(0, g.getPhi())
    o.update_efield()
    g.updateEfield()
    g.updateParticleVelocity()
    o.update_velocity()
    for s in range(2):
        a, b, d = match(g.getParticles(s), o.particles(s))
        for k in ("vx", "vy", "vz"):
            assert np.max(np.abs(a[k] - b[k])) < 1e-5 * np.max(np.abs(b[k]))
    g.updateParticlePosition()
    o.update_position()
    for s in range(2):
        a, b, d = match(g.getParticles(s), o.particles(s))
        # per particle: |dx| / max(|x|, 1 cell) and |dv| / |v| within 1e-5
        xa, xb = np.stack([a[k] for k in "xyz"], 1), np.stack([b[k] for k in "xyz"], 1)
        va, vb = (np.stack([r[k] for k in ("vx", "vy", "vz")], 1) for r in (a, b))
        assert np.max(np.linalg.norm(xa - xb, axis=1) / np.maximum(np.linalg.norm(xb, axis=1), 1.0)) < 1e-5
        assert np.max(np.linalg.norm(va - vb, axis=1) / np.linalg.norm(vb, axis=1)) < 1e-5


@pytest.mark.parametrize("boundary,n", [("DDDDDD", 33), ("PPPPPP", 32), ("PPDDPP", 24), ("DDDDDD", 30)])
def test_solver_matches_exact_fp64(gpu_available, boundary, n):
    cfg = dirichlet_cfg(n=n, boundary=boundary)
    p = cfg.params
    rng = np.random.default_rng(5)
    shape = (p.nx + 2, p.ny + 2, p.nz + 2)
    rho = np.zeros(shape)
    sl = unknown_slices(p)
    rho[sl] = rng.standard_normal(rho[sl].shape) * 1e6 + 3e5 * np.sin(np.arange(rho[sl].shape[0]))[:, None, None]
    g = RootGrid(cfg)
    g.set_field(_abi.FIELD_RHO0, rho)
    assert g.solvePoisson() == 0
    st = g.stats()
    assert st.converged and st.residual_last <= 1e-10
    o = orc.Oracle(p)
    o.set_solver(1, exact_tol=1e-13)
    o.set_field(1, rho)
    o.solve()
    assert rel_err(demean(g.getPhi(), sl), demean(o.field(0), sl)) < 1e-7
    if boundary == "DDDDDD":
        assert rel_err(g.getPhi(), o.field(0)) < 1e-7


def test_solver_default_tolerance_error(gpu_available):
    cfg = dirichlet_cfg(n=65, tol=1e-8)
    p = cfg.params
    rng = np.random.default_rng(9)
    rho = np.zeros((p.nx + 2,) * 3)
    rho[2:-2, 2:-2, 2:-2] = rng.standard_normal((63, 63, 63)) * 1e6
    g = RootGrid(cfg)
    g.set_field(_abi.FIELD_RHO0, rho)
    g.solvePoisson()
    st = g.stats()
    assert st.converged and st.vcycles_last <= 3   # direct corrections
    o = orc.Oracle(p)
    o.set_solver(1, exact_tol=1e-13)
    o.set_field(1, rho)
    o.solve()
    assert rel_err(g.getPhi(), o.field(0)) < 1e-6


def test_fused_step_equals_phased_step(gpu_available):
    cfg = periodic_cfg()
    n = 16 ** 3 * 4
    parts = [random_particles(n, (-1, -1, -1), (16, 16, 16), 0.1, 300 + s, s) for s in range(2)]
    a = RootGrid(cfg)
    b = RootGrid(cfg)
    for s in range(2):
        a.load_particles(s, parts[s])
        b.load_particles(s, parts[s])
    a.initialize()
    b.initialize()
    a.mainLoopES(1)
    b.updateParticleVelocity()
    b.emitParticlesFromObjects()
    b.updateParticlePosition()
    b.injectParticlesFromBoundary()
    b.updateRho()
    b.solvePoisson()
    b.updateEfield()
    b.advance_timestep()
    for s in range(2):
        assert np.array_equal(a.getRho(s), b.getRho(s))
    assert np.array_equal(a.getPhi(), b.getPhi())
    pa, pb = a.getEnergy(), b.getEnergy()
    assert abs(pa[0] - pb[0]) <= 1e-9 * abs(pb[0])
    assert abs(pa[1] - pb[1]) <= 1e-12 * abs(pb[1])


def test_multi_step_periodic_tracks_oracle(gpu_available):
    cfg = periodic_cfg(n=16, ppc=4, tol=1e-10)
    n = 16 ** 3 * 4
    parts = [random_particles(n, (0, 0, 0), (16, 16, 16), 0.1, 400 + s, s) for s in range(2)]
    g, o = load_both(cfg, parts)
    g.initialize()
    o.initialize()
    for _ in range(5):
        g.mainLoopES(1)
        o.main_loop(1)
    check_rho_bit_exact(g, cfg)
    pe_g, fe_g = g.getEnergy()
    pe_o, fe_o = o.energy()
    assert abs(pe_g - pe_o) < 1e-5 * pe_o
    assert abs(fe_g - fe_o) < 2e-3 * fe_o
    for s in range(2):
        a, b, d = match(g.getParticles(s), o.particles(s))
        assert np.max(np.abs(a["x"] - b["x"])) < 1e-4


@pytest.mark.parametrize("boundary,n", [("DDDDDD", 33), ("PPDDPP", 24)])
def test_pointwise_residual_matches_reference_measure(gpu_available, boundary, n):
    """fopis_stats.residual_pointwise is RootGrid::checkPhiResidual's measure
    (src/Grid/RootGrid/RootGridField.cpp:267-317) of the solve's result."""
    cfg = dirichlet_cfg(n=n, boundary=boundary, tol=1e-8)
    p = cfg.params
    rng = np.random.default_rng(17)
    rho = np.zeros((p.nx + 2, p.ny + 2, p.nz + 2))
    sl = unknown_slices(p)
    rho[sl] = rng.standard_normal(rho[sl].shape) * 1e6
    g = RootGrid(cfg)
    g.set_field(_abi.FIELD_RHO0, rho)
    assert g.solvePoisson() == 0
    st = g.stats()
    o = orc.Oracle(p)
    o.set_field(0, g.getPhi())
    o.set_field(1, rho)
    ref = o.pointwise_residual()
    assert ref > 0 and abs(st.residual_pointwise - ref) <= 1e-9 * ref, (st.residual_pointwise, ref)
