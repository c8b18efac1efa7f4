"""The fast-diagonalisation correction of the Poisson solve (direct.cu) at the
sizes where its tiles, passes and folds end: single unknowns, odd and even
periodic axes, axes around the multiples of the 8 modes, 16 matrix rows, 64
lines and 128-mode passes it works in, and axes beyond its limit, which the
multigrid cycle takes as long as it converges: where halved even counts make it
diverge, the direct correction takes over, in the EM mode as well. The residual of the returned potential, formed here in
FP64, has to meet the tolerance the solve reports; a correction lowers it to 1e-3
or less at these sizes, and what it leaves is noise, which the next lowers to 1e-5
or less, so two or three suffice for 1e-10."""
import numpy as np
import pytest

from fopis_b200 import RootGrid, _abi, config
from fopis_b200.config import SpeciesInfo, make_params, plasma_units

from helpers import em_config

pytestmark = pytest.mark.gpu

TOL = 1e-10


def residual(p, rho, phi):
    """||f - A phi|| / ||f|| over the unknowns, faces held at zero, mean-free when every axis is periodic."""
    dims = (p.nx, p.ny, p.nz)
    per = [p.boundary[2 * a:2 * a + 1] == b"P" for a in range(3)]
    inner = tuple(slice(1, n + 1) if q else slice(2, n) for n, q in zip(dims, per))
    f = rho[inner] / p.eps0
    if all(per):
        f = f - f.mean()
    u = phi[inner]
    r = f - 6.0 * u
    for a in range(3):
        for d in (1, -1):
            v = np.roll(u, d, axis=a)
            if not per[a]:
                np.moveaxis(v, a, 0)[0 if d == 1 else -1] = 0.0
            r = r + v
    return np.linalg.norm(r) / np.linalg.norm(f)


@pytest.mark.parametrize("nxyz,boundary,direct", [
    ((3, 3, 3), "DDDDDD", True), ((4, 3, 6), "DDNNDD", True), ((3, 4, 5), "PPPPPP", True),
    ((17, 18, 19), "PPPPPP", True), ((33, 34, 35), "DDDDDD", True), ((66, 35, 34), "DDPPDD", True),
    ((65, 130, 33), "PPDDPP", True), ((130, 131, 20), "DDPPNN", True), ((128, 72, 9), "PPPPPP", True),
    ((145, 146, 60), "PPDDDD", True), ((261, 20, 12), "DDDDDD", True), ((20, 270, 16), "PPPPDD", True),
    ((12, 10, 300), "NNDDPP", True), ((10, 9, 514), "DDDDDD", True), ((66, 50, 58), "DDDDDD", True), ((98, 64, 82), "DDPPDD", True),
    ((9, 8, 515), "DDDDDD", False), ((516, 64, 48), "PPPPDD", False), ((515, 66, 65), "DDDDDD", False),
    ((66, 66, 660), "DDDDDD", False), ((720, 50, 66), "DDDDDD", False), ((42, 1020, 50), "DDPPDD", False)])
def test_residual_meets_tolerance(gpu_available, nxyz, boundary, direct):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, 1)]
    p, norm = make_params(nxyz, boundary, dx, dt, sp, tol=TOL, guess=_abi.GUESS_ZERO)
    g = RootGrid(config.SimConfig(params=p, norm=norm, species=sp))
    rng = np.random.default_rng(31)
    shape = tuple(n + 2 for n in nxyz)
    smooth = sum(np.cos(0.7 + 2.0 * np.pi * np.arange(s) / s).reshape([-1 if q == a else 1 for q in range(3)])
                 for a, s in enumerate(shape))
    rho = rng.standard_normal(shape) * 1e6 + 4e6 * smooth
    g.set_field(_abi.FIELD_RHO0, rho)
    rc = g.solvePoisson()
    st = g.stats()
    phi = g.getPhi()
    g.close()
    assert rc == 0 and st.converged and 1 <= st.vcycles_last
    assert st.vcycles_last <= 3 if direct else st.vcycles_last > 3
    assert residual(p, rho, phi) <= TOL + rounding(p, rho, phi)


def rounding(p, rho, phi):
    """The reported residual is the last one formed; storing phi adds its rounding, 12 ulp of max |phi| a node."""
    return 12 * 2.0 ** -52 * np.abs(phi).max() * np.sqrt(phi.size) / np.linalg.norm(rho / p.eps0)


@pytest.mark.parametrize("n,boundary,boxes", [
    (42, "DDDDDD", None), (50, "DDDDDD", None), (66, "DDDDDD", None), (82, "DDPPDD", None),
    (50, "DDDDDD", [((-2, -2, -2), (2, 2, 2))])])
def test_em_solves_where_v_cycles_fail(gpu_available, n, boundary, boxes):
    """Held axes whose even counts the V-cycles halve: the start-up of an EM run, and with a body its steps."""
    cfg = em_config(n=n, boundary=boundary, ppc=2, boxes=boxes)
    g = RootGrid(cfg)
    if boxes:
        g.initializeObjectsCmatrix(0)
    g.generate_ambient()
    assert g.initialize() == 0
    phi, rho = g.getPhi(), g.getRho()
    assert residual(cfg.params, rho, phi) <= TOL + rounding(cfg.params, rho, phi)
    assert g.mainLoopEM(2) == 0
    if boxes:   # every step solves: by the direct corrections from the first failure on
        st = g.stats()
        assert st.converged and st.solves_step == 1 and 1 <= st.vcycles_step <= 3
    g.close()


@pytest.mark.parametrize("nxyz", [(16, 16, 16), (17, 18, 19), (96, 80, 100)])
def test_near_uniform_periodic_charge(gpu_available, nxyz):
    """Charge that is its mean, or differs from it by little more than roundings: solved to the tolerance, or to a
    rounding of the mean where that is more, from zero and from the last potential."""
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, 1)]
    p, norm = make_params(nxyz, "PPPPPP", dx, dt, sp)
    g = RootGrid(config.SimConfig(params=p, norm=norm, species=sp))
    tol, inner = 1e-8, (slice(1, -1),) * 3
    rng = np.random.default_rng(4)
    for value in (1.0, 0.3, 1e6, 123456.789, -7.7e3, 3e-12, 1.0 / 3.0):
        for noise in (0.0, 1e-15, 1e-12, 1e-10, 1e-8):
            rho = np.pad(value * (1.0 + noise * rng.standard_normal(nxyz)), 1, mode="wrap")
            g.set_guess_mode(_abi.GUESS_ZERO if rng.random() < 0.5 else _abi.GUESS_WARM)
            g.set_field(_abi.FIELD_RHO0, rho)
            assert g.solvePoisson() == 0, (value, noise, g.stats().residual_last)
            phi = g.getPhi()
            f = rho[inner] / p.eps0
            r = f - f.mean() - 6.0 * phi[inner]
            for a in range(3):
                r += np.roll(phi[inner], 1, axis=a) + np.roll(phi[inner], -1, axis=a)
            # a rounding of the mean, as much again for the storing of phi (which the mean's removal rounds anew)
            most = tol * np.linalg.norm(f - f.mean()) + (2.0 ** -53 * abs(f.mean()) + 24 * 2.0 ** -53 * np.abs(phi).max()) * np.sqrt(f.size)
            assert np.linalg.norm(r - r.mean()) <= most
    g.close()


@pytest.mark.parametrize("nxyz,boundary,cap", [
    ((33, 34, 35), "DDDDDD", 100), ((20, 19, 18), "PPPPPP", 100), ((66, 35, 34), "DDPPNN", 100), ((24, 24, 24), "PPPPPP", 1),
    ((515, 66, 65), "DDDDDD", 100)])
def test_host_driven_loop_gives_the_same(gpu_available, monkeypatch, nxyz, boundary, cap):
    """FOPIS_SOLVE_HOST_LOOP=1 runs the same kernels with the host deciding: the same potential bit for bit, the same
    counts and residuals, the hand-over from diverging V-cycles included."""
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, 1)]
    p, norm = make_params(nxyz, boundary, dx, dt, sp, tol=1e-12, guess=_abi.GUESS_ZERO, max_vcycles=cap)
    rho = np.random.default_rng(8).standard_normal(tuple(n + 2 for n in nxyz)) * 1e6 + 3e5
    got = []
    for env in ("0", "1"):
        monkeypatch.setenv("FOPIS_SOLVE_HOST_LOOP", env)
        g = RootGrid(config.SimConfig(params=p, norm=norm, species=sp))
        g.set_field(_abi.FIELD_RHO0, rho)
        rc = g.solvePoisson()
        st = g.stats()
        got.append((rc, st.converged, st.vcycles_last, st.residual_last, st.residual_initial, g.getPhi()))
        g.close()
    assert got[0][0] == (0 if cap > 1 else _abi.ERR_NOT_CONVERGED)
    assert got[0][:5] == got[1][:5] and np.array_equal(got[0][5], got[1][5])
