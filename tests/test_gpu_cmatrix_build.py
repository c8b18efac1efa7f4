"""The capacity matrix from the Green's function table and the blocked inversion
against numpy in FP64: held, periodic and mixed boxes, bodies off the centre and
beside a face, fewer nodes than one 32-pivot step and counts that leave a
remainder of it. A body on a face has no positive definite matrix and is
refused before any solve. Two parts so far apart that the table takes more than
its 4 GiB go through one solve per node."""
import numpy as np
import pytest

from fopis_b200 import FopisError, RootGrid, _abi, config
from fopis_b200.config import SpeciesInfo, make_params, plasma_units

pytestmark = pytest.mark.gpu


def grid(nxyz, boundary, *boxes):
    dx, dt = plasma_units()
    sp = [SpeciesInfo("Electron", "ambient", 1.0, -1.0, 1e7, 1.0, 1)]
    p, norm = make_params(nxyz, boundary, dx, dt, sp)
    obj = config.objects_from_boxes(list(boxes), nxyz)
    return RootGrid(config.SimConfig(params=p, norm=norm, species=sp, objects=[obj])), p, obj


def response(nxyz, boundary, nodes, eps0):
    """phi at every node for a unit charge at every node, by the eigenvectors of each axis."""
    S, lam, at = [], [], []
    for a in range(3):
        per = boundary[2 * a] == "P"
        n = nxyz[a] if per else nxyz[a] - 2
        A = 2.0 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
        if per:
            A[0, -1] -= 1.0
            A[-1, 0] -= 1.0
        w, v = np.linalg.eigh(A)
        S.append(v)
        lam.append(w)
        at.append(nodes[:, a] - (1 if per else 2))
    L = lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :]
    G = np.where(L > 1e-9, 1.0 / np.maximum(L, 1e-9), 0.0)
    F = np.einsum("ik,il,im->iklm", S[0][at[0]], S[1][at[1]], S[2][at[2]]).reshape(len(nodes), -1)
    return (F * G.ravel()) @ F.T / eps0


@pytest.mark.parametrize("nxyz,boundary,box", [
    ((9, 10, 11), "DDDDDD", ((-1, -1, -1), (0, 0, 0))), ((17, 15, 18), "DDDDDD", ((-5, -3, 2), (-2, 1, 5))),
    ((16, 13, 15), "PPDDPP", ((-3, -2, -2), (2, 2, 3))), ((15, 16, 14), "NDPPDN", ((-2, -4, -3), (2, 1, 3))),
    ((12, 12, 13), "PPPPPP", ((-2, -2, -2), (2, 2, 2))), ((14, 14, 14), "DDDDDD", ((-5, -1, -1), (-3, 1, 1)))])
def test_matches_numpy(gpu_available, nxyz, boundary, box):
    g, p, obj = grid(nxyz, boundary, box)
    g.initializeObjectsCmatrix(0)
    C = g.get_cmatrix(0)
    g.close()
    B = response(nxyz, boundary, np.asarray(obj.nodes, np.int64), p.eps0)
    ref = np.linalg.inv(B)
    # both inverses are backward stable: off by the condition of B times its size times a rounding
    assert np.max(np.abs(C - ref)) <= len(B) * np.linalg.cond(B) * 2.0 ** -52 * np.max(np.abs(ref))


def test_body_on_a_face_is_refused(gpu_available):
    g, _, _ = grid((12, 12, 12), "DDDDDD", ((-6, -1, -1), (-3, 1, 1)))
    with pytest.raises(FopisError) as e:
        g.initializeObjectsCmatrix(0)
    assert e.value.code == _abi.ERR_DEVICE
    assert g.stats().vcycles_step == 0
    g.close()


def test_far_apart_parts_are_solved_node_by_node(gpu_available):
    nxyz = (301, 300, 301)
    g, p, obj = grid(nxyz, "DDDDDD", ((-146, -145, -144), (-145, -144, -143)), ((144, 143, 145), (145, 144, 146)))
    nodes = np.asarray(obj.nodes, np.int64)
    counts = [3 * int(np.ptp(nodes[:, a])) + 2 for a in range(3)]
    assert np.prod(counts, dtype=np.int64) > 1 << 29   # doubles: the table does not fit
    g.initializeObjectsCmatrix(0)
    assert g.stats().vcycles_last >= 1                 # solved
    C = g.get_cmatrix(0)
    g.close()
    # phi at every node for a unit charge at one: sines of each axis, one charge at a time
    S, lam = [], []
    for a in range(3):
        n = nxyz[a] - 2
        k = np.arange(1, n + 1)
        S.append(np.sqrt(2.0 / (n + 1)) * np.sin(np.pi * np.outer(nodes[:, a] - 1, k) / (n + 1)))
        lam.append(2.0 - 2.0 * np.cos(np.pi * k / (n + 1)))
    inv = 1.0 / (lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :])
    B = np.empty((len(nodes), len(nodes)))
    for j in range(len(nodes)):
        t = (inv @ (S[2] * S[2][j]).T)                          # [k][l][i]
        t = np.einsum("kli,il->ki", t, S[1] * S[1][j])
        B[:, j] = np.einsum("ki,ik->i", t, S[0] * S[0][j])
    B /= p.eps0
    ref = np.linalg.inv(B)
    # the solves go to ||r|| <= 1e-10 ||f||, phi off by at most 1e-10 / lambda_min of a unit charge
    off = 1e-10 / min(l.min() for l in lam) / p.eps0 * len(B)
    assert np.linalg.norm(C - ref, 2) <= 2.0 * np.linalg.norm(ref, 2) ** 2 * off
