"""The factorisation kernel against the assembled matrix, on both sides of the row width at which its form changes (80
blocks of 3x3, 64 of 4x4) and where a pivot's list takes one fetch, several, and a part of one."""
import numpy as np
import pytest

from cfdsfemmpi_b200 import meshgen
from cfdsfemmpi_b200._lib import ilu_pattern_build

pytestmark = pytest.mark.gpu

CASES = [("quad", 2), ("quad", 19), ("quad", 20), ("quad", 45), ("hex", 2), ("hex", 4), ("hex", 6)]


@pytest.mark.parametrize("kind,n", CASES, ids=["%s%d" % c for c in CASES])
def test_complete_factors_multiply_to_the_matrix(kind, n):
    """Row i of A - L U.  A block of it is a sum of at most w products of ndof terms each, taken off one at a time: at
    most (w ndof + 2) u of |L| |U|, u = 2^-53.  The multipliers use the stored inverse D of U_pp, so that L_ip U_pp is
    W (D U_pp): (D U_pp - I) of |L_ip| |U_pp| on top, and the rounding of that product."""
    sp = pytest.importorskip("scipy.sparse")
    from cfdsfemmpi_b200 import Handle
    mesh = meshgen.cavity2d(n) if kind == "quad" else meshgen.cavity3d(n)
    h = Handle(mesh, meshgen.control_for(5, 0.1, 0.01), ksp="preonly", pc="bjacobi", ilu_levels=-1)
    rng = np.random.default_rng(5)
    h.set_element_state(*[rng.uniform(-1, 1, h.n) for _ in range(3)])
    vals, _ = h.assemble_export(0)
    p, f = h.export_pattern(), h.ilu_factors()
    N, nb = mesh.nNode, mesh.ndof
    perm = ilu_pattern_build(mesh, -1, 1)["perm"]
    dof = (perm[:, None] * nb + np.arange(nb)).ravel()
    A = sp.bsr_matrix((vals, p["colidx"], p["rowptr"]), shape=(h.n, h.n)).tocsr()[dof][:, dof].toarray()
    rows = np.repeat(np.arange(N), np.diff(f["rowptr"]))
    F = sp.bsr_matrix((f["vals"], f["colidx"], f["rowptr"]), shape=(h.n, h.n)).toarray()
    block = np.repeat(np.arange(N), nb)
    low = block[:, None] > block[None, :]
    L, U = np.where(low, F, 0.0) + np.eye(h.n), np.where(low, 0.0, F)
    u, w = 2.0 ** -53, int(np.bincount(rows).max())
    D, Ud = f["dinv"], f["vals"][f["diag"]]
    off = np.abs(D @ Ud - np.eye(nb)) + 2 * (nb + 2) * u * (np.abs(D) @ np.abs(Ud))
    E = sp.block_diag(list(np.abs(Ud) @ off)).toarray()
    bound = 2 * (w * nb + 4) * u * (np.abs(L) @ np.abs(U)) + 2 * np.abs(L) @ E
    assert np.all(np.abs(A - L @ U) <= bound + 1e-300)
