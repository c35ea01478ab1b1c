"""Restarted GMRES where its kernels' forms change, in long cycles (several columns a thread in the rotations, back
substitution over many blocks, more than one batch of terms in the update, a CTA per vector from 148 vectors on) and on
both sides of the lines between the narrow and the wide update (14,208 unknowns) and between the forms of the 3x3
product (14,208 nodes)."""
import numpy as np
import pytest

from cfdsfemmpi_b200 import meshgen
from test_gmres_kernels import _least_residuals

pytestmark = pytest.mark.gpu

CASES = [
    # mesh, pc, restart, iterations, time step (a long one from rest converges slowly, so that late vectors count)
    ("quad", 36, "pbjacobi", 320, 257, 10.0), ("quad", 36, "jacobi", 400, 300, 10.0), ("hex", 16, "jacobi", 200, 160, 0.1),
    ("quad", 66, "pbjacobi", 60, 50, 0.1), ("quad", 68, "jacobi", 60, 50, 0.1),
    ("quad", 118, "pbjacobi", 30, 20, 0.1), ("quad", 119, "pbjacobi", 30, 20, 0.1), ("quad", 119, "jacobi", 30, 20, 0.1),
]


@pytest.mark.parametrize("kind,n,pc,restart,its,dt", CASES, ids=["%s%d-%s-%d-%d" % c[:5] for c in CASES])
def test_residual_is_the_least_of_the_krylov_space(kind, n, pc, restart, its, dt):
    """The residual against the least one over the Krylov space, found with a twice orthogonalised basis.  Single
    Gram-Schmidt leaves the basis orthogonal to about u k^2, k its condition, which the reduction of the residual
    bounds: that much of the least residual, with a factor of 100 for the dimension, at least 1e-6 as in short cycles,
    and 1e-12 of the first residual for the rounding of evaluating it.  Repeats agree bitwise."""
    sp = pytest.importorskip("scipy.sparse")
    from cfdsfemmpi_b200 import Handle
    mesh = meshgen.cavity2d(n) if kind == "quad" else meshgen.cavity3d(n)
    h = Handle(mesh, meshgen.control_for(5, dt, 0.01), ksp="gmres", pc=pc, restart=restart, rtol=1e-30, max_it=its)
    rng = np.random.default_rng(11)
    h.set_element_state(*[(dt < 1.0) * rng.uniform(-1, 1, h.n) for _ in range(3)])
    vals, _ = h.assemble_export(0)
    p = h.export_pattern()
    nb, N = mesh.ndof, mesh.nNode
    A = sp.bsr_matrix((vals, p["colidx"], p["rowptr"]), shape=(h.n, h.n)).tocsr()
    diag = vals[[p["rowptr"][i] + int(np.searchsorted(p["colidx"][p["rowptr"][i]:p["rowptr"][i + 1]], i)) for i in range(N)]]
    if pc == "jacobi":
        d = 1.0 / np.einsum("nii->ni", diag).ravel()
        inv = lambda r: d * r
    else:
        D = np.linalg.inv(diag)
        inv = lambda r: np.einsum("nij,nj->ni", D, r.reshape(N, nb)).ravel()
    b = rng.uniform(-1, 1, h.n)
    x, got, _ = h.solve_export(b)
    assert got == its
    assert np.array_equal(h.solve_export(b)[0], x)
    r0 = np.linalg.norm(inv(b))
    least = _least_residuals(lambda v: inv(A @ v), inv(b), restart, its)
    res = np.linalg.norm(inv(b - A @ x))
    tol = 1e-6 + 100 * 2.0 ** -53 * (r0 / least) ** 2
    assert tol < 0.01                                           # the case says something
    assert abs(res - least) <= tol * least + 1e-12 * r0
    assert h.true_residual(x, b) == pytest.approx(np.linalg.norm(b - A @ x), rel=1e-9)
    h.close()
