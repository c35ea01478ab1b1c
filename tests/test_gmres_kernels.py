"""The kernels of the restarted GMRES at the sizes where their forms change: the multi-dot has one CTA per vector up to
2048 16-byte chunks and tiles beyond, the update is narrow up to 18,944 chunks and wide beyond, the solution update
changes at 16 vectors, the back substitution works on 32 columns at a time, and 2D meshes use the 3x3 product."""
import numpy as np
import pytest

from cfdsfemmpi_b200 import meshgen

pytestmark = pytest.mark.gpu

CASES = [
    # mesh, pc, restart, iterations
    ("quad", 2, "jacobi", 50, 3), ("quad", 9, "pbjacobi", 50, 1), ("quad", 10, "jacobi", 50, 16),
    ("quad", 10, "pbjacobi", 50, 17), ("quad", 35, "pbjacobi", 100, 64), ("quad", 36, "jacobi", 100, 65),
    ("quad", 36, "pbjacobi", 20, 49), ("quad", 111, "pbjacobi", 40, 33), ("quad", 112, "pbjacobi", 40, 32),
    ("hex", 5, "pbjacobi", 50, 31), ("hex", 20, "jacobi", 50, 34),
    ("hex", 21, "pbjacobi", 50, 35),
]


def _least_residuals(op, r0, restart, its):
    """Norm of the residual after `its` steps of GMRES(restart) with a twice orthogonalised basis."""
    r, done = r0, 0
    while done < its:
        k = min(restart, its - done)
        Q, AQ = [r / np.linalg.norm(r)], []
        for _ in range(k):
            w = op(Q[-1])
            AQ.append(w.copy())
            for _ in range(2):
                for q in Q:
                    w -= (q @ w) * q
            Q.append(w / np.linalg.norm(w))
        AQ = np.array(AQ).T
        r = r - AQ @ np.linalg.lstsq(AQ, r, rcond=None)[0]
        done += k
    return np.linalg.norm(r)


@pytest.mark.parametrize("kind,n,pc,restart,its", CASES, ids=["%s%d-%s-%d-%d" % c for c in CASES])
def test_residual_is_the_least_of_the_krylov_space(kind, n, pc, restart, its):
    """GMRES's residual is the least one over the Krylov space, so that it is known without GMRES's own arithmetic.
    Single Gram-Schmidt leaves the basis orthogonal to u k^2, k its condition, at most the reduction of the residual:
    below 1e5 in these few steps, so the least residual is met to 1e-6 of itself (and 1e-12 of the first one, the
    rounding of evaluating it); a missing or doubled term in any sum shows as far more.  Repeats agree bitwise."""
    sp = pytest.importorskip("scipy.sparse")
    from cfdsfemmpi_b200 import Handle
    mesh = meshgen.cavity2d(n) if kind == "quad" else meshgen.cavity3d(n)
    h = Handle(mesh, meshgen.control_for(5, 0.1, 0.01), ksp="gmres", pc=pc, restart=restart, rtol=1e-30, max_it=its)
    rng = np.random.default_rng(7)
    h.set_element_state(*[rng.uniform(-1, 1, h.n) for _ in range(3)])
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
    r0 = inv(b)
    least = _least_residuals(lambda v: inv(A @ v), r0, restart, its)
    res = np.linalg.norm(inv(b - A @ x))
    assert abs(res - least) <= 1e-6 * least + 1e-12 * np.linalg.norm(r0)
    assert h.true_residual(x, b) == pytest.approx(np.linalg.norm(b - A @ x), rel=1e-9)
