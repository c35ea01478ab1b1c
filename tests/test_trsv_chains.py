"""Triangular solves by chains of rows: which orders of the nodes take that schedule, and the kernel against the exported
factors at chains of one row, of several and of the longest, rows within and beyond the blocks that a lane holds, and
fewer and more chains than the grid has warps; and the FP32 solves of both schedules, which no other test compares."""
import numpy as np
import pytest

from cfdsfemmpi_b200 import io, meshgen
from cfdsfemmpi_b200._lib import trsv_by_chains
from test_trsv_plan import test_solves_invert_the_exported_factors as check_solves


def _in_order(mesh, order):
    p = np.empty(mesh.nNode, int)
    p[order] = np.arange(mesh.nNode)
    coords = np.empty_like(mesh.coords)
    coords[p] = mesh.coords
    dbc = mesh.dbc.copy()
    dbc[:, 0] = p[mesh.dbc[:, 0].astype(int)]
    return io.Mesh(ndim=mesh.ndim, npElem=mesh.npElem, coords=coords, conn=p[mesh.conn].astype(np.int32), dbc=dbc,
                   output_nodes=mesh.output_nodes)


def _runs(mesh, k):
    """Runs of k consecutive nodes in random order."""
    n = mesh.nNode
    o = np.random.default_rng(k).permutation(-(-n // k))
    return _in_order(mesh, np.concatenate([np.arange(b * k, min(n, b * k + k)) for b in o]))


Q, H = meshgen.cavity2d, meshgen.cavity3d


@pytest.mark.parametrize("build,levels,by_chains", [
    (lambda: Q(64), 0, False), (lambda: Q(64), -1, False), (lambda: H(24), 2, False), (lambda: H(48), 2, True),
    (lambda: _runs(Q(64), 1), 0, True), (lambda: _runs(Q(8), 1), 0, False), (lambda: _runs(H(16), 1), 0, True),
    (lambda: _runs(H(4), 1), 0, False), (lambda: _runs(H(12), 1), 1, True), (lambda: _runs(Q(200), 12), 0, True), (lambda: _runs(Q(200), 32), 0, False),
    (lambda: _runs(H(30), 32), 1, False), (lambda: meshgen.cylinder_ogrid(), 3, False)])
def test_which_orders_go_by_chains(build, levels, by_chains):
    mesh = build()
    assert [trsv_by_chains(mesh, levels, 1, u) for u in (False, True)] == [by_chains] * 2


CASES = [("quad70_random", lambda: _runs(Q(70), 1), 0, 1), ("quad70_random", lambda: _runs(Q(70), 1), 3, 1),
         ("quad40_blocks", lambda: _runs(Q(40), 1), 1, 5), ("quad260_random", lambda: _runs(Q(260), 1), 0, 1),
         ("quad200_runs12", lambda: _runs(Q(200), 12), 0, 1), ("quad90_runs5", lambda: _runs(Q(90), 5), 2, 1),
         ("hex12_random", lambda: _runs(H(12), 1), 0, 1), ("hex16_random", lambda: _runs(H(16), 1), 1, 1),
         ("hex20_runs3", lambda: _runs(H(20), 3), 0, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("name,build,levels,blocks", CASES, ids=[f"{c[0]}-{c[2]}-{c[3]}" for c in CASES])
def test_chain_solves_invert_the_exported_factors(name, build, levels, blocks):
    """The bound of the solves by groups: it holds for a row's sum in any order."""
    mesh = build()
    assert trsv_by_chains(mesh, levels, blocks) and trsv_by_chains(mesh, levels, blocks, True)
    check_solves(name, lambda: mesh, levels, blocks)


FP32 = [c for c in CASES if c[0] != "quad260_random"] + [
    ("quad33", lambda: Q(33), 0, 1), ("quad64_lu", lambda: Q(64), -1, 1), ("hex7", lambda: H(7), 0, 1),
    ("hex9", lambda: H(9), 1, 1), ("hex8_lu", lambda: H(8), -1, 1), ("hex6_blocks", lambda: H(6), 2, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("name,build,levels,blocks", FP32, ids=[f"{c[0]}-{c[2]}-{c[3]}" for c in FP32])
def test_fp32_solves_invert_their_factors(name, build, levels, blocks):
    """The FP32 solves of mixed precision, by chains and by groups, rows of one piece and of several.  Products and sums
    are FP64 and each result is rounded once, v = 2^-24: y_i = (r_i - sum)(1 + v) leaves at most v |y| of r - L y, and
    z_i = D s (1 + v) leaves |U_ii D - I| |s| + v |U_ii| |z_i| of y - U z with |s| <= |U_ii| |z_i| but for terms of
    higher order (the factor 2, which also covers the FP64 roundings)."""
    sp = pytest.importorskip("scipy.sparse")
    from cfdsfemmpi_b200 import Handle
    from cfdsfemmpi_b200._lib import ilu_pattern_build
    mesh = build()
    h = Handle(mesh, meshgen.control_for(5, 0.1, 0.01), pc="bjacobi", precision="mixed", ilu_levels=levels,
               bjacobi_blocks=blocks)
    rng = np.random.default_rng(3)
    n, N, nb = h.n, mesh.nNode, mesh.ndof
    h.set_element_state(*[rng.uniform(-1, 1, n) for _ in range(3)])
    h.assemble_export(0, want_values=False)
    f = h.ilu_factors(values=False)
    perm = ilu_pattern_build(mesh, levels, blocks)["perm"]
    dof = (perm[:, None] * nb + np.arange(nb)).ravel()
    rows = np.repeat(np.arange(N), np.diff(f["rowptr"]))
    r = rng.uniform(-1, 1, n).astype(np.float32)
    z, vals, D = h.ilu32_apply(r)
    for _ in range(3):
        assert np.array_equal(h.ilu32_apply(r)[0], z)
    h.close()
    vals, D = vals.astype(float), D.astype(float)

    def part(keep):
        ptr = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=N))])
        return sp.bsr_matrix((vals[keep], f["colidx"][keep], ptr), shape=(n, n)).tocsr()

    L, U = part(f["colidx"] < rows) + sp.identity(n, format="csr"), part(f["colidx"] >= rows)
    zf, rf = z[dof].astype(float), r[dof].astype(float)
    y, v = U @ zf, 2.0 ** -24
    Ui = vals[f["diag"]]
    Uz = (np.abs(Ui) @ np.abs(zf).reshape(N, nb, 1))
    off = ((np.abs(Ui @ D - np.eye(nb)) @ Uz) + v * Uz).ravel()
    bound = v * (np.abs(y) + off) + abs(L) @ off
    assert np.all(np.abs(rf - L @ y) <= 2 * bound + 1e-40)
