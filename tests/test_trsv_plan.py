"""Host-only checks of the triangular solves' schedule (cfdgpu_trsv_plan_build).

The kernel's warps poll shared-memory slots until a value arrives, so it makes
progress and computes the right thing exactly if (1) every block of every row
is in one piece of one warp, with the slot of its column; (2) an input from
elsewhere belongs to a group handed out earlier; (3) the warps of a group,
each going through its pieces in order, can always finish.  Meshes: those on
which a rule of the builder changes sides (short strands, long rows, groups cut
to fit) and the ordinary ones.  No GPU is needed.
"""
import numpy as np
import pytest

from cfdsfemmpi_b200 import io, meshgen
from cfdsfemmpi_b200._lib import ilu_pattern_build, trsv_plan_build

FIRST, LAST, DIRECT = 1 << 16, 1 << 17, 1 << 20


def _renumbered(mesh, seed):
    rng = np.random.default_rng(seed)
    p = rng.permutation(mesh.nNode)
    coords = np.empty_like(mesh.coords)
    coords[p] = mesh.coords
    dbc = mesh.dbc.copy()
    dbc[:, 0] = p[mesh.dbc[:, 0].astype(int)]
    return io.Mesh(ndim=mesh.ndim, npElem=mesh.npElem, coords=coords, conn=p[mesh.conn].astype(np.int32), dbc=dbc,
                   output_nodes=mesh.output_nodes)


def _strip(ndim, length):
    """A strip (bar) of elements, width + 1 nodes across, in two halves.  Nodes of the second half are numbered
    from the strip's end on, except that the end itself comes last: by the fill-path theorem its rows of the complete
    factorisation of that half have every node of the half as an input."""
    base = meshgen.cavity2d(3) if ndim == 2 else meshgen.cavity3d(2)
    per = 4 if ndim == 2 else 9
    cross = base.coords[base.coords[:, -1] == 0.0][:, :-1]
    ends = [c for c in base.conn if set(c[:]) <= set(range(2 * per))]
    lay = [[(v // per, v % per) for v in c] for c in ends]         # (layer, node of the cross section)
    new = {}
    half = length // 2
    for layer in range(half):
        for v in range(per):
            new[layer, v] = len(new)
    for layer in list(range(length - 2, half - 1, -1)) + [length - 1]:
        for v in range(per):
            new[layer, v] = len(new)
    coords = np.zeros((per * length, ndim))
    for (layer, v), i in new.items():
        coords[i] = np.append(cross[v], 0.5 * layer)
    conn = np.array([[new[layer + dl, v] for dl, v in c] for layer in range(length - 1) for c in lay], np.int32)
    dbc = np.array([(new[0, v], dof, 0.0) for v in range(per) for dof in range(ndim)] + [(new[0, 0], ndim, 0.0)])
    return io.Mesh(ndim=ndim, npElem=conn.shape[1], coords=coords, conn=conn, dbc=dbc, output_nodes=np.zeros(0, np.int32))


CASES = [
    ("wide_quad4", lambda: _strip(2, 2104), -1, 2), ("wide_hex8", lambda: _strip(3, 580), -1, 2),
    ("quad4_1", lambda: meshgen.cavity2d(1), 0, 1), ("quad4_9", lambda: meshgen.cavity2d(9), 0, 1),
    ("quad4_9", lambda: meshgen.cavity2d(9), 3, 2), ("quad4_21_lu", lambda: meshgen.cavity2d(21), -1, 1),
    ("quad4_70_lu", lambda: meshgen.cavity2d(70), -1, 1), ("quad4_3x200", lambda: meshgen.cavity2d(200), 0, 1),
    ("hex8_1", lambda: meshgen.cavity3d(1), 0, 1), ("hex8_7", lambda: meshgen.cavity3d(7), 0, 1),
    ("hex8_9_ilu1", lambda: meshgen.cavity3d(9), 1, 1), ("hex8_8_blocks", lambda: meshgen.cavity3d(8), 1, 3),
    ("hex8_6_lu", lambda: meshgen.cavity3d(6), -1, 1),
    ("hex8_renumbered", lambda: _renumbered(meshgen.cavity3d(6), 3), 0, 1),
    ("quad4_renumbered", lambda: _renumbered(meshgen.cavity2d(40), 4), 1, 1),
    ("ogrid", lambda: meshgen.cylinder_ogrid(nt=48, nr=140), 3, 1),
]


@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("name,build,levels,blocks", CASES, ids=[f"{c[0]}-{c[2]}-{c[3]}" for c in CASES])
def test_plan_covers_every_block_and_can_always_go_on(name, build, levels, blocks, upper):
    mesh = build()
    f = ilu_pattern_build(mesh, levels, blocks)
    d = trsv_plan_build(mesh, levels, blocks, upper)
    info, n = d["info"], mesh.nNode
    rp, ci = f["rowptr"], f["colidx"]
    diag = np.array([rp[i] + int(np.searchsorted(ci[rp[i]:rp[i + 1]], i)) for i in range(n)])
    lo, hi = (diag + 1, rp[1:]) if upper else (rp[:-1], diag)
    solved = np.zeros(n, bool)
    seen_blocks, direct_rows, wide = 0, 0, []
    zero = int(d["groups"][:, [0, 2]].sum(1).max()) * mesh.ndof
    assert d["wptr"][0, 0] == 0 and d["wptr"][-1, -1] == info.npieces
    for g in range(info.ngroups):
        rows, e0, ne, _ = d["groups"][g]
        assert 0 < rows and rows + ne <= info.slots_max
        ext = d["ext"][e0:e0 + ne]
        assert np.all(solved[ext]) and len(set(ext.tolist())) == ne        # (2)
        wp = d["wptr"][g]
        if g:
            assert wp[0] == d["wptr"][g - 1, -1]
        holder = np.full(rows + ne, -1)
        holder[rows:] = ext
        lists = []
        for w in range(info.warps):
            out = []
            for t in range(wp[w], wp[w + 1]):
                q0, m, ds, at = d["pieces"][t]
                k = m & 0xffff
                assert 0 <= k <= info.cap and (m >> 18) & 3 == (q0 & 3)
                row, node, again, own = d["desc"][4 * ds:4 * ds + 4]
                assert again == m and node == f["perm"][row] and at == (row if upper else node)
                per = 4 if mesh.ndim == 3 else 8
                table = d["desc"][4 * ds + 4:4 * ds + 4 + 4 * per].reshape(per, 4).T.ravel()
                if m & DIRECT:     # a row with more inputs than slots: it names them by their place in the vector
                    cols = table[:k] // mesh.ndof
                    assert rows == 1 and ne == 0 and np.all(cols * mesh.ndof == table[:k]) and own == own & 0xffff | zero << 16
                    assert cols.tolist() == [f["perm"][c] if upper else c for c in ci[q0:q0 + k]]
                    wide += cols.tolist()
                    if m & LAST:
                        assert sorted(f["perm"][c] if upper else c for c in ci[lo[row]:hi[row]]) == sorted(wide)
                        holder[0] = row
                        seen_blocks += len(wide)
                        wide, direct_rows = [], direct_rows + 1
                    continue
                assert np.all(table % (8 * mesh.ndof) == 0) and (own & 0xffff) % mesh.ndof == 0
                offsets = np.append((own & 0xffff) // mesh.ndof, table // (8 * mesh.ndof))
                assert own >> 16 == (offsets[1 if upper else k] if k else offsets[-1]) * mesh.ndof
                assert np.all(offsets[1 + k:] == d["groups"][:, [0, 2]].sum(1).max())     # a slot that holds zero
                slots = offsets[:1 + k].tolist()
                assert slots[0] < rows
                if m & FIRST:
                    out.append([row, [], slots[0]])
                assert out[-1][0] == row and out[-1][2] == slots[0]
                out[-1][1] += list(zip(range(q0, q0 + k), slots[1:]))
                if m & LAST:
                    assert sorted(q for q, _ in out[-1][1]) == list(range(lo[row], hi[row]))      # (1)
                    holder[slots[0]] = row
            assert wp[w] == wp[w + 1] or d["pieces"][wp[w + 1] - 1][1] & LAST
            lists.append(out)
        assert np.all(holder >= 0) and len(set(holder.tolist())) == rows + ne
        own = holder[:rows]
        assert not solved[own].any()
        done = set(ext.tolist())
        left = [list(x) for x in lists]
        while any(left):                                                    # (3)
            moved = False
            for x in left:
                while x and all(holder[s] in done for _, s in x[0][1]):
                    row, bl, _ = x.pop(0)
                    assert [holder[s] for _, s in bl] == [ci[q] for q, _ in bl]
                    done.add(row)
                    seen_blocks += len(bl)
                    moved = True
            assert moved
        solved[own] = True
    assert (direct_rows > 0) == (name.startswith("wide") and not upper)
    assert solved.all() and seen_blocks == int((hi - lo).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("name,build,levels,blocks", CASES, ids=[f"{c[0]}-{c[2]}-{c[3]}" for c in CASES])
def test_solves_invert_the_exported_factors(name, build, levels, blocks):
    """The residual of z = (L U)^-1 r, row by row.  A solve's row is a sum of w products (any order) and one
    subtraction: its error is at most (w + 2) u times the magnitudes, u = 2^-53.  The upper solve multiplies the sum s
    by the stored inverse D of U_ii, which leaves (U_ii D - I) s on top of the rounding of that product, at most
    (ndof + 2) u |U_ii| |D| |s|.  The result does not depend on scheduling: repeats agree bitwise."""
    sp = pytest.importorskip("scipy.sparse")
    from cfdsfemmpi_b200 import Handle
    mesh = build()
    h = Handle(mesh, meshgen.control_for(5, 0.1, 0.01), pc="bjacobi", ilu_levels=levels, bjacobi_blocks=blocks)
    rng = np.random.default_rng(3)
    n, N, nb = h.n, mesh.nNode, mesh.ndof
    h.set_element_state(*[rng.uniform(-1, 1, n) for _ in range(3)])
    h.assemble_export(0, want_values=False)
    f = h.ilu_factors()
    perm = ilu_pattern_build(mesh, levels, blocks)["perm"]
    dof = (perm[:, None] * nb + np.arange(nb)).ravel()
    rows = np.repeat(np.arange(N), np.diff(f["rowptr"]))

    def part(keep, extra=0.0):
        ptr = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=N))])
        m = sp.bsr_matrix((f["vals"][keep], f["colidx"][keep], ptr), shape=(n, n)).tocsr()
        return m + sp.identity(n, format="csr") if extra else m

    L, U = part(f["colidx"] < rows, 1.0), part(f["colidx"] >= rows)
    r = rng.uniform(-1, 1, n)
    z = h.pc_apply(r)
    for _ in range(3):
        assert np.array_equal(h.pc_apply(r), z)
    zf, rf = z[dof], r[dof]
    y = U @ zf
    u = 2.0 ** -53
    w = int(max(np.diff(L.indptr).max(), np.diff(U.indptr).max()))
    D, Ui = f["dinv"], f["vals"][f["diag"]]
    off = np.abs(Ui @ D - np.eye(nb)) + 2 * (nb + 2) * u * (np.abs(Ui) @ np.abs(D))      # (and the rounding of this)
    s = np.abs(Ui) @ np.abs(zf).reshape(N, nb, 1)
    bound = 2 * (w + 4) * u * (abs(L) @ (abs(U) @ abs(zf) + abs(y))) + abs(L) @ (off @ s).ravel()
    assert np.all(np.abs(rf - L @ y) <= 2 * bound + 1e-300)
