"""Rows of more than 65,535 blocks, which the end of a long strip gets from the complete factorisation when its nodes are
numbered last (test_trsv_plan._strip)."""
import numpy as np
import pytest

from cfdsfemmpi_b200 import meshgen
from cfdsfemmpi_b200._lib import ilu_pattern_build
from test_trsv_plan import _strip, test_solves_invert_the_exported_factors as check_solves

CASES = [(2, 33000), (3, 14600)]


@pytest.mark.parametrize("ndim,length", CASES)
def test_the_pattern_of_a_wide_row_is_built(ndim, length):
    mesh = _strip(ndim, length)
    f = ilu_pattern_build(mesh, -1, 2)
    widths = np.diff(f["rowptr"])
    assert widths.max() == mesh.nNode // 2 > 65535
    assert (widths > 100).sum() == (4 if ndim == 2 else 9)


@pytest.mark.gpu
@pytest.mark.parametrize("ndim,length", CASES)
def test_factors_of_wide_rows_multiply_to_the_matrix(ndim, length):
    """Row i of A - L U for the two diagonal blocks of A.  A block of it is a sum of at most w products of ndof terms
    each, taken off one at a time: at most (w ndof + 2) u of |L| |U|, u = 2^-53, w the largest number of pivots that
    change a block of the row, which is the number of rows with it in their upper part.  The multipliers use the stored
    inverse D of U_pp: (D U_pp - I) of |L_ip| |U_pp| on top, and the rounding of that product."""
    sp = pytest.importorskip("scipy.sparse")
    from cfdsfemmpi_b200 import Handle
    mesh = _strip(ndim, length)
    h = Handle(mesh, meshgen.control_for(5, 0.1, 0.01), ksp="preonly", pc="bjacobi", ilu_levels=-1, bjacobi_blocks=2)
    rng = np.random.default_rng(5)
    h.set_element_state(*[rng.uniform(-1, 1, h.n) for _ in range(3)])
    vals, _ = h.assemble_export(0)
    p, f = h.export_pattern(), h.ilu_factors()
    h.close()
    N, nb = mesh.nNode, mesh.ndof
    arow = np.repeat(np.arange(N), np.diff(p["rowptr"]))
    half = N // 2
    same = (arow < half) == (p["colidx"] < half)

    def bsr(v, cols, rows):
        ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=N))])
        return sp.bsr_matrix((v, cols, ptr), shape=(N * nb, N * nb)).tocsr()

    A = bsr(vals[same], p["colidx"][same], arow[same])
    rows = np.repeat(np.arange(N), np.diff(f["rowptr"]))
    low = f["colidx"] < rows
    L = bsr(f["vals"][low], f["colidx"][low], rows[low]) + sp.identity(N * nb, format="csr")
    U = bsr(f["vals"][~low], f["colidx"][~low], rows[~low])
    u = 2.0 ** -53
    w = int(np.bincount(f["colidx"][~low], minlength=N).max())
    D, Ud = f["dinv"], f["vals"][f["diag"]]
    off = np.abs(D @ Ud - np.eye(nb)) + 2 * (nb + 2) * u * (np.abs(D) @ np.abs(Ud))
    E = sp.block_diag(list(np.abs(Ud) @ off), format="csr")
    bound = 2 * (w * nb + 4) * u * (abs(L) @ abs(U)) + 2 * abs(L) @ E
    diff = abs(A - L @ U)
    assert (diff - bound).max() <= 1e-300


@pytest.mark.gpu
@pytest.mark.parametrize("ndim,length", CASES)
def test_solves_with_wide_rows_invert_the_factors(ndim, length):
    check_solves("wide", lambda: _strip(ndim, length), -1, 2)


@pytest.mark.gpu
def test_a_few_wide_rows_take_little_memory():
    """What the complete factorisation takes beyond ILU(0) of the same strip: for a block of the factors 128 bytes for its
    value, 12 for its indices, 72 for its list of at most nine updates and 12 for its part of the solves' records; nine
    places for rows of 65,700 blocks of 128 bytes; and 2 MB for the rounding of each of some 60 allocations.  (A place
    for each of 256 warps would be 2.2 GB.)"""
    torch = pytest.importorskip("torch")
    from cfdsfemmpi_b200 import Handle
    mesh = _strip(3, 14600)
    torch.zeros(1, device="cuda")
    used, nnz = [], []
    for levels in (0, -1):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        h = Handle(mesh, meshgen.control_for(5, 0.1, 0.01), ksp="preonly", pc="bjacobi", ilu_levels=levels, bjacobi_blocks=2)
        used.append(before - torch.cuda.mem_get_info()[0])
        nnz.append(h.ilu_factors(values=False)["colidx"].size)
        h.close()
    assert used[1] - used[0] <= 224 * (nnz[1] - nnz[0]) + 9 * 65700 * 128 + 60 * 2 ** 21
