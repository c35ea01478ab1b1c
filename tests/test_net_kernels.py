"""The guess network's kernels at the sizes where their tiles and chunks end: fewer nodes than a tile of 64 rows, one
stage of 32 rows per chunk of the weight gradient, several, a ragged last chunk, and neighbourhoods below, at and above
the eight places that the aggregation takes at once."""
import numpy as np
import pytest

import mpnn_ref
from cfdsfemmpi_b200 import io, meshgen

pytestmark = pytest.mark.gpu


def _tri(n):
    q = meshgen.cavity2d(n)
    conn = np.ascontiguousarray(np.concatenate([q.conn[:, s] for s in ([0, 1, 2], [0, 2, 3])]).astype(np.int32))
    return io.Mesh(ndim=2, npElem=3, coords=q.coords, conn=conn, dbc=q.dbc, output_nodes=q.output_nodes)


CASES = {
    "quad2": lambda: meshgen.cavity2d(2),        # 9 nodes
    "tri9": lambda: _tri(9),                     # 100 nodes, up to 7 neighbours
    "quad37": lambda: meshgen.cavity2d(37),      # 1,444 nodes: chunks of one stage
    "quad97": lambda: meshgen.cavity2d(97),      # 9,604 nodes: chunks of two stages, the last one ragged
    "hex13": lambda: meshgen.cavity3d(13),       # 2,744 nodes, 27 neighbours
}


@pytest.mark.parametrize("name", CASES)
def test_gradient_matches_cpu_reference(name):
    """Both sides round activations and gradients to bf16 (2^-9 relative) where they enter a product, about eight times
    along the longest path: 2e-2 of the largest entry of a block covers the values on which they round differently."""
    from cfdsfemmpi_b200 import Handle
    from cfdsfemmpi_b200._lib import Mpnn
    mesh = CASES[name]()
    h = Handle(mesh, meshgen.control_for(3, 0.05, 0.01), restart=2)
    net = Mpnn(h, seed=5)
    rng = np.random.default_rng(11)
    nd = mesh.ndof
    in_s = np.concatenate([np.full(nd, 0.1), np.full(nd, 0.02)]).astype(np.float32)
    out_s = np.full(nd, 0.02, np.float32)
    net.set_scales(in_s, out_s)
    us = [0.1 * rng.standard_normal(h.n) for _ in range(3)]
    net.add_sample(*us, cond=0.3)
    p = net.get_params()
    off, _ = mpnn_ref.layout()
    o = off["Wd"]
    p[o[0]:o[0] + o[1] * o[2]] = 0.2 * rng.standard_normal(o[1] * o[2]).astype(np.float32)
    net.set_params(p)
    loss, g = net.loss_grad(0)
    again = net.loss_grad(0)
    assert again[0] == loss and np.array_equal(again[1], g)
    d = h.export_pattern()
    free = d["dofmap"].reshape(-1, nd) >= 0
    mask = np.zeros((mesh.nNode, mpnn_ref.FOUT), np.float32)
    mask[:, :nd] = free
    loss_ref, g_ref = mpnn_ref.loss_and_grad(p, mpnn_ref.features(us[0], us[1], mesh.coords, nd, mesh.ndim, in_s, 0.3),
                                             mpnn_ref.targets(*us, nd, out_s), mask, d["rowptr"], d["colidx"],
                                             int(free.sum()))
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref)
    for key, ob in off.items():
        size = ob[1] * ob[2] if len(ob) == 3 else ob[1]
        a, b = g[ob[0]:ob[0] + size], g_ref[ob[0]:ob[0] + size]
        assert np.abs(a - b).max() <= 2e-2 * np.abs(b).max(), key
