"""The guess network's weight gradients over chunks of several stages of 32 rows (the fetch of the next stage during the
sums, a short last chunk): targets far from what the network gives on the nodes of one stage only, so that most of the
gradient is gone if that stage is."""
import numpy as np
import pytest

import mpnn_ref
from cfdsfemmpi_b200 import meshgen

pytestmark = pytest.mark.gpu

N_SIDE, STAGE = 170, 32
WIDE, SMALL = 3 * 148 * STAGE, 4 * 148 * STAGE          # rows of one stage for every chunk of the wide and the small layers


def _rows_per_chunk(n_pad, most):
    return -(-n_pad // most) * STAGE


@pytest.mark.parametrize("where", ["second", "third", "last"])
def test_gradient_of_one_stage_matches_cpu_reference(where):
    """Tolerance as for whole gradients: bf16 rounds about eight times along the longest path, 2^-9 each, and both sides
    round in the same places; 2e-2 of the largest entry of a block."""
    from cfdsfemmpi_b200 import Handle
    from cfdsfemmpi_b200._lib import Mpnn
    mesh = meshgen.cavity2d(N_SIDE)
    n_pad = -(-mesh.nNode // 64) * 64
    wide, small = _rows_per_chunk(n_pad, WIDE), _rows_per_chunk(n_pad, SMALL)
    assert wide == 96 and small == 64 and n_pad % wide == 64    # three stages, two, and two in the last wide chunk
    first = {"second": 100 * wide + STAGE, "third": 100 * wide + 2 * STAGE, "last": n_pad - 64}[where]
    h = Handle(mesh, meshgen.control_for(3, 0.05, 0.01), restart=2)
    net = Mpnn(h, seed=5)
    rng = np.random.default_rng(11)
    nd = mesh.ndof
    in_s = np.concatenate([np.full(nd, 0.1), np.full(nd, 0.02)]).astype(np.float32)
    out_s = np.full(nd, 0.02, np.float32)
    net.set_scales(in_s, out_s)
    us = [0.1 * rng.standard_normal(h.n) for _ in range(2)]
    us.append(2 * us[1] - us[0])                                # targets of zero but for the stage's
    us[2].reshape(-1, nd)[first:first + STAGE] += 2000.0 * rng.standard_normal((min(STAGE, mesh.nNode - first), nd))
    net.add_sample(*us, cond=0.3)
    p = net.get_params()
    off, _ = mpnn_ref.layout()
    o = off["Wd"]
    p[o[0]:o[0] + o[1] * o[2]] = 0.2 * rng.standard_normal(o[1] * o[2]).astype(np.float32)
    net.set_params(p)
    loss, g = net.loss_grad(0)
    d = h.export_pattern()
    free = d["dofmap"].reshape(-1, nd) >= 0
    mask = np.zeros((mesh.nNode, mpnn_ref.FOUT), np.float32)
    mask[:, :nd] = free
    loss_ref, g_ref = mpnn_ref.loss_and_grad(p, mpnn_ref.features(us[0], us[1], mesh.coords, nd, mesh.ndim, in_s, 0.3),
                                             mpnn_ref.targets(*us, nd, out_s), mask, d["rowptr"], d["colidx"],
                                             int(free.sum()))
    net.close()
    h.close()
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref)
    for key, ob in off.items():
        size = ob[1] * ob[2] if len(ob) == 3 else ob[1]
        a, b = g[ob[0]:ob[0] + size], g_ref[ob[0]:ob[0] + size]
        assert np.abs(a - b).max() <= 2e-2 * np.abs(b).max(), key
