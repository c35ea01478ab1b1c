"""Kernels that a batch launches in other forms than a handle alone (multi-dot with several vectors a CTA, packed update,
3x3 products by scalar rows, the control block by a copy) compute the same bits: sizes on both sides of each rule."""
import numpy as np
import pytest

from cfdsfemmpi_b200 import meshgen

pytestmark = pytest.mark.gpu

Q, H = meshgen.cavity2d, meshgen.cavity3d
CASES = {
    # 3x3: 1 CTA of the update, its narrow form alone but packed together, beyond the 16 groups (14,208 unknowns),
    # products alone by warps and together by rows; more than 148 vectors
    "quad_pbjacobi": ([Q(3), Q(30), Q(52), Q(66), Q(68), Q(75)], dict(pc="pbjacobi", restart=200, rtol=1e-8)),
    "quad_jacobi": ([Q(16), Q(36), Q(37), Q(60)], dict(pc="jacobi", restart=60, rtol=1e-4)),
    "quad_none": ([Q(9), Q(40), Q(64)], dict(pc="none", restart=40, rtol=1e-2)),
    "quad_ilu": ([Q(20), Q(70), Q(125)], dict(pc="bjacobi", restart=50)),
    "quad_bcgs": ([Q(20), Q(70), Q(125)], dict(pc="bjacobi", ksp="bcgs")),
    "quad_mixed": ([Q(20), Q(70), Q(90)], dict(pc="jacobi", precision="mixed", restart=50)),
    "hex": ([H(3), H(7), H(12), H(14), H(15)], dict(pc="jacobi", restart=100, rtol=1e-8)),
}


@pytest.mark.parametrize("name", CASES)
def test_batch_equals_single_runs_bitwise(name):
    from cfdsfemmpi_b200 import Batch, Handle
    meshes, kw = CASES[name]
    cases = [(m, meshgen.control_for(20, 0.05, 0.01)) for m in meshes]
    steps, ref = 2, []
    for mesh, ctrl in cases:
        h = Handle(mesh, ctrl, **kw)
        its = [h.step(0.05 * (k + 1), 0.05 * (k + 1)).as_dict()["ksp_its"] for k in range(steps)]
        ref.append((h.get_solution(), its))
        h.close()
    b = Batch(cases, **kw)
    for chunk, depth in ((4, 1), (3, 2)):
        b.set_schedule(len(cases), chunk, depth)
        for h in b.handles:
            h.set_solution(np.zeros(h.n))
            h.set_history(np.zeros(h.n), np.zeros(h.n))
        its = [[] for _ in cases]
        for k in range(steps):
            st, _ = b.step(np.full(len(cases), 0.05 * (k + 1)))
            for i, s in enumerate(st):
                its[i].append(s.as_dict()["ksp_its"])
        for i, (sol, n_its) in enumerate(ref):
            assert its[i] == n_its, (i, chunk)
            assert np.array_equal(b.handles[i].get_solution(), sol), (i, chunk)
        if chunk == 4 and name in ("quad_mixed",):
            break
    b.close()
