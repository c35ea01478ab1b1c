"""Block-ILU handles of different sizes used from several host threads at once
compute bit for bit what each computes alone.  The kernels' shared memory depends
on the mesh, so the threads launch the same kernels with different sizes."""
import threading

import numpy as np
import pytest

from cfdsfemmpi_b200 import meshgen

pytestmark = pytest.mark.gpu

SIZES = [24, 64, 8, 96, 16, 40]
OPTS = {"bcgs_ilu0": dict(ksp="bcgs", pc="bjacobi", rtol=1e-10),
        "complete_lu": dict(ksp="preonly", pc="bjacobi", ilu_levels=-1),
        "mixed": dict(pc="bjacobi", precision="mixed")}


def _cases():
    return [(meshgen.cavity2d(n), meshgen.control_for(60, 0.05, 1.0 / re))
            for n, re in zip(SIZES, [100.0, 250.0, 1000.0, 100.0, 400.0, 150.0])]


@pytest.mark.parametrize("name,steps", [("bcgs_ilu0", 50), ("complete_lu", 50), ("mixed", 10)])
def test_batch_of_uneven_ilu_cavities_matches_single_runs(name, steps):
    from cfdsfemmpi_b200 import Batch, Handle
    cases, dt = _cases(), 0.05
    ref = []
    for mesh, ctrl in cases:
        h = Handle(mesh, ctrl, **OPTS[name])
        its = [h.step(dt * (k + 1), min(dt * (k + 1), 1.0)).as_dict()["ksp_its"] for k in range(steps)]
        ref.append((h.get_solution(), its))
        h.close()
    b = Batch(cases, **OPTS[name])
    b.set_schedule(len(cases), 4, 1)
    its = [[] for _ in cases]
    for k in range(steps):
        st, _ = b.step(np.full(len(cases), dt * (k + 1)))
        for i, s in enumerate(st):
            its[i].append(s.as_dict()["ksp_its"])
    sols = [h.get_solution() for h in b.handles]
    b.close()
    for i, (sol, n_its) in enumerate(ref):
        assert its[i] == n_its, i
        assert np.array_equal(sols[i], sol), i


def test_factor_and_solve_from_threads():
    """Factorisation and both solves again and again from a thread per handle."""
    from cfdsfemmpi_b200 import Handle
    hs, rs, zs = [], [], []
    for mesh, ctrl in _cases():
        h = Handle(mesh, ctrl, pc="bjacobi")
        rng = np.random.default_rng(len(hs))
        h.set_element_state(*[rng.uniform(-1, 1, h.n) for _ in range(3)])
        h.assemble_export(0, want_values=False)
        r = rng.uniform(-1, 1, h.n)
        hs.append(h)
        rs.append(r)
        zs.append(h.pc_apply(r))
    wrong = []

    def work(i):
        try:
            for k in range(300):
                if not np.array_equal(hs[i].pc_apply(rs[i]), zs[i]):
                    wrong.append((i, k, "differs"))
                    return
        except Exception as e:
            wrong.append((i, str(e)))

    t = [threading.Thread(target=work, args=(i,)) for i in range(len(hs))]
    for x in t:
        x.start()
    for x in t:
        x.join()
    for h in hs:
        h.close()
    assert not wrong
