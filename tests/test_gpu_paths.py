"""Path readout at the sizes where its way changes: paths of up to 128 rows go to
the host buffer with the plan, longer ones and those past the buffer are copied
on demand.  Against the CPU oracle's path, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W
from kgmt_gb300.config import double_integrator_single
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def straight_query(distance, seed=1):
    """A double integrator flying almost straight along x at 0.29: one step of
    0.0039 per node, so the path has about distance / 0.0039 rows."""
    cfg = double_integrator_single(seed).replace(tree_capacity=60_000, max_iterations=400, min_steps=1, max_steps=1, step_size=0.0134,
                                                 samples_per_node=1, u_min=(0.0,) * 4, u_max=(1e-4, 1e-4, 1e-4, 0.0), goal_radius=0.005,
                                                 epsilon=0.0, coarse_len=64, fine_len=4)
    init, goal = np.zeros(10, np.float32), np.zeros(10, np.float32)
    init[:4], goal[:3] = [0.05, 0.3, 0.3, 0.29], [0.05 + distance, 0.3, 0.3]
    return W.Query(cfg, init, goal, np.zeros((0, 6), np.float32))


@pytest.mark.parametrize("distance", [0.012, 0.2, 0.49, 0.494, 0.498, 0.502, 0.8])
def test_single_plan_path(distance):
    from kgmt_gb300.planner import KGMT
    q = straight_query(distance)
    ref = O.plan(q)
    assert ref["status"] == 1
    p = KGMT(q.config)
    for _ in range(2):  # the second plan's path replaces the first's
        r = p.plan(q.init, q.goal, None, 0)
        assert r["path_len"] == ref["path_len"]
        assert np.array_equal(p.h_controlPathToGoal_.view(np.uint32), ref["path"].view(np.uint32))
    short = np.zeros((3, 10), np.float32)  # fewer rows than the path has
    from kgmt_gb300._abi import C, check, load
    n = C.c_uint32()
    check(load().kgmt_copy_path(p._h, short.ctypes.data, 3, C.byref(n)))
    assert n.value == min(3, ref["path_len"]) and np.array_equal(short[:n.value], ref["path"][:n.value])
    p.close()


def test_batch_paths_past_the_buffer():
    """Twelve queries of 100 to 206 rows: more than the host buffer holds, some
    longer than a path that goes there, one without a path."""
    from kgmt_gb300.planner import BatchPlanner
    qs = [straight_query(d, seed=i + 1) for i, d in enumerate([0.4, 0.4, 0.8, 0.4, 0.5, 0.45, 0.4, 0.4, 0.42, 0.4, 0.4, 0.4])]
    qs[4].config = qs[4].config.replace(max_iterations=5)
    refs = O.plan_batch(qs)
    b = BatchPlanner(len(qs))
    args = W.pack_queries(qs)
    for _ in range(2):
        res = b.plan([q.config for q in qs], *args)
        for i in reversed(range(len(qs))):
            assert res[i]["path_len"] == refs[i]["path_len"]
            assert np.array_equal(b.copy_path(i).view(np.uint32), O.plan(qs[i])["path"].view(np.uint32)), i
    b.close()
