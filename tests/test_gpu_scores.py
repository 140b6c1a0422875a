"""Region scores at the table sizes where their summation changes form (more than
1024 regions), with remainders of its chunks and vector loads, fine cells that
are not a power of two, in the two-kernel chain and in the tail launch.  The
scores steer every acceptance, so a plan equal to the CPU oracle's node for node
has them bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", ["0", "1"])
@pytest.mark.parametrize("model,coarse,fine", [("di", 10, 3), ("di", 11, 2), ("di", 13, 4), ("di", 16, 3), ("di", 33, 1), ("di", 64, 2),
                                               ("unicycle", 33, 5), ("unicycle", 67, 8), ("quad", 17, 4), ("dubins", 12, 4)])
def test_plan_matches_oracle(model, coarse, fine, tail, monkeypatch):
    from kgmt_gb300.planner import KGMT
    monkeypatch.setenv("KGMT_TAIL", tail)
    make = {"di": W.double_integrator_query, "quad": W.quadrotor_query, "dubins": W.dubins_query, "unicycle": W.unicycle_query}[model]
    q = make(seed=coarse, n_obstacles=20)
    q.config = q.config.replace(tree_capacity=12_000, max_iterations=25, coarse_len=coarse, fine_len=fine)
    ref = O.plan(q)
    p = KGMT(q.config)
    res = p.plan(q.init, q.goal, torch.from_numpy(np.ascontiguousarray(W.boxes_for_plan(q))).to("cuda:0"), len(q.obstacles))
    samples, parents, costs = p.copy_tree()
    for k in ("status", "iterations", "tree_size", "goal_index", "samples_drawn"):
        assert res[k] == ref[k], (k, res[k], ref[k])
    assert np.array_equal(parents, ref["parents"])
    assert np.array_equal(samples.view(np.uint32), ref["samples"].view(np.uint32))
    p.close()


@pytest.mark.parametrize("block", [128, 512])
def test_block_sizes(block):
    from kgmt_gb300.planner import BatchPlanner
    qs = W.double_integrator_batch(6, n_obstacles=20, seed=3, tree_capacity=12_000, coarse_len=19, max_iterations=20)
    b = BatchPlanner(len(qs), propagate_block=block)
    for r, ref in zip(b.plan([q.config for q in qs], *W.pack_queries(qs)), O.plan_batch(qs)):
        assert all(r[k] == ref[k] for k in ("status", "iterations", "tree_size", "goal_index", "samples_drawn"))
    b.close()
