"""Admission of plans and batches at the box counts where the grid's build divides
its lanes otherwise (64, 128), where a batch stops ordering the lists (256), and
where a plan's boxes are staged apart (1024).  A plan in a scene whose grid is
wrong differs from the CPU oracle's, which tests every box."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ("status", "iterations", "tree_size", "goal_index", "samples_drawn")


def query(model, n, seed):
    q = {"di": W.double_integrator_query, "unicycle": W.unicycle_query}[model](seed=seed, n_obstacles=1)
    rng = np.random.default_rng(seed)
    lo = rng.uniform(0.12, 0.9, (n, 3))
    edge = min(0.15, (0.05 / n) ** (1.0 / q.config.ws_dims))
    q.obstacles = np.concatenate([lo, lo + rng.uniform(0.5 * edge, 1.5 * edge, (n, 3))], 1).astype(np.float32)
    q.config = q.config.replace(tree_capacity=8_000, max_iterations=10)
    return q


@pytest.mark.parametrize("model", ["di", "unicycle"])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 256, 257, 1024, 1025, 5000])
def test_box_counts(model, n):
    from kgmt_gb300.planner import KGMT, BatchPlanner
    qs = [query(model, n, 40 + i) for i in range(2)]
    refs = [O.plan(q) for q in qs]
    p = KGMT(qs[0].config)
    res = p.plan(qs[0].init, qs[0].goal, torch.from_numpy(np.ascontiguousarray(W.boxes_for_plan(qs[0]))).to("cuda:0"), n)
    assert [res[k] for k in KEYS] == [refs[0][k] for k in KEYS]
    samples, parents, _ = p.copy_tree()
    assert np.array_equal(parents, refs[0]["parents"]) and np.array_equal(samples.view(np.uint32), refs[0]["samples"].view(np.uint32))
    p.close()
    b = BatchPlanner(2)
    for i, (r, ref) in enumerate(zip(b.plan([q.config for q in qs], *W.pack_queries(qs)), refs)):
        assert [r[k] for k in KEYS] == [ref[k] for k in KEYS]
        assert np.array_equal(b.copy_tree(i)[1][: r["tree_size"]], ref["parents"])
    b.close()
