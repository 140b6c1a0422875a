"""The propagate tiles, of which each block keeps two: iterations of less than a
warp to many tiles a block, each block size, boxes around what a launch stages
(64 and 512) and grid items beyond it, one model and all in a launch.  Only the
chain of launches runs; against the CPU oracle, tree for tree."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(qs, monkeypatch, block=256):
    from kgmt_gb300.planner import BatchPlanner
    monkeypatch.setenv("KGMT_TAIL", "0")
    b = BatchPlanner(len(qs), propagate_block=block)
    res = b.plan([q.config for q in qs], *W.pack_queries(qs))
    for i, (q, r) in enumerate(zip(qs, res)):
        ref = O.plan(q)
        for k in ("status", "iterations", "tree_size", "goal_index", "path_len", "samples_drawn"):
            assert r[k] == ref[k], (i, k, r[k], ref[k])
        n = r["tree_size"]
        samples, parents, _ = b.copy_tree(i)
        assert np.array_equal(parents[:n], ref["parents"][:n]), i
        assert np.array_equal(samples[:n].view(np.uint32), ref["samples"][:n].view(np.uint32)), i
    b.close()


@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("n,cap,spn", [(1, 40, 1), (1, 90_000, 8), (3, 700, 33), (40, 6_000, 16)])
def test_iteration_sizes(n, cap, spn, block, monkeypatch):
    qs = W.double_integrator_batch(n, n_obstacles=30, seed=n + spn, tree_capacity=cap, samples_per_node=spn, max_iterations=14, goal_radius=0.01)
    check(qs, monkeypatch, block)


@pytest.mark.parametrize("boxes", [0, 1, 64, 65, 512, 513])
def test_staged_boxes(boxes, monkeypatch):
    """Boxes of up to two cells an axis and more: the lists of 64 and of 512 are
    longer than what is staged of them."""
    qs = W.double_integrator_batch(5, n_obstacles=boxes, seed=boxes, tree_capacity=5_000, max_iterations=12)
    for q in qs[1:3]:
        q.obstacles = q.obstacles[: boxes // 2]  # several numbers of boxes in a launch
    check(qs, monkeypatch)


@pytest.mark.parametrize("block", [128, 512])
def test_all_models(block, monkeypatch):
    qs = W.all_models_batch(9, seed=4, tree_capacity=7_000)
    for i, q in enumerate(qs):
        q.config = q.config.replace(max_iterations=8 + 2 * i)
    check(qs, monkeypatch, block)


@pytest.mark.parametrize("n", [2, 32, 33, 256, 257, 300])
def test_order_of_models(n, monkeypatch):
    """Tiles are taken model by model: slots around a warp's and a block's number
    of them, queries ending at different iterations."""
    qs = W.all_models_batch(n, seed=n, tree_capacity=500)
    for i, q in enumerate(qs):
        q.config = q.config.replace(tree_capacity=300 + 40 * (i % 9), max_iterations=3 + i % 4, coarse_len=4, fine_len=2)
    check(qs, monkeypatch)


@pytest.mark.parametrize("boxes", [33, 64, 65, 200, 256])
def test_box_tests_repeat(boxes):
    """The boxes of a grid cell are listed in order, so the tests made before a
    first hit, and their sum, are the same for every planner of a scene."""
    from kgmt_gb300.planner import BatchPlanner
    qs = W.double_integrator_batch(3, n_obstacles=boxes, seed=7, tree_capacity=6_000, max_iterations=25)
    counts = set()
    for _ in range(6):
        b = BatchPlanner(len(qs))
        b.plan([q.config for q in qs], *W.pack_queries(qs))
        st = b.stats()
        counts.add((st["samples"], st["steps_executed"], st["obstacle_tests"]))
        b.close()
    assert len(counts) == 1, counts


@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("most", [128, 129, 512, 700])
def test_boxes_staged_and_not_in_one_launch(block, most, monkeypatch):
    """Queries whose boxes a launch stages beside some whose boxes it leaves in
    global memory: above 512, and in blocks of 128 above 64 once any has over 128."""
    qs = W.double_integrator_batch(6, n_obstacles=most, seed=most, tree_capacity=4_000, max_iterations=10)
    for q, n in zip(qs, (0, 10, 64, 65, most // 2, most)):
        q.obstacles = q.obstacles[:n]
    check(qs, monkeypatch, block)
