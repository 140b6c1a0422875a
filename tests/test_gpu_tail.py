"""The persistent tail launch with one to as many running queries as it takes,
and one more (which stays in the two-kernel chain until a query ends): how the
queries divide the blocks depends on their number, samples and trees.  Against
the CPU oracle, and tree for tree against the chain alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEYS = ("status", "iterations", "tree_size", "goal_index", "path_len", "samples_drawn")


def plan(qs):
    from kgmt_gb300.planner import BatchPlanner
    b = BatchPlanner(len(qs))
    res = b.plan([q.config for q in qs], *W.pack_queries(qs))
    return b, res


def check(qs, monkeypatch, refs=None):
    b, res = plan(qs)
    st = b.stats()
    monkeypatch.setenv("KGMT_TAIL", "0")
    b0, res0 = plan(qs)
    st0 = b0.stats()
    monkeypatch.delenv("KGMT_TAIL")
    assert st["iterations_tail"] > 0 and st0["iterations_tail"] == 0
    assert st["samples"] == st0["samples"] and st["steps_executed"] == st0["steps_executed"]
    for i, (r, r0, ref) in enumerate(zip(res, res0, refs or O.plan_batch(qs))):
        for k in KEYS:
            assert r[k] == r0[k] == ref[k], (i, k, r[k], r0[k], ref[k])
        n = r["tree_size"]
        for a, a0 in zip(b.copy_tree(i), b0.copy_tree(i)):
            assert np.array_equal(a[:n].view(np.uint32), a0[:n].view(np.uint32)), i
        assert np.array_equal(b.copy_path(i).view(np.uint32), b0.copy_path(i).view(np.uint32)), i
    b.close()
    b0.close()


@pytest.mark.parametrize("n", [1, 2, 3, 8, 31, 32, 33])
def test_number_of_queries(n, monkeypatch):
    """Goals out of reach: the queries run on together for most iterations (of
    33 one ends early, and the launch takes the others)."""
    qs = W.double_integrator_batch(n, n_obstacles=30, seed=n, tree_capacity=9_000, max_iterations=30, goal_radius=0.01)
    if n == 33:
        qs[7].config = qs[7].config.replace(max_iterations=5)
    check(qs, monkeypatch)


def test_uneven_queries(monkeypatch):
    """All models, trees of 60 to 60,000 nodes, region tables of one to 35,937
    regions, some queries ending early: shares of very different sizes."""
    qs = W.all_models_batch(20, seed=9, tree_capacity=8_000)
    for i, q in enumerate(qs):
        cap = (60, 700, 8_000, 60_000)[(i // 4) % 4]
        coarse = 1 if i % 5 == 0 else (33 if i % 7 == 0 else 12)
        q.config = q.config.replace(tree_capacity=cap, max_iterations=12 + 3 * (i % 6), coarse_len=coarse, fine_len=2)
    check(qs, monkeypatch)


@pytest.mark.parametrize("spn", [1, 64])
def test_iterations_around_the_largest_taken(spn, monkeypatch):
    """A single plan whose iterations outgrow the launch and shrink again."""
    q = W.double_integrator_query(seed=3)
    q.config = q.config.replace(tree_capacity=60_000, samples_per_node=spn, max_iterations=40, goal_radius=0.004)
    check([q], monkeypatch)
