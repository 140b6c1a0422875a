"""Samples that take a caller-sized time: up to 10,000 steps against every box of a
scene whose culling grid is refused (a box with a NaN face, which touches nothing).
Most samples leave the speed limits within a few hundred steps and a few stay to
the end, so the other warps of a block, and other blocks, wait for one run of a
second and more.  The same plan in the same scene without that box, which has a
grid and no long run, must come out node for node."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def query(n_boxes, capacity, iterations, spn=1024, seed=3):
    q = W.double_integrator_query(seed=seed, n_obstacles=1)
    q.config = q.config.replace(tree_capacity=capacity, samples_per_node=spn, max_iterations=iterations, min_steps=1, max_steps=10_000,
                                step_size=1e-5, v_min=-2e-4, v_max=2e-4, u_min=(-1.0, 0.0, 0.0, 0.0), u_max=(1.0, 0.0, 0.0, 0.0),
                                goal_radius=1e-3)
    rng = np.random.default_rng(seed)
    lo = rng.uniform(0.2, 0.9, (n_boxes, 3))
    q.obstacles = np.concatenate([lo, lo + 0.01], 1).astype(np.float32)
    refused = np.concatenate([q.obstacles, np.float32([[np.nan, 50, 50, 51, 51, 51]])])
    return q, np.ascontiguousarray(refused)


def plan(q, boxes):
    from kgmt_gb300.planner import KGMT
    p = KGMT(q.config)
    res = p.plan(q.init, q.goal, torch.from_numpy(boxes).to("cuda:0"), len(boxes))
    tree = p.copy_tree()
    p.close()
    return {k: res[k] for k in ("status", "iterations", "tree_size", "goal_index", "samples_drawn")}, tree


def same(a, b):
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


def test_tiles_wait_for_a_long_run(monkeypatch):
    """About 150,000 samples in the third iteration: more tiles than resident
    blocks, so warps that are through with two tiles wait for the last one in
    the first."""
    monkeypatch.setenv("KGMT_TAIL", "0")
    q, refused = query(3000, 150_000, 3)
    got = plan(q, refused)
    assert got[0]["samples_drawn"] > 200_000
    same(got, plan(q, q.obstacles))


@pytest.mark.parametrize("n", [1, 6])
def test_blocks_meet_after_a_long_run(n):
    """The blocks of the tail launch wait for the one that has the longest run,
    some seconds."""
    from kgmt_gb300.planner import BatchPlanner
    qs = [query(20_000, 20_000, 1, spn=max(64, 1024 // n), seed=5 + i) for i in range(n)]
    out = []
    for k in (0, 1):
        b = BatchPlanner(n)
        for q, refused in qs:
            q.boxes = refused if k else q.obstacles
        off = np.cumsum([0] + [len(q.boxes) for q, _ in qs])
        inits, goals, _, _, _ = W.pack_queries([q for q, _ in qs])
        res = b.plan([q.config for q, _ in qs], inits, goals, np.concatenate([q.boxes for q, _ in qs]), off[:-1], np.diff(off))
        assert b.stats()["iterations_tail"] == 1
        out.append([({x: r[x] for x in ("status", "iterations", "tree_size", "goal_index", "samples_drawn")},
                     tuple(a[: r["tree_size"]] for a in b.copy_tree(i))) for i, r in enumerate(res)])
        b.close()
    for a, r in zip(*out):
        same(a, r)
