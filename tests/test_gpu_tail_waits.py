"""The waits of the tail launch: one that runs out ends the plan with
KGMT_ERR_TIMEOUT and nothing goes on from the half-done iteration; the context
and other planners are not affected.  The limit is lowered from the host
(KGMT_FAULT_TAIL_POLLS); nothing here traps, faults or hangs the GPU."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

GIVES_UP = r'''
import numpy as np, torch
from kgmt_gb300 import _abi, workloads as W
from kgmt_gb300.planner import KGMT, BatchPlanner
from oracle import oracle as O
def code(f):
    try:
        f()
        return 0
    except _abi.KgmtError as e:
        assert "gave up" in str(e), e
        return e.code
q = W.double_integrator_query(seed=7)
d_obs = torch.from_numpy(np.ascontiguousarray(q.obstacles)).to("cuda:0")
p = KGMT(q.config)
print("plan", code(lambda: p.plan(q.init, q.goal, d_obs, len(q.obstacles))))
for n in (5, 33):
    # (of 33 one ends early, and the launch takes the others: as in test_gpu_tail.py)
    qs = W.double_integrator_batch(n, n_obstacles=30, seed=n, tree_capacity=9_000, max_iterations=30, goal_radius=0.01)
    if n == 33:
        qs[7].config = qs[7].config.replace(max_iterations=5)
    b = BatchPlanner(n)
    print("batch", code(lambda: b.plan([x.config for x in qs], *W.pack_queries(qs))))
from kgmt_gb300.planner import Server  # runs no tail launch
qs = W.double_integrator_batch(3, n_obstacles=10, seed=3, tree_capacity=6_000)
s = Server(max_slots=3, memory_budget=1 << 28)
at = {s.submit(x.config, x.init, x.goal, x.obstacles): i for i, x in enumerate(qs)}
got = {}
for _ in range(1000):
    s.step()
    got.update({at[r["ticket"]]: r for r in s.poll()})
    if len(got) == 3:
        break
print("served", all(got[i][k] == ref[k] for i, ref in enumerate(O.plan_batch(qs)) for k in ("status", "iterations", "tree_size", "goal_index")))
'''


def test_a_launch_that_gives_up_ends_the_plan():
    env = dict(os.environ, KGMT_FAULT_TAIL_POLLS="1", PYTHONPATH=str(ROOT))
    r = subprocess.run([sys.executable, "-c", GIVES_UP], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    assert r.stdout.split("\n")[:4] == ["plan 4", "batch 4", "batch 4", "served True"], r.stdout
