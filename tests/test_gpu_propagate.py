"""Function-level propagation (propagate_samples) at the sizes where its forms
change: one sample a thread or sorted shares, boxes tested one by one or through
the culling grid, remainders of a warp and of a block.  Against the CPU oracle,
which does the same operations in the same order: bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from kgmt_gb300 import workloads as W
from kgmt_gb300.config import MODEL_DUBINS_AIRPLANE, MODEL_QUADROTOR, MODEL_UNICYCLE
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MAKE = {"di": W.double_integrator_query, "quad": W.quadrotor_query, "dubins": W.dubins_query, "unicycle": W.unicycle_query}


@pytest.fixture(scope="module", autouse=True)
def _need_cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def inputs(cfg, n, seed):
    rng = np.random.default_rng(seed)
    x0 = np.zeros((n, cfg.sample_dim), np.float32)
    x0[:, :3] = rng.uniform(0.0, 1.0, (n, 3))
    if cfg.model == MODEL_UNICYCLE:
        x0[:, 2], x0[:, 3] = rng.uniform(-np.pi, np.pi, n), rng.uniform(0.0, 0.3, n)
    elif cfg.model == MODEL_DUBINS_AIRPLANE:
        x0[:, 3], x0[:, 4], x0[:, 5] = rng.uniform(-np.pi, np.pi, n), rng.uniform(-1.0, 1.0, n), rng.uniform(0.0, 0.3, n)
    elif cfg.model == MODEL_QUADROTOR:
        x0[:, 3:6], x0[:, 6:9], x0[:, 9:12] = (rng.uniform(-a, a, (n, 3)) for a in (0.6, 0.25, 1.5))
    else:
        x0[:, 3:6] = rng.uniform(-0.3, 0.3, (n, 3))
    return x0, ((rng.integers(0, 1 << 24, (n, 8)) + 1) / 2.0 ** 24).astype(np.float32)


def check(cfg, x0, u, obstacles, in_place=False):
    from kgmt_gb300.planner import propagate_samples
    n = x0.shape[0]
    d_x0, d_u = torch.from_numpy(x0).to(DEV), torch.from_numpy(u).to(DEV)
    d_obs = torch.from_numpy(O.boxes(cfg, obstacles)).to(DEV)
    # one guard row behind every output: nothing is written past n
    x1 = d_x0 if in_place else torch.full((n + 1, cfg.sample_dim), 7.0, device=DEV)
    valid = torch.full((n + 1,), 9, dtype=torch.uint8, device=DEV)
    r1, r2 = (torch.full((n + 1,), -5, dtype=torch.int32, device=DEV) for _ in range(2))
    propagate_samples(cfg, d_x0, d_u, d_obs if len(obstacles) else None, len(obstacles), n, x1, valid, r1, r2)
    torch.cuda.synchronize()
    ox, ov, o1, o2 = O.propagate_f32(cfg, x0, u, obstacles)
    assert np.array_equal(valid.cpu().numpy(), np.append(ov, 9))
    assert np.array_equal(r1.cpu().numpy(), np.append(o1, -5)) and np.array_equal(r2.cpu().numpy(), np.append(o2, -5))
    got = x1.cpu().numpy()
    assert in_place or (got[n] == 7.0).all()
    assert np.array_equal(got[:n].view(np.uint32), ox.view(np.uint32))
    return ov


@pytest.mark.parametrize("model", sorted(MAKE))
@pytest.mark.parametrize("n,n_obs", [(1, 0), (31, 1), (129, 12), (4097, 10), (4097, 150), (118_000, 5), (118_013, 60), (250_001, 33)])
def test_sizes_match_oracle(model, n, n_obs):
    q = MAKE[model](seed=5, n_obstacles=n_obs)
    x0, u = inputs(q.config, n, n + n_obs)
    check(q.config, x0, u, q.obstacles)


@pytest.mark.parametrize("n", [900, 120_000])
def test_in_place_and_null_regions(n):
    """End rows over the parents' rows, as a caller may do; region ids left out."""
    from kgmt_gb300.planner import propagate_samples
    q = W.quadrotor_query(seed=6, n_obstacles=80)
    x0, u = inputs(q.config, n, 3)
    check(q.config, x0, u, q.obstacles, in_place=True)
    d = [torch.from_numpy(a).to(DEV) for a in (x0, u, q.obstacles)]
    x1, valid = torch.zeros_like(d[0]), torch.zeros(n, dtype=torch.uint8, device=DEV)
    propagate_samples(q.config, d[0], d[1], d[2], 80, n, x1, valid)
    ox, ov, _, _ = O.propagate_f32(q.config, x0, u, q.obstacles)
    assert np.array_equal(valid.cpu().numpy(), ov) and np.array_equal(x1.cpu().numpy().view(np.uint32), ox.view(np.uint32))


@pytest.mark.parametrize("kind", ["nan", "inverted", "covering", "outside", "many"])
@pytest.mark.parametrize("n", [5000, 120_000])
def test_boxes_the_grid_must_not_lose(kind, n):
    """Boxes that the culling grid refuses (a NaN face; more cell entries than
    it holds) or must still list (inverted, partly or wholly outside, very many)."""
    q = W.double_integrator_query(seed=8, n_obstacles=3500 if kind == "many" else 100)
    rng = np.random.default_rng(4)
    b = q.obstacles
    if kind == "nan":
        b[7, 2] = b[50, 3] = np.nan
    elif kind == "inverted":
        b[::3, :3], b[::3, 3:] = b[::3, 3:].copy(), b[::3, :3].copy()
    elif kind == "covering":
        b[:] = [-1.0, -1.0, 0.4, 2.0, 2.0, 0.42]
        b[:, 2] += rng.uniform(0.0, 0.3, len(b)).astype(np.float32)
        b[:, 5] = b[:, 2] + 0.5
    elif kind == "outside":
        b[::2] += np.float32([0.7, -0.6, 0.0, 0.7, -0.6, 0.0])
    else:
        b[:, 3:] = b[:, :3] + 0.012
    x0, u = inputs(q.config, n, 17)
    check(q.config, x0, u, b)


@pytest.mark.parametrize("model", sorted(MAKE))
@pytest.mark.parametrize("n,n_obs", [(58_368, 7), (58_369, 9), (97_280, 9), (97_281, 7), (1, 400), (9, 400), (600, 5_200), (600, 6_000), (20_000, 5_300)])
def test_edges_of_the_forms(model, n, n_obs):
    """A full wave of the plain and of the wide form and one sample more, and few
    samples and very many boxes, where the grid does not pay or has no room."""
    q = MAKE[model](seed=11, n_obstacles=n_obs if n_obs < 100 else 50)
    if n_obs >= 100:
        rng = np.random.default_rng(n_obs)
        lo = rng.uniform(0.0, 0.97, (n_obs, 3)).astype(np.float32)
        q.obstacles = np.concatenate([lo, lo + np.float32(0.01)], 1)
    x0, u = inputs(q.config, n, n + n_obs)
    check(q.config, x0, u, q.obstacles)
