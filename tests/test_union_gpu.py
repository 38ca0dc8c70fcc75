"""Unions of point clouds and primitives: the primitives are evaluated by a thread a point, the clouds by a warp a
point, wherever they stand in the union."""
import numpy as np
import pytest

from plainmp_gb300 import BoxSDF, CloudSDF, CylinderSDF, Pose, SphereSDF, UnionSDF, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _prims(n, seed=4):
    r = np.random.default_rng(seed)
    out = []
    for k in range(n):
        pose = Pose(r.uniform(-1, 1, 3), W._random_rotation(r) if k % 2 else np.eye(3))
        out.append([BoxSDF(r.uniform(0.05, 0.3, 3), pose), SphereSDF(0.1, pose), CylinderSDF(0.1, 0.3, pose)][k % 3])
    return out


def _cloud(seed):
    return CloudSDF(W.box_surface_cloud(2000, seed=seed).astype(np.float64), 0.01 * seed)


@pytest.mark.parametrize("n,clouds", [(0, [0]), (1, [0]), (1, [1]), (31, [31]), (32, [0, 32]), (33, [32, 33]), (100, [5, 40, 41, 70, 102])])
def test_every_place_in_the_union(n, clouds):
    parts = _prims(n)
    for k, at in enumerate(clouds):
        parts.insert(at, _cloud(k))
    u = UnionSDF(parts)
    rng = np.random.default_rng(n)
    pts = torch.from_numpy(rng.uniform(-1.5, 1.5, (1001, 3))).cuda()
    rad = torch.from_numpy(rng.choice([0.0, 1e-7, 0.05, 0.3], 1001)).cuda()
    each = torch.stack([p.evaluate_points(pts) for p in parts])
    assert torch.equal(u.evaluate_points(pts), each.min(dim=0).values)
    outside = torch.stack([p.is_outside_points(pts, rad) for p in parts])
    assert torch.equal(u.is_outside_points(pts, rad), outside.min(dim=0).values)
    _, cst, _ = scenes.make_constraint(W.chain7_robot(), None)
    Q = torch.from_numpy(W.chain7_configs(65, seed=n)).cuda()
    dist = []
    for p in parts:
        cst.set_sdf(p)
        dist.append(cst.sphere_distances(Q))
    cst.set_sdf(u)
    assert torch.equal(cst.sphere_distances(Q), torch.stack(dist).min(dim=0).values)


def _ms(fn):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    fn()
    t = []
    for _ in range(3):
        a.record()
        fn()
        b.record()
        b.synchronize()
        t.append(a.elapsed_time(b))
    return min(t)


def test_primitives_cost_the_same_beside_a_cloud():
    """1,000 primitives and a cloud take about as long as each by itself in a row (a warp a point for both took 30
    times as long as the primitives alone); 3 allows for two passes over the points and noise."""
    prims, cloud = _prims(1000), CloudSDF(W.box_surface_cloud(20_000).astype(np.float64), 0.0)
    pts = torch.from_numpy(np.random.default_rng(0).uniform(-1, 1, (100_000, 3))).cuda()
    rad = torch.full((100_000,), 0.01, dtype=torch.float64, device="cuda")
    for call in (lambda s: s.evaluate_points(pts), lambda s: s.is_outside_points(pts, rad)):
        alone = _ms(lambda s=UnionSDF(prims): call(s)) + _ms(lambda s=UnionSDF([cloud]): call(s))
        assert _ms(lambda s=UnionSDF([cloud] + prims): call(s)) < 3 * alone
