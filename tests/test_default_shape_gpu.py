"""The launch shape that a call picks where none is set, by the name of the kernel it launches: blocks of 8 or 16
configurations while they are all resident, which depends on the room that the tables leave, then by the shared memory
and the robot's spheres."""
import re

import numpy as np
import pytest

from plainmp_gb300 import BoxSDF, Pose, UnionSDF, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def many_spheres(k):
    """The chain with k spheres a link."""
    r, rng, specs = W.chain7_robot(), np.random.default_rng(1), []
    for s in r.spheres:
        lo, hi = s.relative_positions.min(1, keepdims=True), s.relative_positions.max(1, keepdims=True)
        specs.append(W.SphereSpec(s.parent_link_name, lo + (hi - lo) * rng.uniform(size=(3, k)), rng.uniform(0.01, 0.04, k)))
    return W.Robot(r.urdf, r.control_joints, r.end_link, specs, r.self_pairs)


def boxes(n):
    r = np.random.default_rng(4)
    return UnionSDF([BoxSDF(r.uniform(0.03, 0.1, 3), Pose(r.uniform(-1, 1, 3), W._random_rotation(r))) for _ in range(n)])


def shape_of(call, kernel):
    """(configurations, threads) a block of the call's kernel."""
    from torch.profiler import ProfilerActivity, profile

    call()
    torch.cuda.synchronize()
    for _ in range(3):  # a process's first profile may come back empty
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            call()
            torch.cuda.synchronize()
        names = {m.groups() for e in p.events() if (m := re.search(kernel + r"<(\d+), (\d+)", e.name))}
        if names:
            break
    assert len(names) == 1, names
    return tuple(int(v) for v in names.pop())


@pytest.fixture(scope="module")
def made():
    cache = {}

    def make(robot, scene):
        if (robot, scene) not in cache:
            r = {"chain": W.chain7_robot, "dual": W.dualarm_robot, "350": lambda: many_spheres(50)}[robot]()
            _, cst, _ = scenes.make_constraint(r, W.Scene(cloud=W.box_surface_cloud(20_000)) if scene == "cloud" else None)
            if scene != "cloud":
                cst.set_sdf(boxes(scene) if scene > 20 else scenes.primitives_sdf(W.Scene(W.chain7_scene().primitives[:scene])))
            cache[robot, scene] = cst
        return cache[robot, scene]

    return make


# B: blocks of 8 an SM, plus
@pytest.mark.parametrize("robot,scene,blocks,plus,distances,shape", [
    ("chain", 20, 4, 0, False, (8, 256)), ("chain", 20, 4, 0, True, (8, 256)),
    ("chain", 20, 4, 1, False, (16, 256)), ("chain", 20, 8, 0, True, (16, 256)), ("chain", 20, 8, 1, False, (16, 128)),
    ("chain", 1000, 2, 0, False, (8, 256)), ("chain", 1000, 2, 1, False, (16, 256)), ("chain", 1000, 2, 1, True, (16, 256)),
    ("dual", 20, 8, 1, False, (16, 128)), ("dual", 20, 8, 1, True, (16, 256)), ("dual", "cloud", 8, 1, False, (16, 256)),
    ("350", 8, 4, 1, False, (32, 256)), ("350", 8, 4, 1, True, (16, 256)), ("350", 8, 8, 1, False, (16, 128)),
    ("350", 1000, 4, 1, False, (16, 256)),
])
def test_shape_by_batch_tables_and_spheres(made, robot, scene, blocks, plus, distances, shape):
    cst = made(robot, scene)
    B = 8 * blocks * torch.cuda.get_device_properties(0).multi_processor_count + plus
    Q = torch.from_numpy(np.random.default_rng(B).uniform(-np.pi, np.pi, (B, cst.q_dim()))).cuda()
    assert shape_of(lambda: cst.is_valid_fast(Q, distances=distances), "k_fast_valid") == shape
    ref = cst.is_valid_batch(Q)
    got = cst.is_valid_fast(Q, distances=distances)
    assert torch.equal(got[0] if distances else got, ref)
