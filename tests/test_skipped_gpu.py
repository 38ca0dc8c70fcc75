"""Waypoints of edges already known invalid cost the edge kernel next to nothing, and change no answer."""
import numpy as np
import pytest

from plainmp_gb300 import BoxMotionValidator, Pose, SphereSDF, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


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


def test_long_edge_whose_goal_collides():
    """One edge of 100,000 waypoints: where its goal collides, a chunk of waypoints is a counter, a search and two
    barriers; where it is free, eight phases and more.  A sixth leaves room for a chunk's fixed costs."""
    r = W.chain7_robot()
    _, cst, _ = scenes.make_constraint(r, None, self_collision=False)
    v = BoxMotionValidator(cst, [0.05] * 7)
    s1 = torch.zeros((1, 7), dtype=torch.float64, device="cuda")
    s2 = s1 + 5000.0 * torch.linspace(0.5, 1.0, 7, dtype=torch.float64, device="cuda")
    ms = []
    for radius in (10.0, 0.01):
        cst.set_sdf(SphereSDF(radius, Pose([9.0, 0.0, 0.0], np.eye(3))))
        assert v.check_motion_fast(s1, s2).item() == (radius < 1.0)
        ms.append(_ms(lambda: v.check_motion_fast(s1, s2)))
    assert ms[0] < ms[1] / 6, ms


@pytest.mark.parametrize("E", [1, 3, 40])
def test_mixed_edges(oracle, E):
    """Free edges, edges that collide at the goal or on the way and non-finite ones in one chunk."""
    r, s = W.chain7_robot(), W.chain7_scene()
    _, cst, _ = scenes.make_constraint(r, s)
    _, oc, _ = oracle.make_constraint(r, s)
    s1, s2 = W.chain7_edges(E, seed=E, max_waypoints=9)
    s1, s2 = np.repeat(s1, 30, axis=0), np.repeat(s2, 30, axis=0)
    s2[7::30, 3] = np.nan
    ref, _ = oc.check_motion(s1, s2, 0, width=[0.05] * 7)
    for got in (BoxMotionValidator(cst, [0.05] * 7).check_motion_fast(s1, s2),
                BoxMotionValidator(cst, [0.05] * 7).check_motion_batch(s1, s2)):
        assert np.array_equal(got, ref)
