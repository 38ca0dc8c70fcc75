"""Many edges in one call of the FP64 method: several a block, so short ones and ones without length cost no more
than their waypoints."""
import numpy as np
import pytest

from plainmp_gb300 import BoxMotionValidator, EuclideanMotionValidator, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def chain(oracle):
    r, s = W.chain7_robot(), W.chain7_scene()
    return scenes.make_constraint(r, s)[1], oracle.make_constraint(r, s)[1]


# edges a block: 1 up to 16 per SM, 2 from there, 64 from 512 per SM (times the SMs, plus)
@pytest.mark.parametrize("per_sm,plus", [(1, 1), (16, -1), (16, 0), (16, 1), (20, 7), (511, 3), (512, 0), (600, 5)])
def test_edges_and_counts_at_the_rules_edges(chain, per_sm, plus):
    cst, oc = chain
    E = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + plus
    rng = np.random.default_rng(E)
    s1 = W.chain7_configs(E, seed=1)
    s2 = s1 + rng.uniform(-1, 1, s1.shape) * rng.choice([0.0, 0.03, 0.2], (E, 1), p=[0.2, 0.7, 0.1])
    s2[5] = s1[5] + np.linspace(0.1, 7.0, 7)  # more than 129 waypoints
    s2[E - 1] = s1[E - 1] + 0.5
    a, b = torch.from_numpy(s1).cuda(), torch.from_numpy(s2).cuda()
    for val, kind, args in ((BoxMotionValidator(cst, [0.04] * 7), 0, dict(width=[0.04] * 7)),
                            (EuclideanMotionValidator(cst, 0.05), 1, dict(resolution=0.05))):
        ref, rcount = oc.check_motion(s1, s2, kind, **args, threads=8)
        got, count = val.check_motion_batch(a, b, return_count=True)
        assert np.array_equal(got.cpu().numpy(), ref) and count == rcount


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


def test_one_waypoint_costs_one_state(chain):
    """Edges of one waypoint are that many states to check, and edges without length none: against the batch check of
    the goals, 3 leaves room for the set-up of an edge (a block an edge took 7 times as long)."""
    cst, _ = chain
    goal = torch.from_numpy(W.chain7_configs(100_000, seed=2)).cuda()
    v = BoxMotionValidator(cst, [0.05] * 7)
    states = _ms(lambda: cst.is_valid_batch(goal))
    assert _ms(lambda: v.check_motion_batch(goal + 0.02, goal)) < 3 * states
    assert _ms(lambda: v.check_motion_batch(goal, goal)) < states / 3
