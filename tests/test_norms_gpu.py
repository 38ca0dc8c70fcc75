"""Rotations off unit norm: the URDF's axes and the base pose are taken as they are given (the reference normalizes
neither), so their quaternions scale the link transforms.  The FP32 bounds are derived for unit quaternions and may
clear nothing there.  Against the oracle, which computes in FP64 alone."""
import re

import numpy as np
import pytest

from plainmp_gb300 import BoxMotionValidator, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _robot(scale, base="FIXED"):
    """The chain with its axes scaled: the k-th by scale where k is even, by its reciprocal where k is odd."""
    r = W.chain7_robot()
    k = -1

    def axis(m):
        nonlocal k
        k += 1
        f = scale if k % 2 == 0 else 1.0 / scale
        return '<axis xyz="%s"/>' % " ".join(repr(float(v) * f) for v in m.group(1).split())

    return W.Robot(re.sub(r'<axis xyz="([^"]*)"/>', axis, r.urdf), r.control_joints, r.end_link, r.spheres, r.self_pairs, base_type=base)


CASES = [("axes", 3.0), ("axes", 1.05), ("axes", 1.0001), ("axes", 1.0 + 2e-5), ("base", 1.7), ("base", 1.0 + 1e-4), ("base", 0.4)]


@pytest.fixture(scope="module", params=CASES, ids=lambda c: f"{c[0]}-{c[1]:g}")
def pair(request, oracle):
    what, scale = request.param
    r = _robot(scale) if what == "axes" else W.chain7_robot()
    # a large scene: with scaled rotations the links end tens of metres away
    big = 30.0 if scale > 1.5 and what == "axes" else 1.0
    prims = [W.Primitive(p.kind, np.array([0.55] * 3) + (p.position - 0.55) * big, p.rotation, tuple(s * big for s in p.size))
             for p in W.chain7_scene(1).primitives]
    scene = W.Scene(prims)
    kin, cst, _ = scenes.make_constraint(r, scene)
    m, oc, _ = oracle.make_constraint(r, scene)
    if what == "base":
        pose = np.array([0.1, -0.2, 0.3, 0.5, -0.5, 0.5, 0.5])
        pose[3:] *= scale
        kin.set_base_pose(pose)
        m.set_base_pose(pose)
    # a bound of |q|^2 along the chain: the even joints' axes, the base
    return cst, oc, max(1.0, scale ** 2) ** (4 if what == "axes" else 1)


N = 20000  # enough that an error bound short by a few orders meets a decision or a least term


def test_fp64_method_decides(pair):
    cst, oc, n2 = pair
    Q = W.chain7_configs(N, seed=31)
    ref = oc.is_valid(Q, threads=8)
    assert 0 < ref.sum() < N
    assert np.array_equal(cst.is_valid_batch(Q), ref)
    s1, s2 = Q[:200], Q[:200] + np.linspace(-0.2, 0.2, 7)
    assert np.array_equal(BoxMotionValidator(cst, [0.05] * 7).check_motion_batch(s1, s2), oc.check_motion(s1, s2, 0, width=[0.05] * 7)[0])


def test_fp64_values(pair):
    """The least value is the reference's: same term, so the same bits up to sin and cos (2 units in the last place of
    each joint, carried by transforms of up to 1e3: 1e-9; a wrong term is off by more than its FP32 bound, 1e-6)."""
    cst, oc, n2 = pair
    Q = W.chain7_configs(N, seed=33)
    rv, _ = oc.evaluate(Q, threads=8)
    v, _ = cst.evaluate_batch(Q)
    np.testing.assert_allclose(v, rv, atol=1e-9, rtol=0)


def test_fast_path_decides(pair):
    cst, oc, n2 = pair
    Q = W.chain7_configs(N, seed=35)
    ref = oc.is_valid(Q, threads=8)
    assert np.array_equal(cst.is_valid_fast(Q), ref)
    s1, s2 = Q[:200], Q[:200] + np.linspace(-0.2, 0.2, 7)
    assert np.array_equal(BoxMotionValidator(cst, [0.05] * 7).check_motion_fast(s1, s2), oc.check_motion(s1, s2, 0, width=[0.05] * 7)[0])


def test_fast_path_agrees_on_many_states(pair):
    """Two million states, against the FP64 method: decisions inside a bound that is too small are few."""
    import torch

    cst, _, n2 = pair
    for k in range(10):
        Q = torch.from_numpy(W.chain7_configs(200_000, seed=100 + k)).cuda()
        assert torch.equal(cst.is_valid_fast(Q), cst.is_valid_batch(Q))


def test_fast_distances(pair):
    """The FP32 distance bound of unit rotations (1e-6 + 64 units of roundoff of magnitudes below 20 m) times n2, which
    every error of a rotated vector is proportional to at most."""
    cst, oc, n2 = pair
    Q = W.chain7_configs(2000, seed=37)
    _, d = cst.is_valid_fast(Q, distances=True)
    ref = np.minimum(oc.sphere_distances(Q, threads=8), 0.1)
    assert np.abs(d.astype(np.float64) - ref).max() < (1e-6 + 64 * 2.0 ** -24 * 21) * n2


def test_rounded_axes_keep_the_fast_path(pair):
    """Up to 1e-3 of excess in all, as axes of four digits have, the bounds are widened; above it everything is checked
    exactly."""
    cst, oc, n2 = pair
    _, st = cst.is_valid_fast(W.chain7_configs(3000, seed=39), stats=True)
    assert st["rechecked_configs"] == (0 if n2 < 1.001 else 3000)
