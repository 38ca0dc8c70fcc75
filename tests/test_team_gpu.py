"""The FP64 method by warps (k_is_valid64, k_check_motion64, k_evaluate64) at the edges of its blocks and
launch rules, and on the primitives and spheres whose gates have cases of their own, against the oracle."""
import numpy as np
import pytest

from plainmp_gb300 import BaseType, BoxMotionValidator, KinematicModel, SphereAttachmentSpec, SphereCollisionCst
from plainmp_gb300 import BoxSDF, CloudSDF, CylinderSDF, EuclideanMotionValidator, GroundSDF, Pose, SphereSDF, UnionSDF
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# 4 configurations per block, up to 4 x 152 SMs one
SIZES = [1, 3, 4, 5, 7, 8, 9, 607, 608, 609, 613]


def _mixed(oracle, base):
    """The chain with one self-only link and one link of spheres below 1e-6 m, against every kind of primitive."""
    r = W.chain7_robot()
    r = W.Robot(r.urdf, r.control_joints, r.end_link, r.spheres, r.self_pairs, base_type=base)
    r.spheres[1].only_self_collision = True
    r.spheres[4].radii[:] = 5e-7
    rng = np.random.default_rng(3)
    cloud = W.box_surface_cloud(n_points=4000, n_boxes=3, seed=3, center=(0.3, 0.4, 0.2))
    rot = W._random_rotation(rng)
    rz = np.array([[0.8, -0.6, 0], [0.6, 0.8, 0], [0, 0, 1.0]])
    parts = [("box", ([0.2, 0.3, 0.1], [0.5, -0.4, 0.3], np.eye(3))), ("box", ([0.3, 0.1, 0.2], [-0.5, 0.3, 0.6], rz)),
             ("box", ([0.2, 0.2, 0.2], [0.4, 0.7, 0.9], rot)), ("cylinder", (0.1, 0.4, [-0.3, -0.5, 0.8], rz)),
             ("cylinder", (0.15, 0.2, [0.1, 0.9, 0.4], rot)), ("sphere", (0.2, [0.9, 0.2, 0.5], np.eye(3))), ("ground", (0.9,)),
             ("cloud", (cloud.astype(np.float64), 0.01))]
    mine, ref = [], []
    for kind, a in parts:
        if kind == "box":
            mine.append(BoxSDF(a[0], Pose(a[1], a[2])))
        elif kind == "cylinder":
            mine.append(CylinderSDF(a[0], a[1], Pose(a[2], a[3])))
        elif kind == "sphere":
            mine.append(SphereSDF(a[0], Pose(a[1], a[2])))
        else:
            mine.append(GroundSDF(*a) if kind == "ground" else CloudSDF(*a))
        ref.append(getattr(oracle.Sdf, kind)(*a))
    kin = KinematicModel(r.urdf)
    specs = [SphereAttachmentSpec(s.parent_link_name, s.relative_positions, s.radii, s.only_self_collision) for s in r.spheres]
    cst = SphereCollisionCst(kin, r.control_joints, BaseType[base], specs, r.self_pairs)
    cst.set_sdf(UnionSDF(mine))
    _, oc, _ = oracle.make_constraint(r, None)
    oc.set_sdf(oracle.Sdf.union(ref))
    return cst, oc


def _configs(base, n, seed):
    rng = np.random.default_rng(seed)
    q = W.chain7_configs(n, seed=seed)
    extra = {"FIXED": 0, "PLANAR": 3, "FLOATING": 6}[base]
    return np.concatenate([q, rng.normal(0.0, 0.3, size=(n, extra))], axis=1)


@pytest.mark.parametrize("base", ["FIXED", "PLANAR", "FLOATING"])
def test_mixed_scene_every_block_edge(oracle, base):
    cst, oc = _mixed(oracle, base)
    Q = _configs(base, max(SIZES), seed=17)
    ref = oc.is_valid(Q, threads=8)
    rv, rJ = oc.evaluate(Q, threads=8)
    assert 0 < ref.sum() < len(ref) and (np.abs(rv) < 0.1).any(axis=0).all()
    for n in SIZES:
        assert np.array_equal(cst.is_valid_batch(Q[:n]), ref[:n])
        v, J = cst.evaluate_batch(Q[:n])
        np.testing.assert_allclose(v, rv[:n], atol=1e-9, rtol=0)  # the bars of the plain method's other tests
        np.testing.assert_allclose(J[:, :, :7], rJ[:n, :, :7], atol=1e-9, rtol=0)
        np.testing.assert_allclose(J[:, :, 7:], rJ[:n, :, 7:], atol=1e-6, rtol=0)


def test_non_finite_configurations(oracle):
    cst, oc = _mixed(oracle, "FIXED")
    Q = _configs("FIXED", 64, seed=5)
    Q[::3, 2] = np.nan
    Q[1::3, 0] = np.inf
    assert np.array_equal(cst.is_valid_batch(Q), oc.is_valid(Q, threads=8))


@pytest.mark.parametrize("E", [1, 2, 152, 153])  # up to one edge per SM, a block takes 16 waypoints at a time; then 8
def test_edges_and_counts(oracle, E):
    cst, oc = _mixed(oracle, "FIXED")
    oc.set_sdf(oracle.Sdf.sphere(0.15, [0.6, 0.6, 0.6], np.eye(3)))  # few collisions: edges run to their ends
    cst.set_sdf(SphereSDF(0.15, Pose([0.6, 0.6, 0.6], np.eye(3))))
    rng = np.random.default_rng(E)
    s1 = W.chain7_configs(E, seed=E)
    s2 = s1 + rng.normal(0.0, 0.4, size=s1.shape)
    s2[0] = s1[0] + np.linspace(0.1, 7.0, 7)  # more than 129 waypoints: in order, not farthest first
    if E > 2:
        s2[1] = s1[1]  # no length
        s2[2] = s1[2] + 1e-9
    for val, kind, args in ((BoxMotionValidator(cst, [0.04] * 7), 0, dict(width=[0.04] * 7)),
                            (EuclideanMotionValidator(cst, 0.05), 1, dict(resolution=0.05))):
        got, count = val.check_motion_batch(s1, s2, return_count=True)
        ref, rcount = oc.check_motion(s1, s2, kind, **args)
        assert np.array_equal(got, ref) and count == rcount


@pytest.mark.parametrize("base", ["FIXED", "PLANAR", "FLOATING"])
def test_single_state_check_leaves_the_state(oracle, base):
    """is_valid(q) checks and updates the model in one launch: the answer is the batch's, the spheres of the
    state are update_kintree's, over several states in a row and host batches at the zero-copy limit."""
    cst, oc = _mixed(oracle, base)
    Q = _configs(base, 65, seed=29)
    ref = oc.is_valid(Q, threads=8)
    for n in (63, 64, 65):
        assert np.array_equal(cst.is_valid_batch(Q[:n]), ref[:n])
        v, J = cst.evaluate_batch(Q[:n])
        vd, Jd = cst.evaluate_batch(Q)
        assert np.array_equal(v, vd[:n]) and np.array_equal(J, Jd[:n])
    for q, ok in zip(Q[:6], ref[:6]):
        assert cst.is_valid(q) == bool(ok)
        got = [(*c, r) for c, r in cst.get_all_spheres()]
        cst.update_kintree(q, high_accuracy=base != "FIXED")
        assert np.array_equal(got, [(*c, r) for c, r in cst.get_all_spheres()])
