"""Sizes at which a launch's shared memory passes a limit of the device, each in a process of its own: a larger table
launched before would have raised the limit."""
import re
import subprocess
import sys
import threading
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REPO = Path(__file__).resolve().parent.parent


def chain(links):
    """A constraint of `links` FK slots (the root and a chain): seven control joints, one sphere on every third link."""
    from plainmp_gb300 import scenes
    from plainmp_gb300 import workloads as W

    offsets, axes, centres, radii = W._chain_params(0, links - 1)
    body = W._chain_xml("", "base_link", 0.3 * offsets, axes, mirror_y=False)
    urdf = f'<?xml version="1.0"?>\n<robot name="c">\n  <link name="base_link"/>\n{body}\n</robot>\n'
    specs = [W.SphereSpec(f"link{k}", 0.3 * centres[k - 1][:1].T, 0.3 * radii[k - 1][:1]) for k in range(links - 1, 0, -3)]
    pairs = [(specs[0].parent_link_name, specs[-1].parent_link_name)] if len(specs) > 1 else []
    r = W.Robot(urdf, [f"j{k}" for k in range(1, 8)], f"link{links - 1}", specs, pairs)
    return r, scenes.make_constraint(r, W.chain7_scene())[1]


def one_size(links, edges):
    """Edges of a constraint of that many slots, against the oracle."""
    from oracle import pyoracle
    from plainmp_gb300 import BoxMotionValidator
    from plainmp_gb300 import workloads as W

    r, cst = chain(links)
    _, oc, _ = pyoracle.make_constraint(r, W.chain7_scene())
    s1, s2 = W.chain7_edges(edges, seed=links, max_waypoints=20)
    got = BoxMotionValidator(cst, [0.05] * 7).check_motion_batch(s1, s2)
    ref, _ = oc.check_motion(s1, s2, 0, width=[0.05] * 7, threads=4)
    assert np.array_equal(got, ref)


def _child(call):
    code = f"import sys; sys.path[:0] = [{str(REPO)!r}, {str(REPO / 'tests')!r}]; import test_limits_gpu as t; t.{call}"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


# static and dynamic shared memory together pass 48 KB at 27 slots with 16 waypoints a block (an edge or more per SM),
# and at 53 slots with 8 (more edges than SMs); 64 slots are the most
@pytest.mark.parametrize("links", [26, 27, 28, 52, 53, 54, 55, 64])
def test_edges_of_long_chains(oracle, links):
    import torch

    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    _child(f"one_size({links}, {1 if links < 40 else n_sm + 1})")
    if links == 64:
        _child(f"one_size({links}, 1)")


def two_threads():
    """Constraints of different sizes, each on a thread of its own."""
    from plainmp_gb300 import BoxMotionValidator
    from plainmp_gb300 import workloads as W

    s1, s2 = W.chain7_edges(1, seed=3, max_waypoints=3)
    errors = []

    def work(links):
        try:
            v = BoxMotionValidator(chain(links)[1], [0.05] * 7)
            for _ in range(1500):
                v.check_motion_batch(s1, s2)
        except Exception as e:
            errors.append((links, repr(e)))

    threads = [threading.Thread(target=work, args=(n,)) for n in (60, 30, 45)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors


def test_threads_with_tables_of_different_sizes():
    _child("two_threads()")


def two_threads_of_costs():
    """The same with the differentiable costs."""
    import torch

    from plainmp_gb300 import diff

    made = [chain(n)[1] for n in (60, 40, 50)]
    q = torch.tensor(np.zeros((4, 7), np.float32), device="cuda")
    errors = []

    def work(cst):
        try:
            for _ in range(1500):
                diff.ik_cost_grad(cst, q, None, None)
        except Exception as e:
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(c,)) for c in made]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors


def test_threads_of_costs_with_tables_of_different_sizes():
    _child("two_threads_of_costs()")


def test_largest_tables_of_the_fast_calls():
    """A chain of 6,357 spheres against 20 primitives, about the most that a block's shared memory holds: validity,
    edges and the call that allocates nothing, against the FP64 method."""
    import ctypes as C

    import torch

    from plainmp_gb300._lib import lib

    from plainmp_gb300 import BoxMotionValidator, scenes
    from plainmp_gb300 import workloads as W

    r, rng, specs = W.chain7_robot(), np.random.default_rng(1), []
    for k, s in enumerate(r.spheres):
        lo, hi = s.relative_positions.min(1, keepdims=True), s.relative_positions.max(1, keepdims=True)
        n = 908 + (k == 0)
        specs.append(W.SphereSpec(s.parent_link_name, lo + (hi - lo) * rng.uniform(size=(3, n)), rng.uniform(0.001, 0.01, n)))
    many = W.Robot(r.urdf, r.control_joints, r.end_link, specs, [])
    _, cst, _ = scenes.make_constraint(many, W.chain7_scene(), reorder=False)
    assert cst.n_spheres == 6357
    Q = torch.from_numpy(W.chain7_configs(300, seed=8)).cuda()
    ref = cst.is_valid_batch(Q)
    assert 0 < int(ref.sum()) < len(ref)
    assert torch.equal(cst.is_valid_fast(Q), ref)
    v = BoxMotionValidator(cst, [0.05] * 7)
    assert torch.equal(v.check_motion_fast(Q, Q + 0.07), v.check_motion_batch(Q, Q + 0.07))
    out = torch.full_like(ref, 7)
    torch.cuda.synchronize()
    assert lib.pmgpu_cst_is_valid_fast_noalloc(cst._h, C.c_void_p(Q.data_ptr()), C.c_int64(len(Q)), C.c_void_p(out.data_ptr()), None, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(out, ref)
