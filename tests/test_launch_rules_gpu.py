"""The launch rules of the fast calls (no shape set): batches at the edges of the rules give the plain method's
booleans, and one set of FP32 distances whatever the rule picked."""
import numpy as np
import pytest

from plainmp_gb300 import scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("robot,env", [("chain7", "prims"), ("planar", "cloud"), ("dualarm", "cloud"), ("dualarm", "prims")])
def test_batches_at_the_edges_of_the_rules(robot, env):
    r = {"chain7": W.chain7_robot, "planar": W.planar_chain7_robot, "dualarm": W.dualarm_robot}[robot]()
    scene = W.chain7_scene() if env == "prims" else W.Scene(cloud=W.box_surface_cloud(20_000, seed=2))
    _, cst, _ = scenes.make_constraint(r, scene)
    resident = 4 * torch.cuda.get_device_properties(0).multi_processor_count  # blocks of 256 threads
    sizes = [1, 7, 8, 9, 8 * resident, 8 * resident + 1, 16 * resident, 16 * resident + 1]
    Q = torch.tensor(np.random.default_rng(6).uniform(-np.pi, np.pi, size=(max(sizes), cst.q_dim())), device="cuda")
    ref = cst.is_valid_batch(Q)
    ok, dist = cst.is_valid_fast(Q, distances=True)
    assert torch.equal(ok, ref) and 0 < int(ref.sum()) < len(ref)
    for n in sizes:
        assert torch.equal(cst.is_valid_fast(Q[:n]), ref[:n])
        ok, d = cst.is_valid_fast(Q[:n], distances=True)
        assert torch.equal(ok, ref[:n]) and torch.equal(d, dist[:n])
