"""Batches on both sides of the lines between launch forms that depend on the SM count or lie between host staging
forms, whatever the device."""
import numpy as np
import pytest

from plainmp_gb300 import BoxMotionValidator, scenes
from plainmp_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def chain(oracle):
    r, s = W.chain7_robot(), W.chain7_scene()
    return scenes.make_constraint(r, s)[1], oracle.make_constraint(r, s)[1]


def test_fp64_batches_by_sm_count(chain):
    """One configuration a block up to 4 per SM, then four; edges by block up to one per SM, then several."""
    cst, oc = chain
    n_sm = torch.cuda.get_device_properties(0).multi_processor_count
    Q = W.chain7_configs(4 * n_sm + 5, seed=41)
    ref = oc.is_valid(Q, threads=8)
    rv, rJ = oc.evaluate(Q, threads=8)
    Qd = torch.from_numpy(Q).cuda()
    for n in (4 * n_sm - 1, 4 * n_sm, 4 * n_sm + 1, 4 * n_sm + 5):
        assert np.array_equal(cst.is_valid_batch(Qd[:n]).cpu().numpy(), ref[:n])
        v, J = cst.evaluate_batch(Qd[:n])
        np.testing.assert_allclose(v.cpu().numpy(), rv[:n], atol=1e-9, rtol=0)  # the bars of the method's other tests
        np.testing.assert_allclose(J.cpu().numpy(), rJ[:n], atol=1e-9, rtol=0)
    s1, s2 = W.chain7_edges(n_sm + 1, seed=42, max_waypoints=40)
    e_ref, _ = oc.check_motion(s1, s2, 0, width=[0.05] * 7, threads=8)
    for E in (n_sm - 1, n_sm, n_sm + 1):
        got = BoxMotionValidator(cst, [0.05] * 7).check_motion_batch(torch.from_numpy(s1[:E]).cuda(), torch.from_numpy(s2[:E]).cuda())
        assert np.array_equal(got.cpu().numpy(), e_ref[:E])


def test_host_batches_at_the_zero_copy_limit(chain):
    """Host batches whose kernel reads and writes page-locked memory (up to 2,048 states, validity only) and those
    that are copied."""
    cst, _ = chain
    Q = W.chain7_configs(2049, seed=43)
    ref = cst.is_valid_batch(torch.from_numpy(Q).cuda()).cpu().numpy()
    assert 0 < ref.sum() < len(ref)
    for n in (1, 2047, 2048, 2049):
        assert np.array_equal(cst.is_valid_fast(Q[:n]), ref[:n])
        ok, _ = cst.is_valid_fast(Q[:n], distances=True)
        assert np.array_equal(ok, ref[:n])
