"""Exact FP64 cloud queries (KDTree.query / sqdist, CloudSDF.evaluate / is_outside) where the cooperative
search can go wrong, against a search over every point in the same FP64 expression (bit for bit)."""
import numpy as np
import pytest

from plainmp_gb300 import BoxSDF, CloudSDF, UnionSDF

pytestmark = pytest.mark.gpu


def _brute(points, q):
    d = points[None, :, :] - q[:, None, :]
    return (d[..., 0] * d[..., 0] + (d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2])).min(axis=1)


def _clouds():
    rng = np.random.default_rng(11)
    surface = rng.uniform(-0.4, 0.4, size=(3000, 3))
    surface[:, 2] = 0.05 * np.round(surface[:, 2] / 0.05)
    lattice = np.stack(np.meshgrid(*[np.arange(8) * 0.05] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    return {
        "one": np.array([[0.3, -0.2, 0.7]]),
        "coincident": np.repeat(np.array([[0.1, 0.1, 0.1], [0.1, 0.1, 0.4]]), 70, axis=0),
        "lattice": lattice,  # many equidistant points
        "layers": surface,
        "wide": rng.uniform(-6.0, 6.0, size=(400, 3)),  # most queries far from every point
        "offset": 40.0 + rng.uniform(-0.5, 0.5, size=(500, 3)),  # FP32 resolves 4 um there
    }


@pytest.mark.parametrize("name", ["one", "coincident", "lattice", "layers", "wide", "offset"])
def test_nearest_edges(name):
    pts = _clouds()[name]
    rng = np.random.default_rng(7)
    span = pts.max(0) - pts.min(0) + 0.1
    near = pts[rng.integers(0, len(pts), 257)] + rng.normal(0.0, 0.01, size=(257, 3))
    q = np.concatenate([
        near,
        pts[:31],  # on the points
        (pts[:40] + pts[rng.permutation(len(pts))[: len(pts[:40])]]) / 2,  # equidistant from two points
        pts.mean(0) + rng.uniform(-1.5, 1.5, size=(300, 3)) * span,
        pts.mean(0) + rng.uniform(-1.0, 1.0, size=(33, 3)) * 1e3,
        pts.mean(0) + np.array([[1e9, 0, 0], [0, -1e14, 0], [1e17, 1e17, 0], [0, 0, 1e25]]),
    ])
    sdf = CloudSDF(pts, 0.02)
    ref = _brute(pts, q)
    for n in (1, 2, 31, 33, len(q)):
        sq, at = sdf.nearest(q[:n])
        assert np.array_equal(sq, ref[:n])
        d = at - q[:n]
        assert np.array_equal(d[:, 0] * d[:, 0] + (d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]), ref[:n])
    assert np.array_equal(sdf.evaluate_points(q), np.sqrt(ref) - 0.02)
    box = BoxSDF([0.1, 0.2, 0.3])
    both = UnionSDF([box, sdf]).evaluate_points(q)
    assert np.array_equal(both, np.minimum(box.evaluate_points(q), np.sqrt(ref) - 0.02))
    r = np.sqrt(ref) - 0.02
    r = np.where(np.arange(len(q)) % 3 == 0, np.nextafter(r, np.inf), np.where(np.arange(len(q)) % 3 == 1, np.nextafter(r, -np.inf), r))
    r = np.maximum(r, 0.0)
    assert np.array_equal(sdf.is_outside_points(q, r).astype(bool), np.sqrt(ref) - 0.02 > r)


def test_nearest_non_finite_and_empty():
    sdf = CloudSDF(np.array([[0.0, 0.0, 0.0]]), 0.0)
    q = np.array([[np.nan, 0, 0], [np.inf, 0, 0], [0, -np.inf, 1], [0.5, 0, 0]])
    sq, at = sdf.nearest(q)
    assert np.isinf(sq[:3]).all() and np.isnan(at[:3]).all()
    assert sq[3] == 0.25 and np.array_equal(at[3], np.zeros(3))
