"""afx_build_graph of clouds with more cells than fit in shared memory and more new nodes than shorten their ways up
there, in the cloud's order and in none, empty and grown: nodes, order and copied transforms against the oracle's
sequential walk, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402
from test_graph_build_gpu import _build, _sorted  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,radius", [(14000, 0.016), (40000, 0.0075)])
@pytest.mark.parametrize("order", ["sorted", "none"])
def test_large_graph_equals_sequential_walk(points, radius, order):
    rng = np.random.default_rng(points)
    cloud = (rng.random((points, 3)) * [1.0, 1.0, 0.001]).astype(np.float32)
    if order == "sorted":
        cloud = _sorted(cloud)
    radius = float(np.float32(radius))
    no, ro, To = O.build_graph(cloud, 4, radius)
    assert len(no) > (8192 if points == 40000 else 1800)
    n, r, T = _build(cloud, radius, len(no) + 10)
    assert np.array_equal(n, no) and np.array_equal(r, ro) and np.array_equal(T, To)
    # half the nodes there before, with transforms of their own, one of them met at no distance
    half = len(no) // 2
    T0 = rng.standard_normal((half, 16)).astype(np.float32)
    more = np.ascontiguousarray(np.concatenate([no[half:], cloud[::3] + np.float32([0.0, 1.01, 0.0])]))
    n2o, _, T2o = O.build_graph(more, 4, radius, no[:half], ro[:half], T0, cap=40000)
    n2, _, T2 = _build(more, radius, len(n2o) + 1, no[:half], T0)
    assert np.array_equal(n2, n2o) and np.array_equal(T2, T2o)
