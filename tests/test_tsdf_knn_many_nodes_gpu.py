"""afx_tsdf_knn over more nodes than fit in 24 bits: the supporters of every voxel are those of the same nodes alone,
with their numbers shifted, on both sides of 2^24."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("k", [4, 8])
@pytest.mark.parametrize("total", [1 << 24, (1 << 24) + 25])
def test_node_numbers(total, k):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(k)
    dims, m = (17, 16, 15), 40
    size = tuple(F(0.01) * F(d) for d in dims)
    vs = tuple(F(s) / F(d) for s, d in zip(size, dims))
    near = (rng.uniform(-0.5, 0.5, (m, 3)) * np.array(size)).astype(F)
    near[m // 2:m // 2 + 4] = near[:4]  # equal distances: by node
    radii = np.full(m, 0.02, F)
    per = np.full(3, 5, np.int32)
    nodes = torch.full((total, 3), 1.0e3, device="cuda")  # in no voxel's reach
    nodes[-m:] = torch.from_numpy(near).cuda()
    S = int(np.prod(dims))
    idx = torch.empty((S, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((S, k), device="cuda")
    cnt = torch.empty(S, dtype=torch.int32, device="cuda")
    af.runTsdfKNNGraph(idx, dist, cnt, nodes, torch.full((total,), 0.02, device="cuda"), total, vs, size, dims, per)
    oi, od, oc = O.tsdf_knn(near, radii, vs, size, dims, per, k)
    oi, od, oc = np.asarray(oi).reshape(S, k).astype(np.int64), np.asarray(od).reshape(S, k), np.asarray(oc).ravel()
    c = cnt.cpu().numpy()
    assert np.array_equal(c, oc) and c.max() > 2
    have = np.arange(k)[None] < c[:, None]
    assert np.array_equal(idx.cpu().numpy()[have], oi[have] + total - m)
    assert np.array_equal(dist.cpu().numpy()[have], od[have])
