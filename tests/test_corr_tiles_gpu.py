"""Correspondence pairs at the sizes where their compaction can go wrong: around one tile of 256 vertices, more
tiles than CTAs, no vertex with a pixel and all of them, a capacity below their number.  Compared with the
oracle's pairs, which are in vertex order too."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def frame(rng, h=60, w=80):
    K = np.array([[70.0, 0, 40.0], [0, 70.0, 30.0], [0, 0, 1.0]])
    depth = rng.uniform(0.7, 0.9, (h, w)).astype(np.float32)
    depth[rng.random((h, w)) < 0.2] = np.inf
    v, u = np.mgrid[0:h, 0:w]
    z = np.where(np.isfinite(depth), depth, 0).astype(np.float32)
    verts = np.stack([(u - 40.0) / 70.0 * z, (v - 30.0) / 70.0 * z, z], -1).astype(np.float32)
    return K, depth, verts


@pytest.mark.parametrize("m,near", [(1, 0.7), (255, 0.7), (256, 1.0), (257, 0.0), (511, 0.5), (77824, 0.6), (77825, 0.6), (160001, 0.3)])
def test_pairs(m, near):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(m)
    K, depth, verts = frame(rng)
    ok = verts[np.isfinite(depth)]
    pts = ok[rng.integers(0, len(ok), m)] + np.where(rng.random((m, 1)) < near, 0.001, 0.5).astype(np.float32)
    pts = pts.astype(np.float32)
    want = O.correspondences(pts, K, depth, verts, 0.01)
    cap = m if m != 511 else max(1, len(want) // 2)
    corr = torch.full((cap, 2), -7, dtype=torch.int32, device="cuda")
    n = torch.full((1,), 99, dtype=torch.int32, device="cuda")
    af.runCorrespondencePairsKernel(corr, n, cu(pts), m, K, cu(depth), depth.shape, cu(verts), 0.01)
    assert int(n.item()) == len(want)
    got = corr.cpu().numpy()
    assert np.array_equal(got[:len(want)], want[:cap])
    assert (got[len(want):] == -7).all()
