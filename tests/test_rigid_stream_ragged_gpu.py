"""The rigid stream over volumes whose rows are no multiple of four voxels (no vector stores, no tile loads: brick marks
and marching cubes read from global memory) and over ones whose rows are, with surface across the edges of bricks and
of the sweep's 31 cubes: clouds and volumes against the oracle bit for bit, triangles as a multiset, two frames."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402
from test_rigid_stream_gpu import _pose, _rot, _tri_rows  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(63, 50, 41), (65, 34, 35), (33, 70, 31), (94, 41, 66), (41, 33, 130), (7, 90, 65), (64, 33, 65),
                                  (68, 50, 41), (3, 64, 64), (130, 130, 65)])
def test_rigid_stream_over_ragged_volumes(dims):
    from volumefusion_gb300 import configs
    from volumefusion_gb300.rigid_stream import RigidStream
    cfg = configs.small_nonrigid(n_frames=4)
    frames = configs.small_frames(cfg)
    K = np.asarray(cfg["K"], np.float32)
    H, W = cfg["height"], cfg["width"]
    c2w = [np.eye(4, dtype=np.float32), _pose(_rot("y", 20), [0.15, 0.0, 0.05])]
    _, _, _, cen = O.frame_prep(frames[0], K)
    center = np.asarray(cen, np.float32)
    R = _rot("z", 10).astype(np.float32)
    size = tuple(0.7 * d / max(dims) for d in dims)
    vs = np.array([np.float32(a) / np.float32(b) for a, b in zip(size, dims)], np.float32)
    delta = float(4 * vs.max())
    st = RigidStream([K, K], c2w, W, H, dims, size, delta, center, R)
    some = 0
    for step in range(2):
        mms = [frames[c + step] for c in range(2)]
        st.process([torch.from_numpy(m.astype(np.int16)).cuda() for m in mms])
        cloud, verts, faces, tsdf, weights = (x.cpu().numpy() for x in st.outputs())
        depths = [O.bilateral(O.filter_depth(O.depth_from_mm(mm), 1.2), 2, 0.03, 2.0, 0.09) for mm in mms]
        want = np.concatenate([O.transform_points(O.depth_to_mesh(d, K).reshape(-1, 3), T) for d, T in zip(depths, c2w)])
        assert np.array_equal(cloud, want, equal_nan=True)
        t0 = np.full(int(np.prod(dims)), -1.0, np.float32)
        w0 = np.zeros_like(t0)
        O.integrate_rigid(t0, w0, depths[0], delta, dims, vs, np.array(size, np.float32), R, center, K)
        assert np.array_equal(tsdf, t0) and np.array_equal(weights, w0)
        ev, ef = O.mc_full(t0, w0, dims, vs, size)
        assert len(verts) == len(ev) == 3 * len(faces.reshape(-1, 3))
        assert np.array_equal(_tri_rows(verts), _tri_rows(ev))
        some += len(ev)
    assert some > (500 if min(dims) > 3 else 0)
    st.close()
