"""Rigid integration against the oracle on both sides of the volumes where its blocks change depth, with rows of a multiple
of four voxels and others, in FP32: a scene around the camera (most voxels change) and an object (most blocks are left
out), into a used volume and into a fresh one, bit for bit."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402
from test_integrate_blocks_gpu import _rot  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["room", "object"])
@pytest.mark.parametrize("dims", [(216, 216, 214), (216, 216, 215), (217, 215, 214), (217, 215, 215),  # 10^7 voxels
                                  (272, 272, 270), (272, 272, 271), (273, 271, 270), (273, 271, 271)])  # 2 10^7
def test_integration_over_volume_sizes(dims, scene):
    from volumefusion_gb300 import af
    from volumefusion_gb300._lib import check, lib
    w, h = 320, 240
    K = np.array([[250.0, 0, 160.2], [0, 251.0, 119.6], [0, 0, 1]])
    y, x = np.mgrid[0:h, 0:w]
    d = (0.75 + 0.08 * np.sin(x * 0.05) + 0.05 * np.cos(y * 0.07)).astype(np.float32)
    if scene == "object":
        d[(x - 150) ** 2 + (y - 130) ** 2 > 45 ** 2] = np.inf
    size = np.array([1.0 * v / max(dims) for v in dims], np.float32)
    vs = size / np.array(dims, np.float32)
    R, t = _rot("y", 15), np.array([0.02, -0.01, 0.8 if scene == "object" else 0.5], np.float32)
    delta = float(np.float32(3 * vs.max()))
    S = int(np.prod(dims))
    rng = np.random.default_rng(1)
    t0, w0 = rng.uniform(-1, 1, S).astype(np.float32), rng.integers(0, 16, S).astype(np.float32)
    dt, dw, dd = (torch.from_numpy(a.copy()).cuda() for a in (t0, w0, d))
    af.runIntegrateTSDFFromFrameKernel(dt, dw, dd, (w, h), delta, dims, vs, size, R, t, K)
    O.integrate_rigid(t0, w0, d, delta, dims, vs, size, R, t, K)
    assert np.array_equal(dt.cpu().numpy(), t0) and np.array_equal(dw.cpu().numpy(), w0)
    if dims[0] % 4:
        return
    tf, wf = np.full(S, -1.0, np.float32), np.zeros(S, np.float32)
    O.integrate_rigid(tf, wf, d, delta, dims, vs, size, R, t, K)
    f = lambda a: (C.c_float * len(a))(*[float(v) for v in a])  # noqa: E731
    col = lambda m: f(np.asarray(m, np.float64).T.ravel())  # noqa: E731
    dt.fill_(7.0)
    dw.fill_(7.0)
    check(lib().afx_integrate_tsdf_fresh(dt.data_ptr(), dw.data_ptr(), dd.data_ptr(), w, h, delta, (C.c_int * 3)(*dims), f(vs),
                                         f(size), col(R), f(t), col(K), torch.cuda.current_stream().cuda_stream), "fresh")
    assert np.array_equal(dt.cpu().numpy(), tf) and np.array_equal(dw.cpu().numpy(), wf)
