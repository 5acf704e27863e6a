"""Rigid integration against the oracle where leaving out blocks could go wrong: the camera inside, beside,
behind and at the edge of the volume, blocks that span more pixels than are looked at, ragged volumes,
frames without a valid pixel or with infinities and not-a-numbers.  Volumes bit for bit, integrated
into and initialised + integrated in one pass."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _rot(axis, deg):
    a = np.radians(deg)
    c, s = np.cos(a), np.sin(a)
    m = {"x": [[1, 0, 0], [0, c, -s], [0, s, c]], "y": [[c, 0, s], [0, 1, 0], [-s, 0, c]], "z": [[c, -s, 0], [s, c, 0], [0, 0, 1]]}
    return np.array(m[axis], np.float32)


def _depth(name, w, h, rng):
    y, x = np.mgrid[0:h, 0:w]
    d = (0.7 + 0.1 * np.sin(x * 0.07) + 0.05 * np.cos(y * 0.11)).astype(np.float32)
    if name == "object":  # a disc, nothing around it
        d[(x - w / 2) ** 2 + (y - h / 2) ** 2 > (h / 4) ** 2] = np.inf
    elif name == "odd":
        r = rng.random((h, w))
        d[r < 0.2] = np.inf
        d[(r > 0.2) & (r < 0.22)] = np.nan
        d[(r > 0.22) & (r < 0.24)] = -0.5
        d[(r > 0.24) & (r < 0.26)] = 5e-5
        d[(r > 0.26) & (r < 0.28)] = -np.inf
    elif name == "empty":
        d[:] = np.inf
    return d


@pytest.mark.parametrize("depth", ["wall", "object", "odd", "empty"])
@pytest.mark.parametrize("dims,edge,center,rot", [
    ((64, 48, 33), 0.5, (0.0, 0.0, 0.7), ("y", 20)),     # in front, ragged
    ((40, 40, 40), 2.0, (0.1, 0.0, 0.3), ("x", -35)),    # the camera inside
    ((65, 34, 50), 0.6, (0.0, 0.1, -0.1), ("z", 10)),    # around the camera plane, rows of an odd length
    ((32, 32, 32), 0.4, (0.0, 0.0, -0.8), ("y", 5)),     # behind
    ((64, 64, 64), 0.5, (0.9, -0.6, 0.8), ("y", 60)),    # at the edge of the image
    ((36, 20, 20), 3.0, (0.0, 0.0, 2.0), ("x", 15)),     # blocks over most of the image
])
def test_integration_with_blocks_left_out(depth, dims, edge, center, rot):
    from volumefusion_gb300 import af
    from volumefusion_gb300._lib import check, lib
    rng = np.random.default_rng(7)
    w, h = 200, 150
    K = np.array([[160.0, 0, 101.3], [0, 158.0, 74.6], [0, 0, 1]])
    d = _depth(depth, w, h, rng)
    size = np.array([edge * v / max(dims) for v in dims], np.float32)
    vs = size / np.array(dims, np.float32)
    R, t = _rot(*rot), np.array(center, np.float32)
    delta = float(np.float32(2.5 * vs.max()))
    S = int(np.prod(dims))
    t0, w0 = rng.uniform(-1, 1, S).astype(np.float32), rng.integers(0, 16, S).astype(np.float32)
    to, wo = t0.copy(), w0.copy()
    O.integrate_rigid(to, wo, d, delta, dims, vs, size, R, t, K)
    dt, dw, dd = (torch.from_numpy(a.copy()).cuda() for a in (t0, w0, d))
    af.runIntegrateTSDFFromFrameKernel(dt, dw, dd, (w, h), delta, dims, vs, size, R, t, K)
    assert np.array_equal(dt.cpu().numpy(), to, equal_nan=True)  # the bits of a NaN are the processor's
    assert np.array_equal(dw.cpu().numpy(), wo)
    if dims[0] % 4:
        return
    tf, wf = np.full(S, -1.0, np.float32), np.zeros(S, np.float32)
    O.integrate_rigid(tf, wf, d, delta, dims, vs, size, R, t, K)
    f = lambda a: (C.c_float * len(a))(*[float(x) for x in a])  # noqa: E731
    col = lambda m: f(np.asarray(m, np.float64).T.ravel())  # noqa: E731
    dt.fill_(7.0)
    dw.fill_(7.0)
    check(lib().afx_integrate_tsdf_fresh(C.c_void_p(dt.data_ptr()), C.c_void_p(dw.data_ptr()), C.c_void_p(dd.data_ptr()), w, h,
                                         C.c_float(delta), (C.c_int * 3)(*dims), f(vs), f(size), col(R), f(t), col(K),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)), "fresh")
    assert np.array_equal(dt.cpu().numpy(), tf, equal_nan=True) and np.array_equal(dw.cpu().numpy(), wf)
