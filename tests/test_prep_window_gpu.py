"""Frame pre-processing over filter radii (unrolled ones, others and none) and image sizes around a tile, with windows that
the border clamps, invalid pixels among valid ones and depth steps past the filter's threshold: bit for bit
against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [0, 1, 2, 3, 4, 7])
@pytest.mark.parametrize("w,h", [(8, 5), (33, 17), (40, 34), (64, 48), (97, 50)])
def test_frame(radius, w, h):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(radius * 100 + w)
    v, u = np.mgrid[0:h, 0:w]
    mm = 700 + 3 * np.abs(u - w / 2) + 2 * v + rng.normal(0, 6, (h, w))
    mm = np.where(u > 0.7 * w, mm + 200, mm)  # a step past the threshold
    mm[rng.random((h, w)) < 0.07] = 0
    mm = mm.clip(0, 2000).astype(np.uint16)
    K = np.array([[100.0, 0, w / 2.0], [0, 100.0, h / 2.0], [0, 0, 1.0]])
    want = O.frame_prep(mm, K, r=radius)
    got = af.loadProcessFrame(torch.from_numpy(mm.astype(np.int16)).cuda(), K, bilateral_r=radius)
    for a, b in zip(got[:3], want[:3]):
        assert np.array_equal(a.cpu().numpy(), b, equal_nan=True)
