"""The volume copied out as FP32 in both storage formats, for voxel counts that are and are not multiples of the four a
thread takes, and a reset: an empty volume again, and the same results from collision words that an earlier
sequence has left."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from volumefusion_gb300 import configs  # noqa: E402

pytestmark = pytest.mark.gpu


def session(dims, precision):
    from volumefusion_gb300.fusion import FusionSession
    cfg = configs.small_nonrigid(n_frames=6)
    voxel = cfg["volume_size"][0] / cfg["dims"][0]
    cfg.update(dims=dims, volume_size=tuple(voxel * d for d in dims), precision=precision)
    return FusionSession(cfg), cfg


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("dims", [(64, 64, 64), (63, 61, 59), (65, 33, 31)])
def test_export_and_reset(dims, precision):
    s, cfg = session(dims, precision)
    from volumefusion_gb300 import synth
    cam = dict(width=cfg["width"], height=cfg["height"], fx=float(cfg["K"][0, 0]), fy=float(cfg["K"][1, 1]),
               cx=float(cfg["K"][0, 2]), cy=float(cfg["K"][1, 2]))
    frames = [torch.from_numpy(synth.capsule_pair_frame(10 + f, **cam)[0].astype(np.int16)).cuda() for f in range(5)]

    def sequence():
        s.reset()
        t, w = s.tsdf()
        assert bool((t == -1).all()) and not bool(w.any())
        for f in frames:
            s.process(f)
        return s.tsdf()

    t, w = sequence()
    rt, rw, _ = s.volume_raw()
    assert torch.equal(t, rt.float()) and torch.equal(w, rw.float()) and bool(w.any())
    for _ in range(2):
        t2, w2 = sequence()
        assert torch.equal(t, t2) and torch.equal(w, w2)
    s.close()
