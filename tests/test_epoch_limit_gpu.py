"""Sessions that clear their collision counts within a sequence, at a reset, or both, end with the same volumes, graphs and
statistics as one that never does; alone and as members of a batch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from volumefusion_gb300 import configs  # noqa: E402

pytestmark = pytest.mark.gpu


def run(s, frames, process):
    out = []
    for _ in range(2):  # two sequences
        s.reset()
        for f in frames:
            process(f)
        out += [*s.tsdf(), *s.graph()]
    return out


@pytest.mark.parametrize("batch", [False, True])
def test_counts_cleared_between_frames(batch):
    from volumefusion_gb300._lib import lib
    from volumefusion_gb300.batch import Batch
    from volumefusion_gb300.fusion import FusionSession
    cfg = configs.small_nonrigid(n_frames=8)
    frames = [torch.from_numpy(m.astype(np.int16)).cuda() for m in configs.small_frames(cfg)]
    want = None
    for limit in (None, 1, 2, 5):
        s = FusionSession(cfg)
        if limit is not None:
            assert lib().afx_fusion_set_epoch_limit(s.h, limit) == 0
        b = Batch([s]) if batch else None
        got = run(s, frames, (lambda f: b.process([f])) if batch else s.process)
        if want is None:
            want = got
        assert bool(want[1].any()) and all(torch.equal(x, y) for x, y in zip(got, want)), limit
        if b is not None:
            b.close()
        s.close()


def test_limits_that_do_not_fit_are_refused():
    from volumefusion_gb300._lib import lib
    from volumefusion_gb300.fusion import FusionSession
    s = FusionSession(configs.small_nonrigid(n_frames=2))
    for limit in (0, -1, 1 << 24):
        assert lib().afx_fusion_set_epoch_limit(s.h, limit) == 1
    assert lib().afx_fusion_set_epoch_limit(s.h, (1 << 24) - 1) == 0
    s.close()
