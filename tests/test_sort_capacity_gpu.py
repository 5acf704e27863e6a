"""Sort and unique of clouds much smaller than their room, where most passes have nothing to do, called and as a captured graph
that is replayed for other counts: the points against numpy's, and nothing written past the count."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CAP = 300000
COUNTS = (0, 1, 2048, 2049, 5000, 40000, 299999, CAP, 7)


def cloud(n):
    rng = np.random.default_rng(n)
    p = np.round(rng.normal(size=(CAP, 3)) * 40).astype(np.float32) / 16 + np.float32(0)  # no negative zeros
    p[:n // 3] = p[n // 2:n // 2 + n // 3]
    return p


def expected(p, n):
    return np.unique(p[:n], axis=0) if n else p[:0]  # in lexicographic order


def check(pts, cnt, p, n):
    want = expected(p, n)
    assert int(cnt.item()) == len(want)
    got = pts.cpu().numpy()
    assert np.array_equal(got[:len(want)], want) and np.array_equal(got[n:], p[n:])


def test_small_clouds_in_a_large_room():
    from volumefusion_gb300 import af
    for n in COUNTS:
        p = cloud(n)
        pts, cnt = torch.from_numpy(p.copy()).cuda(), torch.tensor([n], dtype=torch.int32, device="cuda")
        af.sortUnique(pts, cnt)
        check(pts, cnt, p, n)


def test_captured():
    from volumefusion_gb300._lib import lib
    L = lib()
    pts, cnt = torch.zeros((CAP, 3), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(L.afx_sort_unique_points_workspace_size(CAP), dtype=torch.uint8, device="cuda")

    def call():
        assert L.afx_sort_unique_points(pts.data_ptr(), cnt.data_ptr(), CAP, ws.data_ptr(), ws.numel(),
                                        torch.cuda.current_stream().cuda_stream) == 0
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    for n in COUNTS:
        p = cloud(n)
        pts.copy_(torch.from_numpy(p))
        cnt.fill_(n)
        g.replay()
        torch.cuda.synchronize()
        check(pts, cnt, p, n)
