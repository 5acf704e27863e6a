"""The marching-cubes sweep and the general sort + unique at the edges of their tiles, against the oracle:
volumes that end inside a warp's columns, rows or slices, with holes in the weights and surface in most
cubes (the queues fill and empty), and clouds around the sort's tile, its merge passes and a capacity
that allows for more of them.  Vertices and triangles as multisets, sorted clouds bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _rows(a):
    a = np.ascontiguousarray(a)
    return a[np.lexsort(a.T[::-1])]


@pytest.mark.parametrize("dims", [(3, 3, 3), (33, 6, 18), (34, 7, 19), (32, 35, 17), (65, 34, 35), (130, 70, 4)])
def test_sweep_equals_oracle(dims):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(sum(dims))
    S = int(np.prod(dims))
    t = rng.uniform(-1, 1, S).astype(np.float32)
    t[rng.random(S) < 0.02] = 0.0
    w = rng.integers(1, 4, S).astype(np.float32)
    w[rng.random(S) < 0.03] = 0.0
    w = w.reshape(dims[::-1])
    w[:, : dims[1] // 4] = 0.0  # rows without any weight
    w = np.ascontiguousarray(w.ravel())
    size = tuple(0.01 * d for d in dims)
    vs = np.array(size, np.float32) / np.array(dims, np.float32)
    size = np.array(size, np.float32)
    pc = O.mc_pointcloud(t, w, dims, vs, size, cap=15 * S)  # room for every edge and corner of every cube
    v, f = O.mc_full(t, w, dims, vs, size, cap=15 * S)
    dt, dw = torch.from_numpy(t).cuda(), torch.from_numpy(w).cuda()
    pts = torch.zeros((len(pc) + 5, 3), device="cuda")
    cnt, nv, nf = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(3))
    af.runMarchingCubesMeshKernel(pts, cnt, dt, dw, dims, vs, size)
    assert int(cnt.item()) == len(pc)
    assert np.array_equal(_rows(pts[:len(pc)].cpu().numpy()), _rows(pc))
    mv = torch.zeros((len(v) + 3, 3), device="cuda")
    mf = torch.zeros((len(f) + 1, 3), dtype=torch.int32, device="cuda")
    af.runMarchingCubesFullKernel(mv, nv, mf, nf, dt, dw, dims, vs, size)
    assert int(nf.item()) == len(f) and int(nv.item()) == len(v)
    assert np.array_equal(_rows(mv[:len(v)].cpu().numpy().reshape(-1, 9)), _rows(v.reshape(-1, 9)))


@pytest.mark.parametrize("n,cap", [(1, 1), (2, 5000), (2047, 2047), (2048, 2048), (2049, 2049), (4096, 300000), (6145, 6145),
                                   (70001, 70001), (330000, 330000), (200000, 1100000)])
def test_general_sort_unique(n, cap):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(n)
    p = rng.integers(-40, 40, (n, 3)).astype(np.float32) * np.float32(0.25)  # many ties in x and y, repeats
    p[rng.random(n) < 0.3] *= np.float32(1.0 / 3.0)
    p[p == 0] *= rng.choice(np.array([-1.0, 1.0], np.float32), int((p == 0).sum()))  # both zeros
    d = torch.zeros((cap, 3), device="cuda")
    d[:n] = torch.from_numpy(p).cuda()
    cnt = torch.tensor([n], dtype=torch.int32, device="cuda")
    af.sortUnique(d, cnt)
    # the sort's order is total: -0 before +0 in a coordinate, whatever the later ones are; unique goes by
    # equality of consecutive points, for which the two zeros are equal
    u = p.view(np.uint32)
    key = np.where(u & 0x80000000, ~u, u | 0x80000000)
    q = p[np.lexsort((key[:, 2], key[:, 1], key[:, 0]))]
    expect = q[np.concatenate([[True], (q[1:] != q[:-1]).any(1)])]
    m = int(cnt.item())
    assert m == len(expect)
    assert np.array_equal(d[:m].cpu().numpy().view(np.uint32), expect.view(np.uint32))
