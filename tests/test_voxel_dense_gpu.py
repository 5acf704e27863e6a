"""The dense per-voxel kernels at the sizes of their splits: rows of a multiple of four voxels and others, volumes
around the 128 voxels a warp takes, and arrays that start on 16 bytes or do not.  Voxel centres against their
formula in binary32; the warp, weights, collisions and integration of sparse counts against numpy or the other path,
bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
F = np.float32


def cu(a, offset=0):
    """On the GPU, `offset` elements after a 16-byte boundary."""
    a = np.ascontiguousarray(a)
    buf = torch.empty(a.size + offset, dtype=torch.from_numpy(a).dtype, device="cuda")
    out = buf[offset:].view(a.shape)
    out.copy_(torch.from_numpy(a))
    return out


@pytest.mark.parametrize("dims", [(4, 1, 1), (1, 1, 1), (3, 5, 2), (8, 7, 9), (64, 5, 3), (66, 5, 3), (132, 17, 2)])
@pytest.mark.parametrize("offset", [0, 1])
def test_vertices(dims, offset):
    from volumefusion_gb300 import af
    size = tuple(F(0.013) * d for d in dims)
    vs = tuple(F(s) / F(d) for s, d in zip(size, dims))
    S = int(np.prod(dims))
    v = cu(np.full((S, 3), 7, F), offset)
    af.runGenerateTsdfVerticesKernel(v, vs, size, dims)
    ax = [np.arange(d, dtype=F) * x - F(s) * F(0.5) for d, x, s in zip(dims, vs, size)]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    assert np.array_equal(v.cpu().numpy(), np.stack([x, y, z], -1).reshape(-1, 3))


@pytest.mark.parametrize("S", [1, 127, 128, 129, 1024, 1025, 70001])
@pytest.mark.parametrize("k", [4, 6])
def test_weights_and_warp(S, k):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(S + k)
    n = 40
    cnt = np.where(rng.random(S) < 0.3, rng.integers(1, k + 1, S), 0).astype(np.int32)
    idx = rng.integers(0, n, (S, k)).astype(np.int32)
    idx[np.arange(k)[None] >= cnt[:, None]] = -1
    dist = rng.uniform(0, 0.04, (S, k)).astype(F)
    radii = rng.uniform(0.01, 0.03, n).astype(F)
    T = np.tile(np.eye(4, dtype=F).reshape(-1), (n, 1)) + rng.normal(0, 0.01, (n, 16)).astype(F)
    verts = rng.normal(size=(S, 3)).astype(F)
    out = []
    for offset in (0, 1):
        w = cu(np.full((S, k), 3, F), offset)
        v = cu(verts, offset)
        c, i = cu(cnt, offset), cu(idx, offset)
        af.runComputeTsdfWarpWeightsKernel(w, cu(radii), i, cu(dist, offset), c, S)
        w[torch.from_numpy(rng.random(S) < 0.05).cuda()] = 0.0
        if out:
            w.copy_(torch.from_numpy(out[0][0]))
        af.runWarpTsdfKernel(v, cu(T, offset), i, w, c, None, None, (S, 1, 1))
        out.append((w.cpu().numpy(), v.cpu().numpy()))
    assert np.array_equal(out[0][1], out[1][1])
    w, v = out[0]
    assert (w[(cnt == 0) & (w != 0).all(1)] == 3).all()
    zero = (np.abs(w) <= F(1e-5)).all(1) | (cnt == 0)
    q = np.zeros((S, 3), F)
    for s in range(k):
        M = T[np.maximum(idx[:, s], 0)].reshape(-1, 4, 4)
        o = ((M[:, 0, :3] * verts[:, :1] + M[:, 1, :3] * verts[:, 1:2]) + M[:, 2, :3] * verts[:, 2:]) + M[:, 3, :3]
        q = np.where((s < cnt)[:, None], q + w[:, s:s + 1] * o, q)
    assert np.array_equal(v, np.where(zero[:, None], verts, q))


@pytest.mark.parametrize("dims", [(1, 1, 1), (127, 1, 1), (128, 1, 1), (43, 3, 1), (64, 16, 1), (41, 25, 1), (50, 40, 30)])
def test_collisions(dims):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(dims[0])
    S = int(np.prod(dims))
    size = tuple(F(0.01) * F(d) for d in dims)
    vs = tuple(F(s) / F(d) for s, d in zip(size, dims))
    cnt = (rng.random(S) < 0.3).astype(np.int32)
    target = rng.integers(-1, max(S // 3, 1), S)  # several voxels to a target; -1: outside
    t = np.maximum(target, 0)
    cell = np.stack([t % dims[0], (t // dims[0]) % dims[1], t // (dims[0] * dims[1])], -1)
    verts = ((cell + 0.5) * np.array(vs, np.float64) - 0.5 * np.array(size, np.float64)).astype(F)
    verts[target < 0] = 9.0
    counts = torch.zeros(S, dtype=torch.int32, device="cuda")
    af.runCountCollisionsPerVoxelKernel(counts, cu(verts), cu(cnt), vs, size, dims, np.eye(3), (0.0, 0.0, 0.0))
    want = np.bincount(target[(target >= 0) & (cnt > 0)], minlength=S)
    assert np.array_equal(counts.cpu().numpy(), want)


@pytest.mark.parametrize("dims,n,k,lattice", [((8, 8, 8), 1, 4, False), ((9, 7, 17), 30, 3, False), ((24, 16, 8), 190, 8, False),
                                              ((16, 16, 16), 125, 4, True), ((20, 9, 12), 60, 1, True), ((16, 8, 8), 40, 6, False)])
def test_supporters(dims, n, k, lattice):
    """More supporters than k, equal distances (by node), up to the number of nodes a brick holds."""
    from volumefusion_gb300 import af
    rng = np.random.default_rng(n + k)
    size = tuple(F(0.01) * F(d) for d in dims)
    vs = tuple(F(s) / F(d) for s, d in zip(size, dims))
    half = np.array([F(s) * F(0.5) for s in size], F)
    if lattice:
        m = int(round(n ** (1 / 3)) + 1)
        grid = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        nodes = (grid * F(0.02) + np.array(vs, F) - half).astype(F)
    else:
        nodes = (rng.uniform(-0.6, 0.6, (n, 3)) * np.array(size)).astype(F)
    radii = rng.uniform(0.012, 0.03, n).astype(F) if not lattice else np.full(n, 0.02, F)
    per = np.array([2 * (int(F(0.02) / v) + 1) + 1 for v in vs], np.int32)
    S = int(np.prod(dims))
    idx = torch.empty((S, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((S, k), device="cuda")
    cnt = torch.empty(S, dtype=torch.int32, device="cuda")
    af.runTsdfKNNGraph(idx, dist, cnt, cu(nodes), cu(radii), n, vs, size, dims, per)
    ax = [np.arange(d, dtype=F) * v - h for d, v, h in zip(dims, vs, half)]
    z, y, x = np.meshgrid(*[np.arange(d) for d in (dims[2], dims[1], dims[0])], indexing="ij")
    vox = np.stack([x, y, z], -1).reshape(-1, 3)
    p = np.stack([ax[c][vox[:, c]] for c in range(3)], -1)
    inv = np.array([F(1.0 / float(v)) for v in vs], F)
    base = np.trunc((nodes + half) * inv).astype(np.int64)
    lo = base - (per - 1) // 2
    D = np.full((S, n), np.inf, F)
    for j in range(n):
        d = p - nodes[j]
        r = np.sqrt(d[:, 0] * d[:, 0] + (d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]))
        ok = ((vox >= lo[j]) & (vox <= lo[j] + per - 1)).all(1) & ~(r > radii[j] * F(2))
        D[ok, j] = r[ok]
    order = np.argsort(D, axis=1, kind="stable")[:, :k]
    want_d = np.take_along_axis(D, order, 1)
    have = np.isfinite(want_d)
    c = np.minimum(np.isfinite(D).sum(1), k)
    assert np.array_equal(cnt.cpu().numpy(), c)
    gi, gd = idx.cpu().numpy(), dist.cpu().numpy()
    assert np.array_equal(gi[:, :order.shape[1]][have], order[have]) and np.array_equal(gd[:, :order.shape[1]][have], want_d[have])
