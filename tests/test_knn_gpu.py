"""K nearest nodes over the cases of the search: few and many queries (sorted as a cloud is, and in no order),
fewer nodes than neighbours, more than fit in shared memory; surfaces, volumes, lattices whose distances tie,
isolated clusters, far and non-finite queries, nodes that are not finite or all in one place.  Lists and distances are compared bit for
bit with every binary32 distance ordered by (distance, index); for distances that are NaN, with the
insertion in index order that defines them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
F = np.float32


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def distances(q, nodes):
    with np.errstate(all="ignore"):
        d = (q[:, None, :] - nodes[None, :, :]).astype(F)
        d = d * d
        return (d[..., 0] + d[..., 1]) + d[..., 2]


def inserted(d, k):
    best = []
    for j, v in enumerate(d):
        if len(best) == k:
            if not v < best[-1][0]:
                continue
            best.pop()
        p = len(best)
        while p > 0 and v < best[p - 1][0]:
            p -= 1
        best.insert(p, (v, j))
    return best


def reference(q, nodes, k, excl):
    kk = k + int(excl)
    idx = np.full((len(q), kk), 0xFFFFFFFF, np.uint32)
    dist = np.full((len(q), kk), np.finfo(F).max, F)
    for a in range(0, len(q), 512):
        D = distances(q[a:a + 512], nodes)
        kth = np.partition(D, min(kk, len(nodes)) - 1, axis=1)[:, min(kk, len(nodes)) - 1]
        for r in range(len(D)):
            if np.isnan(D[r]).any():
                best = inserted(D[r], kk)
            else:
                near = np.nonzero(D[r] <= kth[r])[0]
                near = near[np.argsort(D[r, near], kind="stable")[:kk]]
                best = [(D[r, j], j) for j in near]
            for s, (v, j) in enumerate(best):
                idx[a + r, s], dist[a + r, s] = j, np.sqrt(F(v))
    return idx[:, int(excl):], dist[:, int(excl):]


def cloud(kind, n, rng):
    if kind == "surface":
        p = rng.normal(size=(n, 3))
        return (0.4 * p / np.linalg.norm(p, axis=1, keepdims=True) + [0.1, -0.2, 0.9]).astype(F)
    if kind == "volume":
        return rng.uniform(-1, 1, (n, 3)).astype(F)
    if kind == "tube":  # long in x, as a window pays for
        a = rng.uniform(0, 2 * np.pi, n)
        return np.stack([rng.uniform(-0.5, 0.5, n), 0.05 * np.cos(a), 0.8 + 0.05 * np.sin(a)], 1).astype(F)
    if kind == "line":
        return np.stack([rng.uniform(0, 3, n), np.full(n, 0.5), np.full(n, -2.0)], 1).astype(F)
    if kind == "lattice":
        m = int(np.ceil(n ** (1 / 3)))
        return (np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * 0.25).astype(F)
    if kind == "clusters":  # three nodes far from the others
        p = cloud("surface", n, rng)
        p[:3] = np.array([[30, 30, 30], [30.01, 30, 30], [30, 30.02, 30]], F)
        return p
    return np.tile(np.array([[0.3, 0.2, 0.1]], F), (n, 1))  # "point"


CASES = [("surface", n, k, e, 0) for n, k, e in [(1, 4, False), (5, 4, True), (128, 4, False), (700, 6, False),
                                                (5000, 8, True), (12544, 4, False), (13000, 3, False)]]
CASES += [("volume", 3000, 8, True, 0), ("volume", 2000, 16, True, 0), ("line", 400, 4, False, 0), ("lattice", 1000, 8, True, 0),
          ("clusters", 2000, 4, False, 0), ("point", 300, 4, False, 0), ("surface", 900, 1, False, 0)]
CASES += [(kind, n, k, False, m) for kind, n, k, m in [("surface", 3, 4, 8300), ("surface", 129, 4, 8193), ("surface", 7100, 4, 8200), ("tube", 1500, 4, 9000), ("tube", 300, 8, 8300), ("tube", 12544, 3, 8200), ("surface", 128, 9, 8200), ("surface", 4000, 8, 9000),
                                                       ("surface", 12544, 4, 8200), ("surface", 12545, 2, 8200),
                                                       ("volume", 1500, 6, 8500), ("line", 500, 4, 8500), ("lattice", 1000, 4, 8500),
                                                       ("clusters", 800, 4, 8500), ("point", 40, 4, 8500), ("line", 300, 16, 8300)]]


@pytest.mark.parametrize("kind,n,k,excl,many", CASES)
def test_knn(kind, n, k, excl, many):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(n * 31 + k)
    nodes = cloud(kind, n, rng)
    count = many or 700
    near = nodes[rng.integers(0, n, count)] + rng.normal(0, 0.01, (count, 3)).astype(F)
    if many:  # the first half sorted as point clouds are
        half = near[:count // 2]
        near[:count // 2] = half[np.lexsort(half.T[::-1])]
    far = rng.uniform(-40, 40, (60, 3)).astype(F)
    odd = np.array([[np.nan, 0, 0], [np.inf, 0, 0], [0, -np.inf, np.nan], [3e38, 0, 0], [1e20, 1e20, -1e20]], F)
    q = nodes if excl else np.concatenate([near, far, odd]).astype(F)
    idx = torch.empty((len(q), k), dtype=torch.int32, device="cuda")
    dist = torch.empty((len(q), k), device="cuda")
    cap = np.concatenate([nodes, np.zeros((7, 3), F)])  # room after the nodes, as callers have it
    af.getKnnData(idx, dist, cu(cap), cu(np.array([n], np.int32)), cu(q), excludeClosest=excl)
    ri, rd = reference(q, nodes, k, excl)
    assert np.array_equal(idx.cpu().numpy().view(np.uint32), ri)
    assert np.array_equal(dist.cpu().numpy(), rd, equal_nan=True)


@pytest.mark.parametrize("many", [1, 140])
@pytest.mark.parametrize("value", [np.nan, np.inf, 3e38])
def test_knn_with_nodes_that_are_not_ordinary(value, many):
    from volumefusion_gb300 import af
    rng = np.random.default_rng(3)
    nodes = cloud("surface", 400, rng)
    nodes[[2, 250, 399]] = F(value)
    q = np.tile(nodes[:64] + F(0.003), (many, 1))
    idx = torch.empty((len(q), 4), dtype=torch.int32, device="cuda")
    dist = torch.empty((len(q), 4), device="cuda")
    af.getKnnData(idx, dist, cu(nodes), cu(np.array([400], np.int32)), cu(q))
    ri, rd = reference(q, nodes, 4, False)
    assert np.array_equal(idx.cpu().numpy().view(np.uint32), ri)
    assert np.array_equal(dist.cpu().numpy(), rd, equal_nan=True)
