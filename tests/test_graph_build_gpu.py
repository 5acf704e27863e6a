"""afx_build_graph against the oracle's sequential walk where the rounds can go wrong: tiny clouds, clouds
in no spatial order, long chains of nodes, crowded and repeated points, more cells than fit in shared
memory, a graph that grows, and the capacity limit.  Nodes, their order and the copied transforms are
the same bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def _build(cloud, radius, cap, nodes=None, T=None):
    from volumefusion_gb300 import af
    d_n = torch.zeros((cap, 3), device="cuda")
    d_r = torch.zeros(cap, device="cuda")
    d_T = torch.zeros((cap, 16), device="cuda")
    n0 = 0 if nodes is None else len(nodes)
    if n0:
        d_n[:n0] = torch.from_numpy(nodes).cuda()
        d_r[:n0] = radius
        d_T[:n0] = torch.from_numpy(T).cuda()
    nn = torch.tensor([n0], dtype=torch.int32, device="cuda")
    mesh = torch.from_numpy(cloud).cuda()
    af.buildGraph(d_n, d_r, d_T, nn, mesh, torch.tensor([len(cloud)], dtype=torch.int32, device="cuda"), 4, radius)
    n = int(nn.item())
    return d_n[:n].cpu().numpy(), d_r[:n].cpu().numpy(), d_T[:n].cpu().numpy()


def _sorted(p):
    return np.ascontiguousarray(p[np.lexsort(p.T[::-1])])


def _cloud(name):
    rng = np.random.default_rng(len(name))
    if name == "one":
        return rng.random((1, 3)), 0.1
    if name == "warp":
        return rng.random((33, 3)), 0.3
    if name == "unordered":
        return rng.random((20000, 3)) * [1.0, 0.5, 0.02], 0.04
    if name == "ordered":
        return _sorted((rng.random((30000, 3)) * [0.6, 0.3, 0.05]).astype(np.float32)), 0.02
    if name == "line":  # one node after the other: as many rounds as nodes
        return _sorted(np.stack([np.linspace(0, 1, 9000), 1e-4 * rng.random(9000), np.zeros(9000)], 1).astype(np.float32)), 0.004
    if name == "crowded":  # all but one point in one cell, most of them repeated
        p = np.repeat(rng.random((300, 3)) * 0.01, 20, 0)
        return np.concatenate([p, [[1.0, 1.0, 1.0]]]), 0.012
    if name == "lattice":  # distances of exactly the radius and of the cells' size
        g = np.arange(20) * 0.05
        return np.stack(np.meshgrid(g, g, g), -1).reshape(-1, 3), 0.05
    return rng.random((18000, 3)), 0.02  # "cells"


@pytest.mark.parametrize("name", ["one", "warp", "unordered", "ordered", "line", "crowded", "lattice", "cells"])
def test_graph_equals_sequential_walk(name):
    cloud, radius = _cloud(name)
    cloud = np.ascontiguousarray(cloud, np.float32)
    radius = float(np.float32(radius))
    no, ro, To = O.build_graph(cloud, 4, radius)
    n, r, T = _build(cloud, radius, len(no) + 10)
    assert len(n) == len(no)
    assert np.array_equal(n, no) and np.array_equal(r, ro) and np.array_equal(T, To)
    # grown by a shifted cloud, from transforms of its own
    rng = np.random.default_rng(1)
    T0 = rng.standard_normal((len(no), 16)).astype(np.float32)
    T0[0, 3] = -0.0
    more = np.ascontiguousarray(cloud + np.float32([0.3 * radius, 4 * radius, -0.2 * radius]))
    n2o, _, T2o = O.build_graph(more, 4, radius, no, ro, T0, cap=40000)
    n2, _, T2 = _build(more, radius, len(n2o) + 1, no, T0)
    assert np.array_equal(n2, n2o) and np.array_equal(T2, T2o)


def test_full_graph_keeps_the_first_nodes():
    from volumefusion_gb300._lib import AfxError
    cloud, radius = _cloud("ordered")
    radius = float(np.float32(radius))
    no, _, To = O.build_graph(cloud, 4, radius)
    cap = len(no) // 2
    from volumefusion_gb300 import af
    d_n, d_r, d_T = (torch.zeros(s, device="cuda") for s in ((cap, 3), (cap,), (cap, 16)))
    nn = torch.zeros(1, dtype=torch.int32, device="cuda")
    with pytest.raises(AfxError):
        af.buildGraph(d_n, d_r, d_T, nn, torch.from_numpy(cloud).cuda(),
                      torch.tensor([len(cloud)], dtype=torch.int32, device="cuda"), 4, radius)
    assert int(nn.item()) == cap
    assert np.array_equal(d_n.cpu().numpy(), no[:cap]) and np.array_equal(d_T.cpu().numpy(), To[:cap])
