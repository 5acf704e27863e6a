"""K nearest nodes among more nodes than a thread block holds, for more queries than a warp search takes: at the edges of
the parts the nodes are taken in, with every warp of the grid having queries, some of them, and several rounds.
Distances are compared bit for bit with binary32 arithmetic in the same order, and equal ones lie in index order."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def squared(q, p):
    d = q - p
    d = d * d
    return (d[..., 0] + d[..., 1]) + d[..., 2]


@pytest.mark.parametrize("n,m,k,odd", [(12545, 8193, 4, False), (25088, 9000, 9, False), (25089, 20001, 3, True),
                                       (12545, 152 * 32 * 32 + 33, 4, False), (3000, 20001, 4, True), (12544, 9000, 4, True)])
def test_knn_in_parts(n, m, k, odd):
    from volumefusion_gb300 import af
    g = torch.Generator(device="cuda").manual_seed(n + m)
    nodes = torch.randn((n, 3), generator=g, device="cuda")
    nodes = (0.4 * nodes / nodes.norm(dim=1, keepdim=True)).contiguous()
    nodes[n - 2] = nodes[5]  # equal distances, across the parts where there are several
    if odd:
        nodes[n // 3, 1] = float("inf")
    q = nodes[torch.randint(0, n, (m,), generator=g, device="cuda")] + 0.01 * torch.randn((m, 3), generator=g, device="cuda")
    q[~torch.isfinite(q)] = 0.0
    q[-1] = nodes[5]
    idx = torch.empty((m, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((m, k), device="cuda")
    af.getKnnData(idx, dist, nodes, torch.tensor([n], dtype=torch.int32, device="cuda"), q)
    for a in range(0, m, 4096):
        i, d = idx[a:a + 4096].long(), dist[a:a + 4096]
        D = squared(q[a:a + 4096, None], nodes[None])
        assert torch.equal(D.topk(k, largest=False).values.sqrt(), d)
        assert torch.equal(D.gather(1, i).sqrt(), d)
        sq = D.gather(1, i)
        assert bool(((sq[:, 1:] > sq[:, :-1]) | ((sq[:, 1:] == sq[:, :-1]) & (i[:, 1:] > i[:, :-1]))).all())
        last = sq[:, -1:]
        j = torch.arange(n, device="cuda")
        assert int(((D == last) & (j < i[:, -1:])).sum() - (sq[:, :-1] == last).sum()) == 0  # of equal ones the first
    assert idx[-1, :2].tolist() == [5, n - 2]
