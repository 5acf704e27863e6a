"""J^T J assembly at the sizes where its split over a CTA can go wrong: node lists around the 256
rows staged at a time, one to eight slots per vertex, more upper blocks than are summed at a time,
more incoming edges than a warp sorts, nodes nothing refers to, and vertices that list a node twice.
Each entry is compared bit for bit with its rows summed in order in binary32 (numpy)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
F = np.float32
NONE = np.uint32(0xFFFFFFFF)


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def grad(p):
    G = np.zeros((3, 6), F)
    G[0, 1], G[0, 2], G[1, 0], G[1, 2], G[2, 0], G[2, 1] = p[2], -p[1], -p[2], p[0], p[1], -p[0]
    G[0, 3] = G[1, 4] = G[2, 5] = 1
    return G


def reference(s):
    """Dense J^T J: block (a, b >= a) sums rows in the order of a's entries, then of the edges."""
    n, k = len(s["nodes"]), s["midx"].shape[1]
    A = np.zeros((n, n, 6, 6), F)
    touched = np.zeros(n, bool)
    for v, px in s["corr"]:
        G, nrm = grad(s["mesh"][v]), s["normals"][px]
        J = np.zeros((k, 6), F)
        for t in range(k):
            if s["mw"][v, t] >= F(1e-4):
                q = nrm * s["mw"][v, t]
                J[t] = (q[0] * G[0] + (q[1] * G[1] + q[2] * G[2])) * s["lam_d"]
        for a in range(k):
            if s["mw"][v, a] == 0:
                continue
            touched[s["midx"][v, a]] = True
            for b in range(k):
                if s["mw"][v, b] != 0 and s["midx"][v, b] >= s["midx"][v, a]:
                    A[s["midx"][v, a], s["midx"][v, b]] += np.outer(J[a], J[b])
    for i in range(n):
        G = grad(s["nodes"][i]) * s["lam_r"]
        for nb in s["gidx"][i]:
            if nb == NONE:
                continue
            touched[i] = touched[nb] = True
            for ax in range(3):
                P = np.outer(G[ax], G[ax])
                A[i, i] += P
                A[nb, nb] += P
                A[min(i, nb), max(i, nb)] -= P
    for a in range(n):
        if not touched[a]:
            A[a, a] = np.eye(6, dtype=F)
        for b in range(a):
            A[a, b] = A[b, a].T
    return A.transpose(0, 2, 1, 3).reshape(6 * n, 6 * n)


def system(n, m, k, kreg, twice=False, hub=False, share=0.8, seed=0):
    rng = np.random.default_rng(seed + 131 * n + 17 * m + k)
    midx = np.stack([rng.permutation(n)[:k] if n >= k else rng.integers(0, n, k) for _ in range(m)]).astype(np.uint32)
    if twice:
        midx[::3, -1] = midx[::3, 0]
    mw = rng.uniform(0, 1, (m, k)).astype(F)
    mw[:, 1:][rng.random((m, k - 1)) < 0.1] = 0
    mw[:, 1:][rng.random((m, k - 1)) < 0.05] = F(5e-5)
    gidx = np.full((n, kreg), NONE, np.uint32)
    for i in range(n):
        others = np.delete(np.arange(n), i)[:]
        pick = rng.permutation(others)[:kreg]
        gidx[i, :len(pick)] = pick
        if hub and i:
            gidx[i] = NONE
            gidx[i, 0] = 0
    if n > 4:
        gidx[n - 1] = NONE
        gidx[gidx == n - 1] = NONE
        mw[midx == n - 1] = 0
    corr = np.sort(rng.permutation(m)[:max(1, int(share * m))])
    corr = np.stack([corr, rng.permutation(len(corr))], 1).astype(np.int32)
    nrm = rng.normal(size=(m, 3))
    return dict(mesh=rng.normal(size=(m, 3)).astype(F), nodes=rng.normal(size=(n, 3)).astype(F), midx=midx, mw=mw, gidx=gidx,
                corr=corr, normals=(nrm / np.linalg.norm(nrm, axis=1, keepdims=True)).astype(F), lam_d=F(1.0),
                lam_r=F(14.142135))


@pytest.mark.parametrize("n,m,k,kreg,kw", [
    (1, 1, 1, 1, {}), (1, 255, 1, 1, dict(share=1.0)), (1, 256, 1, 1, dict(share=1.0)), (2, 257, 1, 2, dict(share=1.0)),
    (3, 700, 2, 2, {}), (9, 520, 3, 4, {}), (40, 300, 4, 8, {}), (60, 400, 8, 8, {}), (64, 260, 5, 3, dict(share=0.1)),
    (60, 90, 4, 1, dict(hub=True)), (12, 270, 4, 4, dict(twice=True)), (5, 64, 7, 8, dict(twice=True))])
def test_assembly(n, m, k, kreg, kw):
    from volumefusion_gb300 import af
    s = system(n, m, k, kreg, **kw)
    nc = len(s["corr"])
    g = af.GaussNewtonSystem(m + 3, n + 2, k, kreg)
    cnt = lambda v: cu(np.array([v], np.int32))  # noqa: E731
    T = cu(np.tile(np.eye(4, dtype=F).reshape(-1), (n, 1)))
    for _ in range(2):  # the second on used workspaces
        g.build(cu(s["mesh"]), cnt(m), cu(s["midx"].view(np.int32)), cu(s["mw"]), cu(s["corr"]), cnt(nc), cu(s["mesh"]),
                cu(s["normals"]), cu(s["mesh"]), cu(s["nodes"]), T, cnt(n), cu(s["gidx"].view(np.int32)), s["lam_d"], s["lam_r"])
        jtj, jtr, rd, rr = g.export(n, nc)
        assert np.array_equal(jtj.cpu().numpy(), reference(s))
    g.close()
