"""The PCG solve over graph sizes: fewer nodes than the cluster has CTAs could use, several lanes
per matrix row, one lane per row at the largest size of the shared-memory path, and the global-memory path
after it.  Systems are disjoint copies of one small system (as in test_gauss_newton_gpu.py), so each
copy is held to that system's solution: ten iterations to the oracle's binary64 PCG, and a solve to a
tolerance to its true residual, both within the bounds that test derives."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402
from _gn_system import assembled, gn_system  # noqa: E402

pytestmark = pytest.mark.gpu


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def tiled(s, copies):
    n, m, P = len(s["nodes"]), len(s["mesh"]), s["v1"].shape[0] * s["v1"].shape[1]
    inval = np.uint32(0xFFFFFFFF)

    def shifted(idx):
        return np.concatenate([np.where(idx == inval, inval, idx + np.uint32(c * n)) for c in range(copies)]).astype(np.uint32)

    t = {k: np.tile(s[k], (copies, 1)) for k in ("mesh", "mw", "warped", "nodes", "T")}
    t["midx"], t["gidx"] = shifted(s["midx"]), shifted(s["gidx"])
    t["corr"] = np.concatenate([s["corr"] + np.array([c * m, c * P], np.int32) for c in range(copies)])
    t["v1"], t["n1"] = (np.tile(s[k].reshape(-1, 3), (copies, 1)) for k in ("v1", "n1"))
    return t


@pytest.mark.parametrize("fill", ["one", "two", "half", "limit", "past"])
def test_solve_over_graph_sizes(fill):
    from volumefusion_gb300 import af
    s = gn_system(4, 8)
    n = len(s["nodes"])
    copies = {"one": 1, "two": 2, "half": 512 // n, "limit": 1024 // n, "past": 1024 // n + 1}[fill]
    A, b = assembled(s)
    x_o, _ = O.pcg(A, b, 10)
    A64, b64 = A.astype(np.float64), b.astype(np.float64)
    t = tiled(s, copies)
    N, M, NC = n * copies, len(t["mesh"]), len(t["corr"])
    g = af.GaussNewtonSystem(M + 16, N + 8, 4, 8)
    cnt = lambda v: cu(np.array([v], np.int32))  # noqa: E731
    g.build(cu(t["mesh"]), cnt(M), cu(t["midx"].view(np.int32)), cu(t["mw"]), cu(t["corr"]), cnt(NC), cu(t["v1"]),
            cu(t["n1"]), cu(t["warped"]), cu(t["nodes"]), cu(t["T"]), cnt(N), cu(t["gidx"].view(np.int32)),
            s["lam_d"], s["lam_r"])
    x = g.solve(10)[:6 * N].cpu().numpy().reshape(copies, 6 * n)
    xc = g.solve(400, tol=1e-7)[:6 * N].cpu().numpy().astype(np.float64).reshape(copies, 6 * n)
    again = g.solve(10)[:6 * N].cpu().numpy().reshape(copies, 6 * n)
    g.close()
    assert np.array_equal(x, again)
    for c in range(copies):
        assert np.linalg.norm(x[c] - x_o) <= 3e-2 * np.linalg.norm(x_o), c
        assert np.linalg.norm(b64 - A64 @ xc[c]) <= 1e-4 * np.linalg.norm(b64), c
