"""The PCG solve of graphs past the shared-memory path, at the sizes where its layout changes: all
blocks in shared memory, some of them, none but the neighbours, the last size whose search direction
fits, and the global-memory path after it.  Systems are disjoint copies of one small system, so every
copy's iterates have the same bits, and each is held to the oracle's binary64 PCG and true residual
within the bounds that test_gauss_newton_gpu.py derives."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import pyoracle as O  # noqa: E402
from _gn_system import assembled, gn_system  # noqa: E402
from test_pcg_sizes_gpu import cu, tiled  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [1025, 1400, 2501, 5003, 7200, 7700])
def test_solve_past_the_shared_memory_path(nodes):
    from volumefusion_gb300 import af
    s = gn_system(4, 8)
    n = len(s["nodes"])
    copies = -(-nodes // n)
    A, b = assembled(s)
    x_o, _ = O.pcg(A, b, 10)
    A64, b64 = A.astype(np.float64), b.astype(np.float64)
    t = tiled(s, copies)
    N, M, NC = n * copies, len(t["mesh"]), len(t["corr"])
    g = af.GaussNewtonSystem(M, N, 4, 8)
    cnt = lambda v: cu(np.array([v], np.int32))  # noqa: E731
    g.build(cu(t["mesh"]), cnt(M), cu(t["midx"].view(np.int32)), cu(t["mw"]), cu(t["corr"]), cnt(NC), cu(t["v1"]),
            cu(t["n1"]), cu(t["warped"]), cu(t["nodes"]), cu(t["T"]), cnt(N), cu(t["gidx"].view(np.int32)),
            s["lam_d"], s["lam_r"])
    x = g.solve(10)[:6 * N].cpu().numpy().reshape(copies, 6 * n)
    xc = g.solve(400, tol=1e-7)[:6 * N].cpu().numpy().astype(np.float64).reshape(copies, 6 * n)
    x0 = g.solve(0)[:6 * N].cpu().numpy()
    again = g.solve(10)[:6 * N].cpu().numpy().reshape(copies, 6 * n)
    g.close()
    assert np.array_equal(x, again) and not x0.any()
    assert np.array_equal(x, np.tile(x[0], (copies, 1))) and np.array_equal(xc, np.tile(xc[0], (copies, 1)))
    assert np.linalg.norm(x[0] - x_o) <= 3e-2 * np.linalg.norm(x_o)
    assert np.linalg.norm(b64 - A64 @ xc[0]) <= 1e-4 * np.linalg.norm(b64)
