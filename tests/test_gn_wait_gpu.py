"""A solve one of whose waits between thread blocks runs out: the limit is set so low that the first wait gives up at once,
the caller is told, x is not taken for a solution, and the same system is solved afterwards as if nothing had been."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from _gn_system import gn_system  # noqa: E402
from test_pcg_sizes_gpu import cu, tiled  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 6, 35])
@pytest.mark.parametrize("tol", [0.0, 1e-7])
def test_wait_that_runs_out_is_reported(copies, tol):
    from volumefusion_gb300 import af
    from volumefusion_gb300._lib import AfxError, lib
    s = gn_system(4, 8)
    t = tiled(s, copies)
    N, M, NC = len(t["nodes"]), len(t["mesh"]), len(t["corr"])
    g = af.GaussNewtonSystem(M, N, 4, 8)
    cnt = lambda v: cu(np.array([v], np.int32))  # noqa: E731
    st = torch.cuda.current_stream().cuda_stream
    g.build(cu(t["mesh"]), cnt(M), cu(t["midx"].view(np.int32)), cu(t["mw"]), cu(t["corr"]), cnt(NC), cu(t["v1"]),
            cu(t["n1"]), cu(t["warped"]), cu(t["nodes"]), cu(t["T"]), cnt(N), cu(t["gidx"].view(np.int32)),
            s["lam_d"], s["lam_r"])
    want = g.solve(10, tol).cpu().numpy()
    assert np.isfinite(want).all() and lib().afx_gn_status(g.h, st) == 0
    for iterations in (0, 1, 10):
        assert lib().afx_gn_set_wait_limit(g.h, 0) == 0
        x = torch.zeros(6 * N, device="cuda")
        assert lib().afx_gn_solve(g.h, x.data_ptr(), iterations, tol, st) == 0
        assert lib().afx_gn_status(g.h, st) == 7  # AFX_ERR_TIMEOUT
        assert bool(torch.isnan(x).all())
        assert lib().afx_gn_status(g.h, st) == 0  # reported once
        with pytest.raises(AfxError):
            g.solve(iterations, tol)
        assert lib().afx_gn_set_wait_limit(g.h, 1 << 20) == 0
        assert np.array_equal(g.solve(10, tol).cpu().numpy(), want)
    assert lib().afx_gn_set_wait_limit(g.h, -1) == 1
    g.close()
