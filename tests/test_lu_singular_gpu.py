"""afx_lu_solve on matrices with columns that have no pivot: the pivots of the columns before and after them are those of
column-by-column elimination that goes on without updates -- rows that a column has left are not candidates of a later
one, and a column without a pivot moves no rows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def pivots(A):
    """1-based pivots and the first column without one, as elimination by whole columns gives them."""
    A = A.copy()
    n = len(A)
    piv, info = np.zeros(n, np.int64), 0
    with np.errstate(all="ignore"):
        for k in range(n):
            v = np.abs(A[k:, k])
            ok = ~np.isnan(v)
            p = k + int(np.argmax(np.where(ok, v, -1.0))) if ok.any() else n
            piv[k] = p + 1
            if p == n or A[p, k] == 0:
                info = info or k + 1
                continue
            if p != k:
                A[[k, p]] = A[[p, k]]
            A[k + 1:, k] = A[k + 1:, k] / A[k, k]
            if not info:
                A[k + 1:, k + 1:] -= A[k + 1:, k][:, None] * A[k, k + 1:][None, :]
    return piv, info


# within the first half of a panel and the second, across panels, several rows per thread, 16 and 8 columns a panel
@pytest.mark.parametrize("n,bad", [(5, (0,)), (40, (5,)), (40, (25,)), (40, (0, 17)), (70, (31, 32)), (70, (69,)),
                                   (600, (300, 301)), (1100, (40, 700)), (2100, (3, 20)), (4200, (5, 9))])
@pytest.mark.parametrize("nan", [False, True])
def test_pivots_around_columns_without_one(n, bad, nan):
    from volumefusion_gb300._lib import lib
    L = lib()
    rng = np.random.default_rng(n + len(bad))
    A = rng.standard_normal((n, n)).astype(np.float32)
    for c in bad:
        A[:, c] = 0
        if nan:  # in a row that elimination may or may not have moved by then
            A[c, c] = np.nan
    piv, info = pivots(A)
    assert info
    dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    b = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    x, ip = torch.empty_like(b), torch.empty(n, dtype=torch.int32, device="cuda")
    size = L.afx_lu_solve_workspace_size(n, n)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    rc = L.afx_lu_solve(x.data_ptr(), dA.data_ptr(), n, n, b.data_ptr(), ip.data_ptr(), ws.data_ptr(), size,
                        torch.cuda.current_stream().cuda_stream)
    assert rc == 4  # AFX_ERR_SINGULAR
    assert torch.equal(x, b)
    assert np.array_equal(ip.cpu().numpy(), piv)
