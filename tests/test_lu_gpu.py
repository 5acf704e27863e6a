"""afx_lu_solve against column-by-column elimination with partial pivoting in binary32 (every product,
difference and quotient rounded by itself), at the sizes where its panels and tiles change: pivots,
factors and solution are the same bit for bit, since blocking leaves every element's operations and
their order as they are."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def eliminate(A, b):
    """LU = P A (unit lower part below the diagonal), 0-based pivots and x; zero entries are skipped, which
    changes nothing (a - 0 u = a)."""
    A, x = A.copy(), b.copy()
    n = len(b)
    piv = np.zeros(n, np.int64)
    for k in range(n):
        p = k + int(np.argmax(np.abs(A[k:, k])))
        piv[k] = p
        if p != k:
            A[[k, p]] = A[[p, k]]
            x[[k, p]] = x[[p, k]]
        rows = k + 1 + np.nonzero(A[k + 1:, k])[0]
        cols = k + 1 + np.nonzero(A[k, k + 1:])[0]
        A[rows, k] = A[rows, k] / A[k, k]
        if len(rows) and len(cols):
            A[np.ix_(rows, cols)] -= A[rows, k][:, None] * A[k, cols][None, :]
    for k in range(n):
        x[k + 1:] -= A[k + 1:, k] * x[k]
    for k in range(n - 1, -1, -1):
        x[k] = x[k] / A[k, k]
        x[:k] -= A[:k, k] * x[k]
    return A, piv, x


# one column, around a panel, around one and two rows per thread, the 16- and the 8-column panels
@pytest.mark.parametrize("n,lda,block", [(1, 1, 1), (31, 31, 31), (33, 40, 33), (64, 64, 64), (511, 511, 511),
                                         (513, 520, 513), (1024, 1024, 60), (1057, 1057, 60), (2080, 2083, 60),
                                         (4133, 4133, 60)])
def test_blocked_lu_equals_column_elimination(n, lda, block):
    from volumefusion_gb300._lib import lib
    L = lib()
    rng = np.random.default_rng(n)
    A = np.zeros((n, n), np.float32)
    for o in range(0, n, block):  # dense, or blocks whose rows are then mixed over the whole matrix
        m = min(block, n - o)
        A[o:o + m, o:o + m] = rng.standard_normal((m, m)).astype(np.float32)
    A = A[rng.permutation(n)]
    b = rng.standard_normal(n).astype(np.float32)
    lu, piv, x = eliminate(A, b)
    dA = torch.zeros((n, lda), dtype=torch.float32, device="cuda")  # column-major: row j holds column j
    dA[:, :n] = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    db = torch.from_numpy(b).cuda()
    dx = torch.empty(n, dtype=torch.float32, device="cuda")
    dp = torch.empty(n, dtype=torch.int32, device="cuda")
    size = L.afx_lu_solve_workspace_size(n, lda)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    rc = L.afx_lu_solve(dx.data_ptr(), dA.data_ptr(), n, lda, db.data_ptr(), dp.data_ptr(), ws.data_ptr(), size,
                        torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert np.array_equal(dp.cpu().numpy() - 1, piv)
    got = ws[:4 * lda * n].view(torch.float32).reshape(n, lda)[:, :n].cpu().numpy().T
    assert np.array_equal(got, lu)
    assert np.array_equal(dx.cpu().numpy(), x)


def test_failing_column_is_reported():
    """A column without a pivot: singular whatever panel it is in, and x is left as b."""
    from volumefusion_gb300._lib import lib
    L = lib()
    rng = np.random.default_rng(3)
    for n, bad in ((40, 0), (40, 35), (600, 300)):
        A = rng.standard_normal((n, n)).astype(np.float32)
        A[:, bad] = 0
        dA = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        db = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
        dx, dp = torch.empty_like(db), torch.empty(n, dtype=torch.int32, device="cuda")
        size = L.afx_lu_solve_workspace_size(n, n)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        rc = L.afx_lu_solve(dx.data_ptr(), dA.data_ptr(), n, n, db.data_ptr(), dp.data_ptr(), ws.data_ptr(), size,
                            torch.cuda.current_stream().cuda_stream)
        assert rc == 4  # AFX_ERR_SINGULAR
        assert torch.equal(dx, db)
        assert 1 <= int(dp.min()) and int(dp.max()) <= n
