"""The diagonal copy of the operator keeps one half of it: only where the other
half is its mirror image, stored entry by stored entry."""
import numpy as np
import pytest
import scipy.sparse as sp

from statfem_b200 import api

pytestmark = pytest.mark.gpu


# one cluster and the grid (1e5 nonzeros divide them); an entry missing below or above
@pytest.mark.parametrize("n", [200, 50000])
@pytest.mark.parametrize("missing", [None, (100, 99), (99, 100)])
def test_missing_entry_is_not_mirrored(ctx, n, missing):
    """The solution solves the matrix that was inserted, and the reported
    residual is its residual."""
    A = sp.diags([np.ones(n - 1), np.full(n, 4.0), np.ones(n - 1)], [-1, 0, 1]).tocsr()
    if missing is not None:
        A[missing] = 0.0
        A.eliminate_zeros()
        assert A.nnz == 3 * n - 3
    s = api.SystemSolveCuda(ctx, n)
    s.set_options(method=api.SFC_SOLVER_PCG_FP64, tol=1e-10)
    for i in range(n):
        at = slice(A.indptr[i], A.indptr[i + 1])
        s.insertToMatrix(A.data[at].reshape(1, -1), [i], A.indices[at])
    b = np.cos(np.arange(n))
    s.insertToRhs(b, np.arange(n))
    s.finishAssembly()
    s.solveSystem()
    rel = np.linalg.norm(A @ s.giveSolution() - b) / np.linalg.norm(b)
    assert rel <= 1.1e-10
    assert s.last_stats()["max_rel_residual"] <= 1.1e-10
    s.close()
