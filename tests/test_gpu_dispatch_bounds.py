"""The bounds of two rules of the solve phase: block solves whose longest rows
have 127 to 130 entries (a block's warps share rows of over 128), and
programmatic launches against plain ones, to the bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from blood_network_b200 import amg
from test_gpu_hubs import hub_matrix
from test_gpu_solve_paths import _vascular

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("k", [5, 64])
@pytest.mark.parametrize("row", [127, 128, 129, 130])
def test_block_rows_at_the_length_that_warps_share(row, k, precision):
    # a hub's row: its neighbours and the diagonal
    n, ia, ja, val = hub_matrix(side=40, hubs=(row - 1,) * 3, weak_hubs=(), seed=row)
    assert np.diff(ia).max() == row
    A = sp.csr_matrix((val, ja, ia), shape=(n, n))
    B = np.random.default_rng(k).standard_normal((n, k))
    s = amg.AMGSolver(n, ia, ja, val, min_size=100, precision=precision, stop=amg.STOP_RELRES)
    X, its, rel, rc = s.solve_block(B, tol=1e-9)
    single = s.solve(np.ascontiguousarray(B[:, 0]), tol=1e-9)[1]
    s.close()
    assert rc == 0 and abs(its[0] - single) <= 1
    r = np.linalg.norm(B - A @ X, axis=0) / np.linalg.norm(B, axis=0)
    assert (r <= 1.01e-9).all()


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("n", [40, 3000, 60000])
def test_programmatic_launches_keep_every_bit(n, precision, monkeypatch):
    """The same kernels in the same order, and no sum depends on timing: one
    application of the preconditioner, a solve and a segmented solve, several
    times each, give the same bytes with plain launches."""
    m, ia, ja, val = _vascular(n, False)
    A = sp.block_diag([sp.csr_matrix((val, ja, ia), shape=(m, m))] * 2, format="csr")
    ptr = np.array([0, m, 2 * m], np.int32)
    b = np.random.default_rng(n).standard_normal(2 * m)
    out = []
    for pdl in "01":
        monkeypatch.setenv("BN_PDL", pdl)
        s = amg.AMGSolver(m, ia, ja, val, precision=precision, stop=amg.STOP_RELRES)
        t = amg.AMGSolver(2 * m, A.indptr, A.indices, A.data, precision=precision,
                          stop=amg.STOP_RELRES)
        for _ in range(4):
            x, it = s.solve(b[:m], tol=1e-8)
            y, its, _, rc = t.solve_segmented(ptr, b, tol=1e-8)
            assert it > 0 and rc == 0
            out.append((s.precond(b[:m]).tobytes(), x.tobytes(), it, y.tobytes(), tuple(its)))
        s.close()
        t.close()
    assert len(set(out)) == 1
