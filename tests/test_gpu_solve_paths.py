"""The solve phase's kernel choices against each other: an operator that a rule
sends to another kernel keeps the preconditioner up to rounding."""
import numpy as np
import pytest

from blood_network_b200 import amg
from test_gpu_hubs import hub_matrix

pytestmark = pytest.mark.gpu


def precond(n, ia, ja, val, g, **kw):
    s = amg.AMGSolver(n, ia, ja, val, min_size=kw.pop("min_size", 200), **kw)
    x = s.precond(g)
    s.close()
    return x


# row sums of at most 1,500 terms in another order: 1500 * 2^-53 (2^-24) of the
# row's magnitude, through some thirty dependent operations of one application
TOL = {amg.PREC_FP64: 1e-10, amg.PREC_MIXED: 2e-3}


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("deg", [126, 127, 128, 1023, 1024])
def test_irregular_rows_on_the_packed_kernels(deg, precision, monkeypatch):
    n, ia, ja, val = hub_matrix(side=60, hubs=(deg,) * 3, weak_hubs=(), seed=deg)
    g = np.random.default_rng(deg).standard_normal(n)
    x = precond(n, ia, ja, val, g, precision=precision)
    monkeypatch.setenv("BN_PACKED", "0")
    y = precond(n, ia, ja, val, g, precision=precision)
    assert np.linalg.norm(x - y) <= TOL[precision] * np.linalg.norm(y)


@pytest.mark.parametrize("nseg", [1, 3, 64, 593, 700])
def test_segment_dots_of_uneven_segments(nseg):
    """Slices per segment: 64 for one segment, 197 capped to 64 for three, 9 for
    64, none (one slice) from 593 on; segments of 1 to 400 rows, so slices of no
    row among them.  Every segment is a path graph with its own right-hand side."""
    import scipy.sparse as sp
    rng = np.random.default_rng(nseg)
    sizes = rng.integers(1, 400 if nseg < 100 else 12, nseg)
    sizes[0] = 1
    blocks = [sp.diags([-np.ones(m - 1), np.full(m, 2.01), -np.ones(m - 1)], [-1, 0, 1])
              for m in sizes]
    A = sp.block_diag(blocks, format="csr")
    A.sort_indices()
    ptr = np.r_[0, np.cumsum(sizes)].astype(np.int32)
    b = rng.standard_normal(A.shape[0])
    s = amg.AMGSolver(A.shape[0], A.indptr, A.indices, A.data, min_size=50, stop=amg.STOP_RELRES)
    x, its, rel, rc = s.solve_segmented(ptr, b, tol=1e-10)
    s.close()
    assert rc == 0 and (its > 0).all()
    r = b - A @ x
    for k in range(nseg):
        q = slice(ptr[k], ptr[k + 1])
        # the stopping test holds, and the reported residual is the true one
        assert rel[k] < 1e-10
        assert np.linalg.norm(r[q]) <= 1.01e-10 * np.linalg.norm(b[q])


def _random_spd(n, per_row, seed):
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    m = n * per_row // 2
    u, v = rng.integers(0, n, m), rng.integers(0, n, m)
    keep = u != v
    w = sp.coo_matrix((rng.uniform(0.1, 1, keep.sum()), (u[keep], v[keep])), shape=(n, n))
    w = (w + w.T).tocsr()
    a = (sp.diags(np.asarray(w.sum(1)).ravel() + 0.1) - w).tocsr()
    a.sort_indices()
    return n, a.indptr.astype(np.int32), a.indices.astype(np.int32), a.data


def _vascular(n, shuffle):
    import scipy.sparse as sp
    from blood_network_b200.network import vascular_network
    net = vascular_network(depth=max(4, int(round(np.log2(0.2 * n)))), n_nodes=n, seed=5)
    if not shuffle:
        return net.n, net.indptr, net.indices, net.data
    a = sp.csr_matrix((net.data, net.indices, net.indptr), shape=(net.n, net.n))
    q = np.random.default_rng(9).permutation(net.n)
    a = a[q][:, q].tocsr()
    a.sort_indices()
    return net.n, a.indptr.astype(np.int32), a.indices.astype(np.int32), a.data


# one step; a last step of one row; rows of more than four entries; a row with
# over a thousand; one block and several; a numbering that scatters every
# dependency over the blocks; levels wide enough to be dealt
OWN_CASES = {
    "rows33": lambda: _random_spd(33, 4, 1),
    "rows1025": lambda: _random_spd(1025, 3, 2),
    "dense": lambda: _random_spd(900, 14, 3),
    "hub": lambda: hub_matrix(side=40, hubs=(1200,), weak_hubs=(), seed=4),
    "tree": lambda: _vascular(3_000, False),
    "vascular": lambda: _vascular(60_000, False),
    "shuffled": lambda: _vascular(60_000, True),
}


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("name", sorted(OWN_CASES))
def test_owner_sweeps_equal_the_chunked_ones(name, precision, monkeypatch):
    n, ia, ja, val = OWN_CASES[name]()
    g = np.random.default_rng(n).standard_normal(n)
    kw = dict(precision=precision, min_size=30)
    x = precond(n, ia, ja, val, g, **kw)
    monkeypatch.setenv("BN_IC_OWN", "0")
    y = precond(n, ia, ja, val, g, **kw)
    assert x.tobytes() == y.tobytes() and np.isfinite(x).all()


# levels that are all the tail, partly, and with rows taken by a lane group, a
# warp (over 8 entries a lane) and a block (over 256 entries); several sweeps;
# plain Gauss-Seidel order; HMIS hierarchies
TAIL_CASES = {
    "one level": (lambda: _random_spd(200, 4, 6), dict(min_size=500)),
    "two levels": (lambda: _random_spd(601, 4, 7), dict(min_size=500)),
    "vascular 2k": (lambda: _vascular(2_000, False), {}),
    "vascular 60k": (lambda: _vascular(60_000, False), {}),
    "hmis": (lambda: _vascular(20_000, False), dict(coarsening=amg.COARSEN_HMIS, threshold=0.5)),
    "hubs": (lambda: hub_matrix(side=50, hubs=(60, 255, 256, 257, 1100, 2300), weak_hubs=(),
                                seed=8), {}),
    "two sweeps": (lambda: _vascular(5_000, False), dict(nu=2)),
    "plain order": (lambda: _vascular(5_000, False), dict(smoother=amg.SMOOTHER_GS)),
}


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("name", sorted(TAIL_CASES))
def test_tail_equals_the_level_launches(name, precision, monkeypatch):
    make, kw = TAIL_CASES[name]
    n, ia, ja, val = make()
    g = np.random.default_rng(n).standard_normal(n)
    x = precond(n, ia, ja, val, g, precision=precision, **kw)
    monkeypatch.setenv("BN_TAIL", "0")
    y = precond(n, ia, ja, val, g, precision=precision, **kw)
    assert np.linalg.norm(x - y) <= TOL[precision] * np.linalg.norm(y)


def test_tail_after_the_hierarchy_changes(monkeypatch):
    """A new smoother, precision and new values rebuild the tail's programs."""
    n, ia, ja, val = _vascular(4_000, False)
    g = np.random.default_rng(2).standard_normal(n)

    def passes():
        s = amg.AMGSolver(n, ia, ja, val, min_size=200)
        out = [s.precond(g)]
        s.set_smoother(amg.SMOOTHER_GS)
        out.append(s.precond(g))
        s.set_smoother(amg.SMOOTHER_JACOBI, 0.6)
        out.append(s.precond(g))
        s.set_smoother(amg.SMOOTHER_CF_GS)
        out.append(s.precond(g))
        s.set_precision(amg.PREC_MIXED)
        out.append(s.precond(g))
        s.set_precision(amg.PREC_FP64)
        s.update(ia, ja, 2.0 * val)
        out.append(s.precond(g))
        s.close()
        return out

    tail = passes()
    monkeypatch.setenv("BN_TAIL", "0")
    plain = passes()
    assert tail[0].tobytes() == tail[3].tobytes() and tail[0].tobytes() != tail[1].tobytes()
    for k, (x, y) in enumerate(zip(tail, plain)):
        tol = TOL[amg.PREC_MIXED if k == 4 else amg.PREC_FP64]
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), k


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("k", [1, 5, 33, 64])
@pytest.mark.parametrize("deg", [62, 63, 64, 65, 600, 1022, 1023, 1024])
def test_block_rows_split_over_the_warps(deg, k, precision):
    """Many right-hand sides over rows at and around the lengths that a block's
    warps share (64) and that a block of their own takes (1024): every column
    meets the tolerance on the true residual."""
    import scipy.sparse as sp
    n, ia, ja, val = hub_matrix(side=40, hubs=(deg, deg), weak_hubs=(), seed=deg)
    A = sp.csr_matrix((val, ja, ia), shape=(n, n))
    B = np.random.default_rng(k).standard_normal((n, k))
    s = amg.AMGSolver(n, ia, ja, val, min_size=100, precision=precision, stop=amg.STOP_RELRES)
    X, its, rel, rc = s.solve_block(B, tol=1e-9)
    single = s.solve(np.ascontiguousarray(B[:, 0]), tol=1e-9)[1]
    s.close()
    assert rc == 0 and abs(its[0] - single) <= 1
    r = np.linalg.norm(B - A @ X, axis=0) / np.linalg.norm(B, axis=0)
    assert (r <= 1.01e-9).all()


@pytest.mark.parametrize("seed", [1, 2])
def test_block_rows_split_in_some_rounds_only(seed):
    """More rows than the grid's warps, so that a block takes several rounds of
    eight rows, some of them with a row to share and most without."""
    import scipy.sparse as sp
    n, ia, ja, val = hub_matrix(side=130, hubs=(70, 90, 200, 65, 400, 300) * 20, weak_hubs=(),
                                seed=seed)
    q = np.random.default_rng(seed).permutation(n)
    A = sp.csr_matrix((val, ja, ia), shape=(n, n))[q][:, q].tocsr()
    A.sort_indices()
    B = np.random.default_rng(seed).standard_normal((n, 64))
    s = amg.AMGSolver(n, A.indptr, A.indices, A.data, min_size=300, precision=amg.PREC_MIXED,
                      stop=amg.STOP_RELRES)
    X, its, rel, rc = s.solve_block(B, tol=1e-9)
    s.close()
    r = np.linalg.norm(B - A @ X, axis=0) / np.linalg.norm(B, axis=0)
    assert rc == 0 and (r <= 1.01e-9).all()


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("n", [40, 3000, 60000])
def test_programmatic_launches_change_nothing(n, precision, monkeypatch):
    """The same kernels in the same order: a result that differs was read early."""
    m, ia, ja, val = _vascular(n, False)
    b = np.random.default_rng(n).standard_normal(m)
    out = []
    for pdl in "01":
        monkeypatch.setenv("BN_PDL", pdl)
        s = amg.AMGSolver(m, ia, ja, val, precision=precision, stop=amg.STOP_RELRES)
        x = s.solve(b, tol=1e-8)[0]
        out.append((s.precond(b), x))
        s.close()
    for x, y in zip(*out):
        assert np.linalg.norm(x - y) <= TOL[precision] * np.linalg.norm(y)


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("n, per_row", [(65536, 8), (65537, 8), (65537, 16), (65537, 30),
                                        (65537, 50), (65537, 80), (131073, 8), (3000, 5),
                                        (3000, 12), (3000, 40)])
def test_lanes_per_row(n, per_row, precision, monkeypatch):
    """Both sides of every bound of the rule for the Gauss-Seidel lanes, against
    one lane per row."""
    m, ia, ja, val = _random_spd(n, per_row, per_row)
    g = np.random.default_rng(n).standard_normal(m)
    x = precond(m, ia, ja, val, g, precision=precision)
    monkeypatch.setenv("BN_GS_LANES", "1")
    y = precond(m, ia, ja, val, g, precision=precision)
    assert np.linalg.norm(x - y) <= TOL[precision] * np.linalg.norm(y)
