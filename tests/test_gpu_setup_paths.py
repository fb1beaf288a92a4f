"""Setup kernels at the sizes where their row classes change, bit for bit against
the oracle, and the C library's rand() state after a PMIS hierarchy."""
import ctypes as C

import numpy as np
import pytest

from blood_network_b200 import amg
from helpers import bits_equal
from test_gpu_hubs import hub_matrix
from test_gpu_parity import _dcsr, _out
from test_gpu_solve_paths import _random_spd, _vascular

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle():
    import ref
    if not ref.have_oracle():
        pytest.skip("oracle library not built")
    return ref


@pytest.mark.parametrize("c_share", [0.4, 0.05, 0.9])
def test_interpolation_of_rows_with_many_strong_points(oracle, c_share):
    """F rows of 32 and 33 strong points (a thread or a warp / a block), a block's
    most (2048) and one more, F points whose strong neighbours are such rows,
    denominators that vanish (no C point in common)."""
    n, ia, ja, val = hub_matrix(side=70, hubs=(32, 33, 34, 255, 256, 257, 700, 2047, 2048, 2049),
                                weak_hubs=(500,), seed=3)
    lib = amg.load_library()
    A = (ia, ja, val)
    S, _ = oracle.orc_strength(n, *A, 0.25)
    rng = np.random.default_rng(1)
    cf = np.where(rng.random(n) < c_share, 1, -1).astype(np.int32)
    cf[70 * 70:] = -1  # the hubs are F points
    P_ref = oracle.orc_interp(n, A, S, cf)
    dP = amg.DcsrMat()
    lib.rs_standard_interpolation(C.byref(_dcsr(n, n, *A)), C.byref(_dcsr(n, n, *S)),
                                  amg._p(cf), C.byref(dP))
    assert lib.amg_solver_last_status() == 0
    P = _out(dP)
    for j in range(3):
        assert bits_equal(P[j], P_ref[j])


@pytest.mark.parametrize("n,per_row", [(1, 0), (700, 2), (3000, 5), (2000, 9), (600, 30)])
def test_factor_rows_of_every_length(oracle, n, per_row):
    """Factor rows of one entry, up to six and over (register and walking form),
    columns with more than four leading entries, levels of one row."""
    n, ia, ja, val = _random_spd(n, per_row, n + per_row)
    lib = amg.load_library()
    L_ref = oracle.orc_ichol(n, ia, ja, val)
    f = amg.IcholFactor()
    lib.ichol_compute(C.byref(_dcsr(n, n, ia, ja, val)), C.byref(f))
    L = (np.ctypeslib.as_array(f.ia, shape=(n + 1,)).copy(),
         np.ctypeslib.as_array(f.ja, shape=(f.nnz,)).copy(),
         np.ctypeslib.as_array(f.val, shape=(f.nnz,)).copy())
    lib.ichol_free(C.byref(f))
    for j in range(3):
        assert bits_equal(L[j], L_ref[j])


@pytest.mark.parametrize("nodes", [5_000, 60_000])
def test_rand_state_after_a_pmis_hierarchy(nodes):
    """As the reference leaves it: srand(12345) and one draw per point of the last
    level it coarsened, whether the levels drew on the host or on the device."""
    n, ia, ja, val = _vascular(nodes, False)
    libc = C.CDLL(None)
    libc.srand(777)
    s = amg.AMGSolver(n, ia, ja, val)
    got = [libc.rand() for _ in range(3)]
    last = s.level(s.num_levels - 2)["n"]
    s.close()
    libc.srand(12345)
    for _ in range(last):
        libc.rand()
    assert got == [libc.rand() for _ in range(3)]


def test_rap_rows_of_every_class(oracle):
    """Coarse rows of given numbers of products and of distinct columns, both sides of
    each bound of the row classes, A rows of 0 to 3,000 entries among them."""
    rng = np.random.default_rng(8)
    # products without the diagonal's own, distinct columns
    want = [(0, 1), (63, 64), (64, 40), (300, 65), (512, 500), (1023, 90), (1024, 90),
            (1025, 512), (1025, 513), (4000, 20), (9000, 512), (16383, 512), (16383, 513),
            (16383, 4096), (16383, 4097), (16384, 512), (16384, 3000)]
    nc = 5000
    R, Arows = [[] for _ in range(nc)], [[] for _ in range(nc)]
    for ic, (products, width) in enumerate(want):
        cols = np.r_[np.arange(min(width, products)), rng.integers(0, width, max(0, products - width))]
        rng.shuffle(cols)
        at = 0
        while at < products:
            m = int(rng.choice([0, 1, 3, 8, 33, 3000 if products > 10_000 else 5]))
            R[ic].append(len(Arows))
            Arows.append(cols[at:at + m])
            at += m
    nf = len(Arows)

    def csr(rows):
        ia = np.r_[0, np.cumsum([len(r) for r in rows])].astype(np.int32)
        ja = np.concatenate([np.asarray(r, np.int32) for r in rows] + [np.zeros(0, np.int32)])
        return ia, ja.astype(np.int32), rng.standard_normal(len(ja))

    R, A = csr(R), csr(Arows)
    P = csr([[i] if i < nc else [] for i in range(nf)])
    ref_ = oracle.orc_rap(nc, nf, R, A, P)
    out = amg.DcsrMat()
    amg.load_library().dcsr_rap(C.byref(_dcsr(nc, nf, *R)), C.byref(_dcsr(nf, nf, *A)),
                                C.byref(_dcsr(nf, nc, *P)), C.byref(out))
    got = _out(out)
    for j in range(3):
        assert bits_equal(got[j], ref_[j])
