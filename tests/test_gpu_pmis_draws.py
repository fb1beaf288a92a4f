"""pmis_coarsening on both sides of the size from which its draws are made on the
device: the split is the oracle's and the C library is left behind n draws."""
import ctypes as C

import numpy as np
import pytest

from blood_network_b200 import amg
from test_gpu_parity import _dcsr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 40_000, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_pmis_split_and_rand_state(oracle, n):
    # a ring with strong neighbours; one point alone for n = 1
    i = np.arange(n, dtype=np.int64)
    k = 2 if n > 1 else 0
    ia = (np.arange(n + 1) * k).astype(np.int32)
    ja = (np.stack([(i - 1) % n, (i + 1) % n], 1).ravel()[: n * k]).astype(np.int32)
    S = (ia, ja, -np.ones(len(ja)))
    libc = C.CDLL(None)
    cf_ref, _ = oracle.orc_split(n, *S, "pmis")
    want = [libc.rand() for _ in range(2)]
    libc.srand(99)
    cf, nc = np.zeros(n, np.int32), C.c_int()
    amg.load_library().pmis_coarsening(C.byref(_dcsr(n, n, *S)), amg._p(cf), C.byref(nc))
    assert amg.load_library().amg_solver_last_status() == 0
    assert want == [libc.rand() for _ in range(2)]
    assert np.array_equal(cf, cf_ref) and nc.value == (cf == 1).sum()
