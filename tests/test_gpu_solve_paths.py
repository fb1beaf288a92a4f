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
