"""Device memory that a handle keeps."""
import numpy as np
import pytest

from blood_network_b200 import amg
from test_gpu_solve_paths import _random_spd, _vascular

pytestmark = pytest.mark.gpu


def _used():
    """Bytes in use in the device's stream-ordered pool."""
    import torch
    from cuda.bindings import runtime as rt
    torch.cuda.synchronize()
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    err, used = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    assert err == rt.cudaError_t.cudaSuccess
    return int(used)


def _kept(monkeypatch, own, first, second=None):
    monkeypatch.setenv("BN_IC_OWN", own)
    before = _used()
    s = amg.AMGSolver(*first, min_size=100)
    g = np.random.default_rng(1).standard_normal(first[0])
    s.precond(g)
    if second is not None:
        s.set_matrix(*second[1:])
        s.precond(g)
    kept = _used() - before
    s.close()
    return kept


def test_no_owner_schedule_is_kept_where_the_form_is_not_used(monkeypatch):
    """Rows of over four entries throughout leave the form out: the handle holds
    what it holds with the form switched off; also after a matrix that had it."""
    sparse = _vascular(4_000, False)
    dense = _random_spd(sparse[0], 14, 3)
    _kept(monkeypatch, "1", dense)  # loads the kernels
    assert _kept(monkeypatch, "1", sparse) > _kept(monkeypatch, "0", sparse)
    assert _kept(monkeypatch, "1", dense) == _kept(monkeypatch, "0", dense)
    assert _kept(monkeypatch, "1", sparse, dense) == _kept(monkeypatch, "0", sparse, dense)
