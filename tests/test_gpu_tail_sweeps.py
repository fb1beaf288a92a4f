"""The number of sweeps of the reference's slashes and preconditioners is the
call's own: each call on one hierarchy does the sweeps that it asks for,
whatever the calls before it asked for."""
import contextlib
import ctypes as C

import numpy as np
import pytest

from blood_network_b200 import amg
from test_gpu_compat import _dcsr
from test_gpu_solve_paths import TOL, _vascular

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def _hierarchy(n, ia, ja, val, nu, min_size=200, max_levels=20):
    lib = amg.load_library()
    A = _dcsr(ia, ja, val, n)
    d = amg.AmgData()
    d.threshold, d.min_size, d.max_levels, d.nu = 0.25, min_size, max_levels, nu
    d.smoother, d.omega_jacobi, d.coarsening = amg.SMOOTHER_CF_GS, 0.5, amg.COARSEN_PMIS
    lib.amg_build_hierarchy(C.byref(d), C.byref(A))
    assert lib.amg_solver_last_status() == 0, lib.amg_solver_last_error()
    try:
        yield lib, d, A
    finally:
        lib.amg_free(C.byref(d))


def _calls(lib, d, A, nus, f):
    """One slash of each kind per entry of nus on levels 0 and 1, and the
    preconditioners with amg->nu set to it."""
    out = []
    for nu in nus:
        for lev in (0, 1):
            m = d.levels[lev].n
            g = np.random.default_rng(lev).standard_normal(m)
            for call in (lib.amg_backslash, lib.amg_fwdslash):
                x = np.zeros(m)
                call(C.byref(d), lev, amg._p(g), amg._p(x), nu)
                assert lib.amg_solver_last_status() == 0, lib.amg_solver_last_error()
                out.append(x)
        keep, d.nu = d.nu, nu
        g = np.random.default_rng(9).standard_normal(d.levels[0].n)
        for args in ((lib.amg_vcycle_precond, (C.byref(d),)),
                     (lib.amg_ichol_precond, (C.byref(d), C.byref(A), C.byref(f)))):
            x = np.zeros(len(g))
            args[0](*args[1], amg._p(g), amg._p(x))
            assert lib.amg_solver_last_status() == 0, lib.amg_solver_last_error()
            out.append(x)
        d.nu = keep
    return out


# the handle's own number first and last, and between others that come before
# its program exists (the second list) or need more operations than one launch takes
@pytest.mark.parametrize("built, nus", [(1, [1, 2, 1, 40, 1]), (1, [2, 1, 3]), (2, [1, 2, 1])])
@pytest.mark.parametrize("nodes", [2_000, 20_000])
def test_each_call_does_its_own_sweeps(nodes, built, nus, monkeypatch):
    n, ia, ja, val = _vascular(nodes, False)
    got = {}
    for tail in ("1", "0"):
        monkeypatch.setenv("BN_TAIL", tail)
        with _hierarchy(n, ia, ja, val, built) as (lib, d, A):
            f = amg.IcholFactor()
            lib.ichol_compute(C.byref(A), C.byref(f))
            try:
                got[tail] = _calls(lib, d, A, nus, f)
            finally:
                lib.ichol_free(C.byref(f))
    per = len(got["0"]) // len(nus)
    for k, (x, y) in enumerate(zip(got["1"], got["0"])):
        # sums in another order only, nu times the operations of one application
        tol = TOL[amg.PREC_FP64] * max(nus[k // per], 1)
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y), (k // per, k % per)
    # the number matters: two calls that differ in it alone differ
    assert np.linalg.norm(got["0"][0] - got["0"][per]) > 1e-3 * np.linalg.norm(got["0"][0])
