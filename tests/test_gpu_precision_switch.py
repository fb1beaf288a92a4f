"""Handles that change precision between changes of their values."""
import numpy as np
import pytest

from blood_network_b200 import amg
from test_gpu_solve_paths import OWN_CASES, _random_spd, _vascular

pytestmark = pytest.mark.gpu

VASCULAR = _vascular(4_000, False)


def _scaled(ia, ja, val, seed):
    """Other conductances on the same segments, the ground conductances kept."""
    import scipy.sparse as sp
    n = len(ia) - 1
    A = sp.csr_matrix((val, ja, ia), shape=(n, n))
    d = np.random.default_rng(seed).uniform(0.2, 5.0, n)
    W = sp.diags(d) @ (A - sp.diags(A.diagonal())) @ sp.diags(d)
    B = (sp.diags(A @ np.ones(n) - np.asarray(W.sum(1)).ravel()) + W).tocsr()
    B.sort_indices()
    assert np.array_equal(B.indices, ja)
    return ia, ja, B.data


@pytest.mark.parametrize("change", ["update", "set_matrix"])
def test_values_changed_between_the_precisions(change):
    """FP64, mixed, FP64, new values, mixed again: the FP32 factor is that of the
    new values, as in a handle that was mixed throughout (bit for bit)."""
    n, ia, ja, val = VASCULAR
    # another matrix may have another pattern, here a longer one
    new = _scaled(ia, ja, val, 3) if change == "update" else _random_spd(n, 12, 4)[1:]
    g = np.random.default_rng(1).standard_normal(n)
    s = amg.AMGSolver(n, ia, ja, val, min_size=200)
    s.set_precision(amg.PREC_MIXED)
    s.precond(g)
    s.set_precision(amg.PREC_FP64)
    s.precond(g)
    getattr(s, change)(*new)
    s.set_precision(amg.PREC_MIXED)
    x = s.precond(g)
    s.close()
    s = amg.AMGSolver(n, ia, ja, val, min_size=200, precision=amg.PREC_MIXED)
    getattr(s, change)(*new)
    y = s.precond(g)
    s.close()
    assert x.tobytes() == y.tobytes() and np.isfinite(x).all()


def test_fp32_timing_between_fp64_solves():
    """The FP32 kernels of an FP64 handle timed after new values: the solves before
    and after agree (the timing makes FP32 copies, the solve's graph stays right)."""
    n, ia, ja, val = VASCULAR
    b = np.random.default_rng(2).standard_normal(n)
    s = amg.AMGSolver(n, ia, ja, val, min_size=200)
    s.bench_kernel(3, precision=1, reps=1)
    s.update(*_scaled(ia, ja, val, 5))
    x = s.solve(b, tol=1e-8)
    s.bench_kernel(3, precision=1, reps=1)
    junk = [np.zeros(n) for _ in range(4)]
    other = amg.AMGSolver(n, ia, ja, val, min_size=200)  # takes freed memory over
    other.precond(junk[0])
    y = s.solve(b, tol=1e-8)
    other.close()
    s.close()
    assert x[1] == y[1] and x[0].tobytes() == y[0].tobytes()


def _sweep_kernels(s, g):
    """Names of the IC(0) sweep kernels of one preconditioner application."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        x = s.precond(g)
        torch.cuda.synchronize()
    return x, {e.name for e in p.events() if "k_tri_" in e.name}


def test_owner_sweeps_in_the_precision_at_hand():
    """The sweeps that keep rows by their blocks serve a handle in either precision,
    whichever it was made in, and after a new smoother or new values; the results
    are the chunked sweeps' bits, as in a handle made in that precision."""
    n, ia, ja, val = VASCULAR
    g = np.random.default_rng(3).standard_normal(n)
    want = {}
    for p in (amg.PREC_FP64, amg.PREC_MIXED):
        s = amg.AMGSolver(n, ia, ja, val, min_size=200, precision=p)
        want[p] = s.precond(g).tobytes()
        s.close()

    def check(s, p):
        x, names = _sweep_kernels(s, g)
        assert x.tobytes() == want[p]
        kind = "k_tri_own<double" if p == amg.PREC_FP64 else "k_tri_own<float"
        assert names and all(kind in m for m in names), names

    for first, second in ((amg.PREC_MIXED, amg.PREC_FP64), (amg.PREC_FP64, amg.PREC_MIXED)):
        s = amg.AMGSolver(n, ia, ja, val, min_size=200, precision=first)
        check(s, first)
        s.set_precision(second)
        check(s, second)
        s.set_smoother(amg.SMOOTHER_GS)
        s.set_smoother(amg.SMOOTHER_CF_GS)
        check(s, second)
        s.update(ia, ja, val)
        s.set_precision(first)
        check(s, first)
        s.bench_kernel(3, precision=1, reps=1)
        check(s, first)
        s.close()


@pytest.mark.parametrize("precision", [amg.PREC_FP64, amg.PREC_MIXED])
@pytest.mark.parametrize("name", sorted(OWN_CASES))
def test_owner_schedule_over_smoothers(name, precision, monkeypatch):
    """A new smoother numbers the vectors anew; the sweeps' schedule stays and gives
    the chunked sweeps' bits after each change."""
    n, ia, ja, val = OWN_CASES[name]()
    g = np.random.default_rng(n).standard_normal(n)
    out = {}
    for own in "10":
        monkeypatch.setenv("BN_IC_OWN", own)
        s = amg.AMGSolver(n, ia, ja, val, precision=precision, min_size=30)
        out[own] = []
        for smoother in (amg.SMOOTHER_GS, amg.SMOOTHER_JACOBI, amg.SMOOTHER_CF_GS):
            s.set_smoother(smoother)
            out[own].append(s.precond(g).tobytes())
        s.close()
    assert out["1"] == out["0"] and len(set(out["1"])) == 3
