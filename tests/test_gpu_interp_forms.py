"""Interpolation of matrices that a solver would not build but the reference's
drop-in takes, against the oracle."""
import ctypes as C

import numpy as np
import pytest

from blood_network_b200 import amg
from helpers import bits_equal
from test_gpu_hubs import hub_matrix
from test_gpu_parity import _dcsr, _out

pytestmark = pytest.mark.gpu


def _interp(n, A, S, cf):
    dP = amg.DcsrMat()
    amg.load_library().rs_standard_interpolation(C.byref(_dcsr(n, n, *A)), C.byref(_dcsr(n, n, *S)),
                                                 amg._p(cf), C.byref(dP))
    assert amg.load_library().amg_solver_last_status() == 0
    return _out(dP)


def _rows(ia, ja, val, f):
    """The matrix with every row's entries passed through f(i, columns, values)."""
    out = [f(i, ja[ia[i]:ia[i + 1]], val[ia[i]:ia[i + 1]]) for i in range(len(ia) - 1)]
    return (np.r_[0, np.cumsum([len(c) for c, _ in out])].astype(np.int32),
            np.concatenate([c for c, _ in out]).astype(np.int32),
            np.concatenate([v for _, v in out]))


def _problem(seed):
    # rows of every class: a thread, a warp (over 32 entries; neighbours of over
    # 96), a block (over 32 strong points), hub tables (over 512 entries)
    n, ia, ja, val = hub_matrix(side=40, hubs=(20, 33, 60, 300, 700), weak_hubs=(40, 600), seed=seed)
    rng = np.random.default_rng(seed)
    cf = np.where(rng.random(n) < 0.4, 1, -1).astype(np.int32)
    cf[1600:] = -1  # the hubs are F points
    return n, (ia, ja, val), rng, cf


@pytest.mark.parametrize("which", ["some", "all", "longest"])
def test_columns_held_more_than_once(oracle, which):
    """Entries of A split into up to forty of the same column, in rows of every
    class and in their neighbours' (over 32 entries at one strong point), or in
    the longest row alone."""
    n, A, rng, cf = _problem(5)
    S, _ = oracle.orc_strength(n, *A, 0.25)
    lens = np.diff(A[0])

    def split(i, c, v):
        if which == "longest" and lens[i] < lens.max() or which == "some" and rng.random() > 0.02:
            return c, v
        k = np.where(rng.random(len(c)) < 0.3, rng.integers(2, 41, len(c)), 1)
        at = rng.permutation(k.sum())
        return np.repeat(c, k)[at], np.repeat(v / k, k)[at]

    A2 = _rows(*A, split)
    P, want = _interp(n, A2, S, cf), oracle.orc_interp(n, A2, S, cf)
    for a, b in zip(P, want):
        assert bits_equal(a, b)


def test_strong_points_held_twice(oracle):
    """A strong point held twice has two places in P's row; the terms go to one of
    them, and the column's sum is the oracle's."""
    n, A, rng, cf = _problem(6)
    S = _rows(*oracle.orc_strength(n, *A, 0.25)[0],
              lambda i, c, v: (np.r_[c, c[: i % 3]], np.r_[v, v[: i % 3]]))
    P, want = _interp(n, A, S, cf), oracle.orc_interp(n, A, S, cf)
    assert bits_equal(P[0], want[0]) and bits_equal(P[1], want[1])
    rows = np.repeat(np.arange(n), np.diff(P[0]))
    for a in (P, want):
        a[2][:] = np.bincount(np.unique(rows * n + a[1], return_inverse=True)[1], a[2])[
            np.unique(rows * n + a[1], return_inverse=True)[1]]
    assert np.array_equal(P[2], want[2])


@pytest.mark.parametrize("form", ["order", "extra", "diagonal", "undecided"])
def test_strong_points_unlike_the_row(oracle, form):
    """Strong points in another order than A's entries, some that A has no entry
    for, the point itself among them, points that are neither C nor F."""
    n, A, rng, cf = _problem(7)

    def other(i, c, v):
        if form == "extra":
            more = np.setdiff1d(rng.integers(0, 1600, 3), np.r_[c, A[1][A[0][i]:A[0][i + 1]]])
            c, v = np.r_[c, more], np.r_[v, rng.standard_normal(len(more))]
        if form == "diagonal":
            c, v = np.r_[c, i], np.r_[v, 1.0]
        at = rng.permutation(len(c))
        return c[at], v[at]

    S = _rows(*oracle.orc_strength(n, *A, 0.25)[0], other)
    if form == "undecided":
        cf[rng.random(n) < 0.2] = 0
    P, want = _interp(n, A, S, cf), oracle.orc_interp(n, A, S, cf)
    for a, b in zip(P, want):
        assert bits_equal(a, b)
