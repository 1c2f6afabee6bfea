"""The row-by-row expansion of sparse matrices (expand_rows) on the GPU: bands,
whose width fixes the number of open columns, against an exact integer
evaluation; cancelling and structurally zero permanents; and the walk in its
place when its tables cannot be allocated."""
import numpy as np
import pytest

from superman_b200 import _lib
from superman_b200 import workloads as W

pytestmark = pytest.mark.gpu


def band(n, width, seed, signed=True):
    """Row i holds integers of 1..5, with signs,, in `width` columns around
    the diagonal (fewer at the ends)."""
    rng = np.random.default_rng(seed)
    a = np.zeros((n, n))
    for i in range(n):
        for j in range(max(0, min(i - width // 2, n - width)), min(n, i - width // 2 + width)):
            a[i, j] = rng.integers(1, 6) * (rng.choice((-1, 1)) if signed else 1)
    return a


def exact(a):
    """Exact integer permanent, row by row over the sets of used columns."""
    n = a.shape[0]
    last = [max(np.nonzero(a[:, j])[0]) for j in range(n)]
    sets = {0: 1}
    for i in range(n):
        closed = sum(1 << j for j in range(n) if last[j] == i)
        nz = [(1 << int(j), int(a[i, j])) for j in np.nonzero(a[i])[0]]
        out = {}
        for s, v in sets.items():
            for bit, x in nz:
                if not s & bit:
                    t = s | bit
                    out[t] = out.get(t, 0) + v * x
        sets = {s: v for s, v in out.items() if v and s & closed == closed}
    return sets.get((1 << n) - 1, 0)


def shuffled(a, seed):
    rng = np.random.default_rng(seed)
    return np.ascontiguousarray(a[rng.permutation(a.shape[0])][:, rng.permutation(a.shape[0])])


@pytest.mark.parametrize("n,width", [(34, 2), (34, 5), (34, 10), (36, 11), (36, 12), (33, 13), (33, 14), (32, 15),
                                     (63, 6), (27, 3)])
def test_bands_against_exact(spb, n, width):
    """Widths on both sides of the steps one CTA takes alone (11 open columns) and
    of what one cluster takes (13): two CTAs, clusters of four and eight, the
    cooperative grid; from 12 on a half has no narrow step left at its cut."""
    for signed in (False, True):
        a = band(n, width, 10 * n + width, signed)
        want = exact(a)
        r = spb.perm_sparse(shuffled(a, n))
        assert r.launches == 1 and r.active_rows < n
        got = r.permanent + r.permanent_lo
        # a few roundings of 2^-104 per row and state, of sums of terms of either
        # sign; got itself is a double
        terms = exact(np.abs(a))
        assert abs(got - want) <= 2.0 ** -52 * abs(want) + 4 * n * 2.0 ** -104 * terms, (got, want)
        assert 0.0 < r.err_est < np.inf


def test_heavy_cancellation(spb):
    """Two nearly equal products: 14 digits cancel, the rest is there."""
    n = 28
    a = np.eye(n)
    a[:, :] += np.eye(n, k=1)
    a[n - 1, 0] = -1.0 + 2.0 ** -46  # perm = 1 + a[n-1,0] = 2^-46
    r = spb.perm_sparse(shuffled(a, 3))
    assert r.launches == 1 and r.permanent == 2.0 ** -46 and 0.0 < r.err_est < 1e-6


def test_zero_by_cancellation_and_by_structure(spb):
    """A permanent that cancels to zero has no relative error to state; one whose
    pattern holds no perfect matching is zero exactly."""
    n = 26
    a = np.eye(n) + np.eye(n, k=1)
    a[n - 1, 0] = -1.0
    r = spb.perm_sparse(shuffled(a, 4))
    assert r.launches == 1 and r.permanent == 0.0 and r.err_est == np.inf
    b = W.sparse_perm_plus(n, 5)
    b[3, :] = 0.0
    b[3, 7] = 1.0
    b[9, :] = 0.0
    b[9, 7] = 2.0  # two rows with one column between them
    r = spb.perm_sparse(b)
    assert r.launches == 1 and r.permanent == 0.0 and r.err_est == 0.0


@pytest.mark.parametrize("n,extra", [(22, 2), (24, 3), (28, 3)])
def test_walk_runs_when_the_tables_do_not_fit(spb, n, extra):
    a = W.sparse_perm_plus(n, 7, extra=extra)
    r = spb.perm_sparse(a, precision="dd")
    assert r.launches == 1
    _lib.lib().spb_debug_fail_allocations(1)
    try:
        w = spb.perm_sparse(a, precision="dd")
    finally:
        _lib.lib().spb_debug_fail_allocations(0)
    assert w.launches > 1
    assert abs(w.permanent - r.permanent) <= 1e-12 * abs(r.permanent)
