"""The derivative walk (rows divided by a pivot column, half the subsets) and
the plain walk it falls back to when every column holds a zero: both against
the exact permanent, at the smallest sizes, with the pivot at either end, with
pivots far from the rows' maxima, and over each way units are listed for the
double-double refinement."""
import ctypes

import numpy as np
import pytest

from superman_b200 import _lib
from superman_b200 import workloads as W

pytestmark = pytest.mark.gpu


_exact = {}


def EXACT(oracle, a):
    """The oracle's exact value, kept per matrix (seconds each at n = 24)."""
    k = a.tobytes()
    if k not in _exact:
        _exact[k] = oracle.exact_perm_complex(a) if np.iscomplexobj(a) else oracle.exact_perm(a)
    return _exact[k]


def full(r):
    return r.permanent + r.permanent_lo


def no_pivot(a, seed):
    """One zero in every column, at different rows: no column can be divided by."""
    a = a.copy()
    n = a.shape[0]
    a[np.random.default_rng(seed).permutation(n), np.arange(n)] = 0.0
    return a


def only_pivot(a, c, seed):
    """Column c is the only one without a zero."""
    b = no_pivot(a, seed)
    b[:, c] = a[:, c] + 0.25
    return b


@pytest.mark.parametrize("small_call", [0, -1])
@pytest.mark.parametrize("precision", ["fp64", "dd"])
@pytest.mark.parametrize("n", [23, 24])
def test_real_pivot_and_no_pivot(spb, oracle, n, precision, small_call):
    u = W.dense_uniform(n, 40 + n)
    for a in (u, no_pivot(u, n), only_pivot(u, 0, n), only_pivot(u, n - 1, n)):
        r = spb.perm_dense(a, precision=precision, small_call=small_call, sparse_walk=1)
        # FP64 products in an alternating sum: kappa sqrt(n/6) 2^-52, kappa about 2e2
        assert oracle.rel_err(full(r), EXACT(oracle, a)) <= (4e-13 if precision == "fp64" else 2e-13)


@pytest.mark.parametrize("precision", ["fp64", "dd"])
@pytest.mark.parametrize("n", [21, 22])
def test_complex_pivot_and_no_pivot(spb, oracle, n, precision):
    u = W.haar_block(n, 60 + n, N=64)
    for a in (u, no_pivot(u, n), only_pivot(u, 0, n)):
        er, ei = EXACT(oracle, a)
        r = spb.perm_complex(a, precision=precision)
        scale = float(np.prod(np.abs(a).sum(axis=1)))
        assert abs(r.permanent - complex(float(er), float(ei))) <= 1e-14 * scale


def test_pivots_far_from_the_row_maxima(spb, oracle):
    """A small entry in every column: quotients up to 2^30 times the row's scale
    keep the range (derivative walk).  Rows 2^-50 outside one entry: products of
    quotients would reach 2^1100, and the plain walk runs."""
    n = 24
    u = W.dense_uniform(n, 5) + 0.5
    one = np.eye(n, dtype=bool)
    for a in (np.where(one, u * 2.0 ** -30, u), np.where(one, u, u * 2.0 ** -50)):
        for small_call in (0, -1):
            r = spb.perm_dense(a, precision="dd", small_call=small_call)
            assert oracle.rel_err(full(r), EXACT(oracle, a)) <= 2e-13


def two_permutations(n, background, seed):
    """Two permutations of entries near 1 over a small background."""
    rng = np.random.default_rng(seed)
    a = background * (0.5 + rng.random((n, n)))
    p = rng.permutation(n)
    for s in (0, 1):
        a[np.arange(n), np.roll(p, s)] = 0.5 + rng.random(n)
    return a


@pytest.mark.parametrize("small_call", [0, -1])
@pytest.mark.parametrize("background", [1e-3, 1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9])
def test_wide_range_is_refined(spb, oracle, background, small_call):
    """Quotients by entries of the background reach 2^13 to 2^33, products of
    them 2^360 to 2^800: the refinement, which squares them, still has finite
    sums to choose its units by, whichever walk that takes.  (These matrices
    hardly cancel: only a tight tolerance asks for refined units.)"""
    a = two_permutations(24, background, 7)
    r = spb.perm_dense(a, precision="dd", small_call=small_call, rel_tol=1e-16)
    assert 0.0 < r.err_est <= 1e-16 and r.refined_units > 0
    assert oracle.rel_err(full(r), EXACT(oracle, a)) <= 1e-15  # a few times the tolerance and full's rounding


@pytest.mark.parametrize("background", [1e-3, 1e-5, 1e-6, 1e-7])
def test_wide_range_is_refined_n28(spb, background):
    a = two_permutations(28, background, 8)
    r = [spb.perm_dense(np.ascontiguousarray(m), precision="dd", rel_tol=1e-16) for m in (a, a.T)]
    for x in r:
        assert 0.0 < x.err_est <= 1e-16 and x.refined_units > 0
    assert abs(full(r[0]) - full(r[1])) <= 2e-15 * abs(full(r[0]))


@pytest.mark.parametrize("background", [1e-6, 1e-8])
def test_wide_range_is_refined_complex(spb, oracle, background):
    n = 22
    rng = np.random.default_rng(9)
    a = two_permutations(n, background, 9) * np.exp(2j * np.pi * rng.random((n, n)))
    er, ei = EXACT(oracle, a)
    ex = complex(float(er), float(ei))
    r = spb.perm_complex(a, precision="dd", rel_tol=1e-16)
    # (the plain walk at this size meets the cap of an eighth of the units, and
    # the rest leaves 1.1e-15 by the estimate)
    assert 0.0 < r.err_est <= 2e-15 and r.refined_units > 0
    assert abs(r.permanent - ex) <= 4.0 * r.err_est * abs(ex)


@pytest.mark.parametrize("exp", [-300, -600])
@pytest.mark.parametrize("n", [11, 22])
def test_complex_tiny_pivot(spb, oracle, n, exp):
    """One entry of 2^-300 or 2^-600 in the only column without a zero: its
    square leaves the FP64 range, its quotients do not.  n = 11 as a batch of one,
    n = 22 as a whole-GPU call."""
    import torch
    a = only_pivot(W.haar_block(n, 5 + n, N=64), 3, n)
    a[n // 2, 3] *= 2.0 ** exp
    er, ei = EXACT(oracle, a)
    if n <= 20:
        d = torch.from_numpy(a.view(np.float64)).cuda()
        out = torch.zeros(4, dtype=torch.float64, device="cuda")
        _lib.check(_lib.lib().spb_perm_batch_dev(ctypes.c_void_p(d.data_ptr()), n, 1, 1,
                                                 ctypes.c_void_p(out.data_ptr()), None))
        torch.cuda.synchronize()
        got = complex(float(out[0]), float(out[2]))
    else:
        got = spb.perm_complex(a, precision="fp64").permanent
    scale = float(np.prod(np.abs(a).sum(axis=1)))
    assert abs(got - complex(float(er), float(ei))) <= 1e-14 * scale


@pytest.mark.parametrize("pivot", [True, False])
def test_refinement_listings_agree(spb, oracle, pivot):
    """Many units refined (signed entries, tight tolerance): the first pass's
    list, the fused call's list and the replay select the same units."""
    a = np.random.default_rng(5).standard_normal((24, 24))
    if not pivot:
        a = no_pivot(a, 7)
    kw = dict(precision="dd", rel_tol=1e-16, sparse_walk=1)
    exact = EXACT(oracle, a)
    rs = [spb.perm_dense(a, small_call=0, **kw), spb.perm_dense(a, small_call=-1, **kw),
          spb.perm_dense(a, replay_listing=1, **kw)]
    assert rs[0].refined_units == rs[1].refined_units == rs[2].refined_units > 0
    for r in rs:
        assert oracle.rel_err(full(r), exact) <= 1e-12


def test_complex_refinement_listings_agree(spb, oracle):
    rng = np.random.default_rng(8)
    a = rng.standard_normal((22, 22)) + 1j * rng.standard_normal((22, 22))
    er, ei = EXACT(oracle, a)
    ex = complex(float(er), float(ei))
    r1 = spb.perm_complex(a, precision="dd", rel_tol=1e-16)
    r2 = spb.perm_complex(a, precision="dd", rel_tol=1e-16, replay_listing=1)
    assert r1.refined_units == r2.refined_units > 0
    assert abs(r1.permanent - ex) <= 1e-13 * abs(ex) and abs(r2.permanent - ex) <= 1e-13 * abs(ex)


@pytest.mark.parametrize("n", [30, 31])
def test_bound_pass_sizes(spb, n):
    """n = 30 (2^20 units: every unit listed, the bound pass ends at once) and
    31 (listed from the bound pass's bin): the transpose agrees."""
    a = W.dense_uniform(n, 300 + n)
    r1 = spb.perm_dense(a, precision="dd")
    r2 = spb.perm_dense(np.ascontiguousarray(a.T), precision="dd")
    assert r1.refined_units > 0
    assert abs(full(r1) - full(r2)) <= 3e-13 * abs(full(r1))  # as the n = 32 transpose test


@pytest.mark.parametrize("n", [10, 11, 12, 16, 18])
@pytest.mark.parametrize("cplx", [False, True])
def test_batch_mixes_both_walks(spb, oracle, n, cplx):
    """Matrices with and without a pivot in one launch, each on one warp or
    (n >= 16, a launch this small) shared by the CTAs of a cluster."""
    import torch
    mats = []
    for k in range(9):
        u = W.haar_block(n, 900 + k, N=64) if cplx else W.dense_uniform(n, 900 + k)
        mats.append(u if k % 3 == 0 else no_pivot(u, k) if k % 3 == 1 else only_pivot(u, k % n, k))
    m = np.ascontiguousarray(np.stack(mats))
    d = torch.from_numpy(m.view(np.float64)).cuda()
    c = 2 if cplx else 1
    out = torch.full((len(mats), c, 2), float("nan"), dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().spb_perm_batch_dev(ctypes.c_void_p(d.data_ptr()), n, int(cplx), len(mats),
                                             ctypes.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    for k, a in enumerate(mats):
        scale = float(np.prod(np.abs(a).sum(axis=1)))
        if cplx:
            er, ei = EXACT(oracle, a)
            assert abs(complex(o[k, 0, 0], o[k, 1, 0]) - complex(float(er), float(ei))) <= 1e-14 * scale
        else:
            assert oracle.rel_err(o[k, 0, 0], EXACT(oracle, a)) <= 1e-13


@pytest.mark.parametrize("n,cplx", [(16, False), (19, False), (21, True), (24, False), (24, True)])
def test_batch_split_is_the_same_as_alone(spb, n, cplx):
    """A launch of few matrices splits each over a cluster, a launch of many
    gives each a warp: the same values."""
    import torch
    few, many = 2, 600 if n <= 21 else 470
    u = [W.haar_block(n, 40 + k, N=64) if cplx else W.dense_uniform(n, 40 + k) for k in range(few)]
    got = []
    for count in (few, many):
        m = np.ascontiguousarray(np.stack([u[k % few] for k in range(count)]))
        d = torch.from_numpy(m.view(np.float64)).cuda()
        out = torch.zeros((count, 2 if cplx else 1, 2), dtype=torch.float64, device="cuda")
        _lib.check(_lib.lib().spb_perm_batch_dev(ctypes.c_void_p(d.data_ptr()), n, int(cplx), count,
                                                 ctypes.c_void_p(out.data_ptr()), None))
        torch.cuda.synchronize()
        got.append(out.cpu().numpy())
    for k in range(many):
        a, b = got[0][k % few, :, 0], got[1][k, :, 0]
        assert np.all(np.abs(a - b) <= 2.0 ** -52 * np.abs(a)), (k, a, b)


@pytest.mark.parametrize("n,cplx", [(16, False), (16, True), (17, False), (18, True)])
def test_batch_counts_around_the_split(spb, n, cplx):
    """Launches of 1 to 2400 matrices, i.e. clusters of eight, four and two CTAs,
    a CTA each (with more CTAs than SMs, too) and a warp each: the same values; a
    matrix of zeros, which takes no walk, gives 0 in each."""
    import torch
    few = 3
    u = [W.haar_block(n, 60 + k, N=64) if cplx else W.dense_uniform(n, 60 + k) for k in range(few)]
    first = None
    for count in (1, 5, 20, 100, 600, 2400):
        m = np.ascontiguousarray(np.stack([u[k % few] for k in range(count)]))
        m[count // 2] *= 0.0 if count > 1 else 1.0
        d = torch.from_numpy(m.view(np.float64)).cuda()
        out = torch.full((count, 2 if cplx else 1, 2), 7.0, dtype=torch.float64, device="cuda")
        _lib.check(_lib.lib().spb_perm_batch_dev(ctypes.c_void_p(d.data_ptr()), n, int(cplx), count,
                                                 ctypes.c_void_p(out.data_ptr()), None))
        torch.cuda.synchronize()
        o = out.cpu().numpy()
        if count > 1:
            assert np.all(o[count // 2] == 0.0)
        for k in range(count):
            if count > 1 and k == count // 2:
                continue
            if k < few and (first is None or k not in first):
                first = {**(first or {}), k: o[k, :, 0]}
            a = first[k % few]
            assert np.all(np.abs(a - o[k, :, 0]) <= 2.0 ** -52 * np.abs(a)), (count, k)


def test_launch_shapes_that_only_the_plain_walk_fits(spb):
    """Shapes whose shared memory holds the plain walk but not the derivative
    walk's low words beside it: accepted, on the plain walk (real n=24 with 2^10
    terms at 128 threads 228160 B against 230272 B of 228352; complex n=24 with 2^8
    terms, whose refinement takes 218752 B against 229888 B)."""
    a = W.dense_uniform(24, 12)
    want = spb.perm_dense(a).permanent
    r = spb.perm_dense(a, unit_bits=10, threads_per_block=128, small_call=-1)
    assert abs(r.permanent - want) <= 1e-12 * abs(want)
    c = W.haar_block(24, 13, N=64)
    want = spb.perm_complex(c, precision="dd").permanent
    r = spb.perm_complex(c, precision="dd", unit_bits=8)
    assert abs(r.permanent - want) <= 1e-12 * abs(want)


def test_fused_call_keeps_its_unit_width(spb):
    """n = 26 without a pivot: 2^8 terms a unit, the fused call's 2^17 units in two
    passes (narrower units would take more, each with bases of its own)."""
    a = no_pivot(W.dense_uniform(26, 2), 2)
    r, s = (spb.perm_dense(a, precision="dd", sparse_walk=1, unit_bits=b) for b in (0, 8))
    assert (r.permanent, r.permanent_lo, r.refined_units) == (s.permanent, s.permanent_lo, s.refined_units)


def test_noalloc_without_a_pivot(spb):
    import torch
    a = no_pivot(W.dense_uniform(24, 3), 4)
    d = torch.from_numpy(a).cuda()
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    _lib.check(_lib.lib().spb_perm_dense_f64_noalloc(ctypes.c_void_p(d.data_ptr()), 24,
                                                     ctypes.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    want = spb.perm_dense(a, small_call=-1, sparse_walk=1).permanent
    assert abs(float(out[0]) - want) <= 1e-13 * abs(want)
