"""The expanded 0/1 walk (one column expanded, the others walked): bit-exact
at the edges of its halves, i.e. as the expanded column's ones end inside or at
the end of the first four halves of rows, past the last one the walk takes
(the plain walk then runs), and with the line being a row."""
import numpy as np
import pytest

from superman_b200 import workloads as W

pytestmark = pytest.mark.gpu


def with_column_ones(n, m, seed, p):
    """Bernoulli(p) with exactly m ones in one column, every other line
    holding more where n allows."""
    rng = np.random.default_rng(seed)
    a = (rng.random((n, n)) < p).astype(np.uint8)
    np.fill_diagonal(a, 1)
    c = int(rng.integers(0, n))
    a[:, c] = 0
    a[rng.permutation(n)[:m], c] = 1
    return a


# rows per half: 7 at n = 22, 6 at 23 .. 36; below n = 22 the plain walk runs
@pytest.mark.parametrize("n,m", [(4, 1), (4, 4), (5, 2), (9, 9), (10, 8), (10, 9), (10, 10), (12, 8), (12, 9),
                                 (16, 7), (16, 8), (16, 14), (16, 15), (16, 16), (17, 6), (20, 1), (20, 13),
                                 (20, 14), (20, 15), (20, 20), (22, 1), (22, 7), (22, 8), (22, 14), (22, 15),
                                 (22, 20), (22, 21), (22, 22), (23, 6), (23, 7), (23, 12), (23, 13), (23, 18),
                                 (23, 19), (23, 23), (24, 24), (25, 24), (25, 25)])
def test_expanded_words_bit_exact(spb, oracle, n, m):
    a = with_column_ones(n, m, 100 * n + m, 0.95)
    want = oracle.binary_u128(a)
    assert spb.perm_binary(a).permanent == want
    assert spb.perm_binary(a.T.copy()).permanent == want  # the line is a row


@pytest.mark.parametrize("n", [16, 21, 22, 24, 25])
def test_all_ones_around_the_last_half(spb, n):
    """m = n: within four halves up to n = 24 (6 rows a half there), the plain
    walk past it, and the launch shapes the options allow."""
    import math
    a = np.ones((n, n), dtype=np.uint8)
    assert spb.perm_binary(a).permanent == math.factorial(n)
    assert spb.perm_binary(a, unit_bits=3, threads_per_block=64, blocks=5).permanent == math.factorial(n)


@pytest.mark.parametrize("n", [37, 38, 41])
def test_wide_accumulators_closed_form(spb, n):
    """Block diagonal of all-ones blocks at sizes with 5-row halves and more
    than four limbs."""
    import math
    a = np.zeros((n, n), dtype=np.uint8)
    k = n // 3
    for lo, hi in ((0, k), (k, 2 * k), (2 * k, n)):
        a[lo:hi, lo:hi] = 1
    want = math.factorial(k) ** 2 * math.factorial(n - 2 * k)
    assert spb.perm_binary(a[:, np.random.default_rng(n).permutation(n)]).permanent == want
