"""The drop-in right-hand side on arrays large enough for the threaded copies
(8 MB in all; fields of more than one 1 MB piece, with a remainder): against
the oracle, and from two threads at once, each with a pool of pieces."""
import threading

import numpy as np
import pytest

import oracle as O
from amss_b200 import dropin

from helpers import generic_state, relerr

pytestmark = pytest.mark.gpu


def _inputs(ex, seed):
    X = [-2.0 + (np.arange(n) + 0.5) * 0.1 for n in ex]
    return X, generic_state(*X, seed=seed, amp=0.5)


@pytest.fixture(scope="module", autouse=True)
def pools():
    """A pool is made once 256 MB have been copied for want of one: two threads
    copy 104 MB a call until there are two."""
    X, st = _inputs((54, 53, 51), 3)

    def go():
        for _ in range(8):
            dropin.compute_rhs_bssn(*X, st, eps=0.1, co=0)

    threads = [threading.Thread(target=go) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()


def test_smallest_threaded_call_equals_the_plain_copies():
    """30,996 points, 8.4 MB in: the entry that allocates nothing runs the same
    kernel over plain copies."""
    X, st = _inputs((27, 28, 41), 3)
    got = dropin.compute_rhs_bssn(*X, st, eps=0.1, co=0)
    ref = dropin.compute_rhs_bssn_noalloc(*X, st, eps=0.1, co=0)
    assert got[0] == ref[0] == 0
    for g, r in zip(got[1:], ref[1:]):
        assert np.array_equal(g, r)


def test_large_block_matches_the_oracle():
    """Fields of 1.17 MB.  The bar of test_gpu_bssn_rhs.py, 1e-12 at spacings of
    0.25, scaled to 0.1: what rounds is a second derivative, whose weights grow
    as 1/dx^2, so (0.25 / 0.1)^2 = 6.25 times it."""
    X, st = _inputs((54, 53, 51), 3)
    ref = O.compute_rhs_bssn(X[0], X[1], X[2], st, eps=0.1, co=0)
    got = dropin.compute_rhs_bssn(X[0], X[1], X[2], st, eps=0.1, co=0)
    assert got[0] == ref[0] == 0
    for r, g in zip(ref[1:], got[1:]):
        for f in range(r.shape[0]):
            assert relerr(g[f], r[f]) <= 6.25e-12, f


def test_two_threads_at_once():
    cases = [_inputs((54, 53, 51), s) for s in (3, 4)]
    serial = [dropin.compute_rhs_bssn(*X, st, eps=0.1, co=0) for X, st in cases]
    got = [None, None]

    def go(m):
        for _ in range(3):
            got[m] = dropin.compute_rhs_bssn(*cases[m][0], cases[m][1], eps=0.1, co=0)

    threads = [threading.Thread(target=go, args=(m,)) for m in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, serial):
        for x, y in zip(a[1:], b[1:]):
            assert np.array_equal(x, y)
