"""GPU: Pauli sums whose masks have many terms each: a round's terms shared out among blocks
where there are few tiles (edges: one tile, as many blocks as tiles, a round that no block
shares), sums of one mask on both sides of the line to a sweep; against the oracle, and not
slower than masks that fit no window."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import State, abi
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu


def make(rows):
    terms = np.zeros(len(rows), dtype=abi.TERM_DTYPE)
    for t, (c, x, z) in zip(terms, rows):
        t["coefficient"], t["xmask"], t["zmask"], t["ny"] = c, x, z, bin(x & z).count("1")
    return terms


def energy(st, terms):
    out = C.c_double()
    call("lq_expectation_pauli", st.handle, abi.term_ptr(terms), len(terms), abi.Y_REFERENCE,
         C.byref(out), None)
    return out.value


def check(n, rows):
    terms = make(rows)
    v = random_state(n, n)
    st = State(n)
    st.set_vector(v)
    want = oracle.expectation(v, terms, abi.Y_REFERENCE)
    assert abs(energy(st, terms) - want) < 1e-12 * np.abs(terms["coefficient"]).sum()
    st.close()


@pytest.mark.parametrize("n", [5, 9, 12, 13, 16, 18, 19])
@pytest.mark.parametrize("per_mask", [1, 16, 17, 300])
def test_rounds_shared_out(n, per_mask):
    r = np.random.default_rng(n)
    masks = [0, 1, 6, 9, 15] + [int(x) for x in r.integers(0, 1 << min(n, 8), 6)]
    check(n, [(float(r.normal()), x, int(r.integers(0, 1 << n)))
              for x in masks for _ in range(per_mask)])


@pytest.mark.parametrize("x", [0, 3])
@pytest.mark.parametrize("n,count", [(4, 1000), (8, 2000), (18, 2000), (19, 64), (19, 65),
                                     (20, 32), (20, 33)])
def test_one_mask(n, count, x):
    r = np.random.default_rng(n + count)
    check(n, [(float(r.normal()), x, int(r.integers(0, 1 << n))) for _ in range(count)])


@pytest.mark.parametrize("x", [0, 3, 1 << 6])
@pytest.mark.parametrize("n,count", [(13, 1), (13, 300), (18, 40), (19, 64), (19, 65)])
def test_one_mask_that_fits_beside_masks_that_do_not(n, count, x):
    r = np.random.default_rng(n + count)
    wide = [(float(r.normal()), 1 << 4 | 1 << (n - 1) | k, int(r.integers(0, 1 << n)))
            for k in range(3)]
    check(n, wide[:2] + [(float(r.normal()), x, int(r.integers(0, 1 << n)))
                         for _ in range(count)] + wide[2:])


@pytest.mark.parametrize("n", [13, 14])
def test_masks_of_a_window_are_not_slower_than_masks_that_fit_none(n):
    """16 masks of 400 terms: 0.26 ms in a window's rounds (1.0 ms with a round's terms in one
    block), 0.45 as a sweep per mask."""
    r = np.random.default_rng(n)
    wide = 1 << 4 | 1 << (n - 1)
    near, far = (make([(float(r.normal()), x ^ up, int(r.integers(0, 1 << n)))
                       for x in range(16) for _ in range(400)]) for up in (0, wide))
    st = State(n)
    st.set_vector(random_state(n, n))

    def least(terms):
        energy(st, terms)
        t = []
        for _ in range(10):
            a = time.perf_counter()
            energy(st, terms)
            t.append(time.perf_counter() - a)
        return min(t)

    assert least(near) < least(far)
    st.close()
