"""GPU: gradients when the reverse sweep has no room for its states (the allocation
limit stands for a full device): the shifted circuits run for that call, the sweep again
once there is room, and what the attempt left behind is not the caller's error."""
import contextlib
import ctypes as C
import math

import numpy as np
import pytest

from logosq_b200 import State, abi, workloads
from logosq_b200._lib import call, lib
from logosq_b200.batch import heisenberg_batch

pytestmark = pytest.mark.gpu
BAR = 1e-10


@contextlib.contextmanager
def limit(nbytes):
    call("lq_set_alloc_limit", C.c_uint64(nbytes))
    try:
        yield
    finally:
        call("lq_set_alloc_limit", C.c_uint64(0))


def quiet():
    return lib().lq_last_error()


def test_plain_gradient_within_the_limit_runs_the_shifted_circuits():
    n = 13
    gates = workloads.basic_entangling_template(n, 1)
    terms = workloads.heisenberg_terms(n, [0.5] * (n - 1), [0.4] * (n - 1), [0.3] * (n - 1), 0.2)
    theta = np.linspace(-2, 2, 2 * n)
    st = State(n)

    def energy(th):
        e = C.c_double()
        call("lq_ansatz_energy", st.handle, abi.gate_ptr(gates), len(gates), abi.f64_ptr(th),
             len(th), abi.term_ptr(terms), len(terms), abi.Y_REFERENCE, C.byref(e))
        return e.value

    def gradient():
        g = np.zeros(len(theta))
        call("lq_parameter_shift", st.handle, abi.gate_ptr(gates), len(gates),
             abi.f64_ptr(theta), len(theta), abi.term_ptr(terms), len(terms), abi.Y_REFERENCE,
             math.pi / 2, abi.f64_ptr(g))
        return g

    rule = np.zeros(len(theta))
    for k in range(len(theta)):
        up, down = theta.copy(), theta.copy()
        up[k] = theta[k] + math.pi / 2
        down[k] = theta[k] - math.pi / 2
        rule[k] = (energy(up) - energy(down)) / 2.0
    State(2).close()  # (clears the thread's error)
    free = gradient()
    with limit(16 << n):  # the handle fits, a second state does not
        within = gradient()
        assert quiet() == b""
    assert np.array_equal(within, rule)  # the same circuits
    assert np.abs(free - rule).max() < BAR
    assert np.array_equal(gradient(), free)
    st.close()


def test_batch_returns_to_the_sweep_when_there_is_room_again():
    recs = workloads.heisenberg_instances(6, seed=3, n_lo=11, n_hi=15)
    theta = np.concatenate([r["theta"] for r in recs])
    with_room = heisenberg_batch(recs)
    e, g = with_room.gradients(theta)
    b = heisenberg_batch(recs)
    with limit(1):
        es, gs = b.gradients(theta)
        assert quiet() == b""
        assert b.tuning()["tile_bits"] in (10, 11, 12)
    assert np.abs(es - e).max() < 1e-12 * max(1.0, np.abs(e).max())
    assert np.abs(gs - g).max() < BAR
    assert not np.array_equal(gs, g)  # (other arithmetic: the shifted circuits)
    e2, g2 = b.gradients(theta)
    assert np.array_equal(e2, e) and np.array_equal(g2, g)
    assert b.tuning()["tile_bits"] == 11
    # a few chains at a time: the same sums
    c = heisenberg_batch(recs)
    with limit((2 * 16 << max(r["n"] for r in recs)) + (1 << 18)):
        e3, g3 = c.gradients(theta)
    assert np.array_equal(e3, e) and np.array_equal(g3, g)
    for x in (with_room, b, c):
        x.close()


def test_the_two_engines_choose_their_widths_independently():
    recs = workloads.heisenberg_instances(3, seed=5, n_lo=13, n_hi=14)
    theta = np.concatenate([r["theta"] for r in recs])
    ref = heisenberg_batch(recs)
    _, g11 = ref.gradients(theta)
    b = heisenberg_batch(recs)
    bad = theta.copy()
    bad[0] = np.nan
    b.gradients(bad)  # the shifted circuits tune their width
    _, g = b.gradients(theta)
    assert b.tuning()["tile_bits"] == 11  # and the sweep keeps its own
    assert np.array_equal(g, g11)
    call("lq_batch_set_tile_bits", b._h, 12)
    assert b.tuning()["tile_bits"] == 12
    call("lq_batch_set_tile_bits", b._h, 0)
    assert b.tuning()["tile_bits"] == 0
    _, g = b.gradients(theta)
    assert np.array_equal(g, g11)
    ref.close()
    b.close()
