"""GPU: the batched engine of shifted circuits, which runs every batch that holds an instance
without a reverse sweep: its tile widths, shared prefixes, HBM slots and energy windows,
against the oracle and against the sweep.  One more instance, with a parameter that turns two
gates, keeps the batches here off the sweep; that another engine answered shows in the last
digits."""
import os

import numpy as np
import pytest

import oracle
from logosq_b200 import abi, workloads
from logosq_b200._lib import call
from logosq_b200.batch import BatchedParameterShift
from test_gpu_batch import _random_observable

pytestmark = pytest.mark.gpu
BAR = 1e-10


def twice_used():
    g = abi.empty_gates(2)
    g["kind"] = abi.RY
    g["q"][:, 0] = [0, 1]
    g["param"][:, 0] = 0
    return (5, g, 1, workloads.heisenberg_terms(5, [0.5] * 4, [0.4] * 4, [0.3] * 4, 0.2))


def chains(recs, layers=4):
    return [(r["n"], workloads.basic_entangling_template(r["n"], layers), 2 * layers * r["n"],
             workloads.heisenberg_terms(r["n"], r["jx"], r["jy"], r["jz"], r["h"])) for r in recs]


def run(specs, theta, tile_bits=0, shifted=True, prefixes=True, calls=1):
    """Energies and gradients of the specs, the extra instance's left out."""
    old = os.environ.get("LQ_BATCH_PREFIX")
    os.environ["LQ_BATCH_PREFIX"] = "1" if prefixes else "0"
    try:
        b = BatchedParameterShift(specs + [twice_used()] if shifted else specs)
    finally:
        if old is None:
            del os.environ["LQ_BATCH_PREFIX"]
        else:
            os.environ["LQ_BATCH_PREFIX"] = old
    if tile_bits:
        call("lq_batch_set_tile_bits", b._h, tile_bits)
    for _ in range(calls):
        e, g = b.gradients(np.append(theta, 0.3) if shifted else theta)
    b.close()
    return e[:len(specs)], g[:len(theta)]


def near(got, want):
    assert np.abs(got[0] - want[0]).max() < 1e-12 * max(1.0, np.abs(want[0]).max())
    assert np.abs(got[1] - want[1]).max() < BAR


@pytest.mark.parametrize("tile_bits", [0, 10, 11, 12])
def test_every_tile_width(tile_bits):
    recs = workloads.heisenberg_instances(5, seed=21, n_lo=11, n_hi=15)
    theta = np.concatenate([r["theta"] for r in recs])
    got = run(chains(recs), theta, tile_bits)
    want = run(chains(recs), theta, shifted=False)
    near(got, want)
    assert not np.array_equal(got[1], want[1])  # another engine
    again = run(chains(recs), theta, tile_bits, calls=3)  # (its graph replayed)
    if tile_bits:
        assert np.array_equal(again[1], got[1])


def test_against_the_oracle():
    recs = workloads.heisenberg_instances(5, seed=4, n_lo=6, n_hi=13)
    theta = np.concatenate([r["theta"] for r in recs])
    specs = chains(recs)
    _, g = run(specs, theta)
    off = 0
    for n, gates, count, terms in specs:
        want = oracle.parameter_shift(n, gates, theta[off:off + count], terms)
        assert np.abs(g[off:off + count] - want).max() < BAR
        off += count


@pytest.mark.parametrize("tile_bits", [10, 11, 12])
def test_shared_prefixes_are_bitwise_the_unshared_launch(tile_bits):
    recs = workloads.heisenberg_instances(10, seed=31, n_lo=9, n_hi=15)
    theta = np.concatenate([r["theta"] for r in recs])
    with_, without = (run(chains(recs), theta, tile_bits, prefixes=p) for p in (True, False))
    assert np.array_equal(with_[0], without[0]) and np.array_equal(with_[1], without[1])
    near(with_, run(chains(recs), theta, shifted=False))


@pytest.mark.parametrize("tile_bits", [10, 11, 12])
def test_general_observables(tile_bits):
    """Several terms per X mask, odd Y counts, and Z strings over every tile bit."""
    r = np.random.default_rng(17)
    specs = [(n, workloads.basic_entangling_template(n, 2), 4 * n, _random_observable(n, r))
             for n in (7, 11, 13, 15)]
    theta = r.uniform(-np.pi, np.pi, sum(s[2] for s in specs))
    got = run(specs, theta, tile_bits)
    near(got, run(specs, theta, shifted=False))
    want = oracle.parameter_shift(7, specs[0][1], theta[:28], specs[0][3])
    assert np.abs(got[1][:28] - want).max() < BAR
