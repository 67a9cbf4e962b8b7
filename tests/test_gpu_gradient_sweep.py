"""GPU: parameter-shift gradients by the reverse sweep, at the sizes where it changes
form (padding below 5 qubits, one warp's tiles, the last one-CTA size, the first tiled
ones) and over the gates its rounds distinguish, against the oracle's shifted circuits.
The bar is the suite's for gradients, 1e-10: the sweep's rounding is some 1e-16 per gate
and inner product, far below it."""
import ctypes as C
import math

import numpy as np
import pytest

import oracle
from logosq_b200 import State, abi, workloads
from logosq_b200._lib import call
from logosq_b200.batch import BatchedParameterShift

pytestmark = pytest.mark.gpu
BAR = 1e-10

ENTANGLERS = {
    "linear": [abi.CNOT, abi.X],
    "diagonal": [abi.CNOT, abi.CZ, abi.CPHASE, abi.RZZ, abi.CRZ],
    "controlled": [abi.CNOT, abi.CRX, abi.CRY, abi.TOFFOLI],
    "pairs": [abi.CNOT, abi.SWAP, abi.RXX, abi.RYY],
}


def ansatz(n, seed, kinds, span=None):
    """Random layers of bound rotations of every kind, runs of them, fixed gates
    between them, and fixed entanglers; returns (gates, parameter count)."""
    r, rows, count = np.random.default_rng(seed), [], 0

    def add(kind, qubits, angles=(), bound=()):
        nonlocal count
        g = abi.empty_gates(1)
        g["kind"] = kind
        g["q"][0, :len(qubits)] = qubits
        g["angle"][0, :len(angles)] = angles
        for k in bound:
            g["param"][0, k] = count
            g["scale"][0, k] = r.uniform(0.5, 2.0)
            count += 1
        rows.append(g)

    for _ in range(3):
        for q in range(n):
            pick = r.integers(6)
            if pick == 0:
                add(abi.U3, [q], r.uniform(0, 3, 3), (0, 1, 2))
            elif pick == 1:
                add(abi.RX, [q], [0.4], (0,))
            elif pick == 2:
                add(abi.RZ, [q], [0.1], (0,))
                add(abi.H, [q])
                add(abi.RY, [q], [0.2], (0,))
            elif pick == 3:
                add(abi.PHASE, [q], [0.3], (0,))
                add(abi.T, [q])
            elif pick == 4:
                add(abi.Y, [q])
                add(abi.U3, [q], r.uniform(0, 3, 3), (1,))
            else:
                add(abi.S, [q])  # a run without a parameter
        for _ in range(n):
            kind = kinds[r.integers(len(kinds))]
            width = {abi.X: 1, abi.TOFFOLI: 3}.get(kind, 2)
            lo = 0 if span is None else int(r.integers(0, n - span + 1))
            near = np.arange(lo, n if span is None else lo + span)
            add(kind, [int(q) for q in r.choice(near, width, replace=False)],
                [] if width != 2 else [float(r.uniform(0, 3))])
    return np.concatenate(rows), count


def observable(n, seed):
    """Odd and even Y counts, several terms per X mask, Z bits anywhere."""
    r, rows = np.random.default_rng(seed), []
    for _ in range(6):
        x = int(r.integers(0, 1 << n))
        for _ in range(3):
            z = int(r.integers(0, 1 << n))
            rows.append((float(r.normal()), x, z, bin(x & z).count("1")))
    rows += [(float(r.normal()), 0, int(r.integers(1, 1 << n)), 0) for _ in range(12)]
    out = np.zeros(len(rows), dtype=abi.TERM_DTYPE)
    for k, (c, x, z, ny) in enumerate(rows):
        out[k]["coefficient"], out[k]["xmask"], out[k]["zmask"], out[k]["ny"] = c, x, z, ny
    return out


def plain(n, gates, theta, terms, shift, conv=abi.Y_REFERENCE):
    st, g = State.zero_state(n), np.zeros(len(theta))
    call("lq_parameter_shift", st.handle, abi.gate_ptr(gates), len(gates), abi.f64_ptr(theta),
         len(theta), abi.term_ptr(terms), len(terms), conv, shift, abi.f64_ptr(g))
    st.close()
    return g


@pytest.mark.parametrize("kinds", sorted(ENTANGLERS))
@pytest.mark.parametrize("n", [3, 5, 6, 9, 12, 13, 15])
def test_plain_gradient_matches_oracle(n, kinds):
    # (a pair further apart than a window runs the shifted circuits: keep some inside)
    gates, count = ansatz(n, n, ENTANGLERS[kinds], span=6 if n > 12 else None)
    theta = np.random.default_rng(n + 7).uniform(-3, 3, count)
    terms = observable(n, n + 1)
    for shift, conv in ((math.pi / 2, abi.Y_REFERENCE), (0.7, abi.Y_TEXTBOOK)):
        got = plain(n, gates, theta, terms, shift, conv)
        want = oracle.parameter_shift(n, gates, theta, terms, shift=shift, y_convention=conv)
        assert np.abs(got - want).max() < BAR


def test_two_qubits_and_an_unused_parameter():
    gates, count = ansatz(2, 5, [abi.CNOT])
    theta = np.random.default_rng(1).uniform(-3, 3, count + 1)
    terms = observable(2, 3)
    got = plain(2, gates, theta, terms, 0.3)
    assert np.abs(got - oracle.parameter_shift(2, gates, theta, terms, shift=0.3)).max() < BAR
    assert got[-1] == 0.0


@pytest.mark.parametrize("kind", [abi.CRX, abi.CPHASE, abi.RZZ])
def test_circuits_without_a_sweep_keep_the_shifted_circuits(kind):
    """A bound two-qubit gate, and a parameter used twice."""
    n = 6
    g = workloads.basic_entangling_template(n, 2).copy()
    two = np.nonzero(g["kind"] == abi.CNOT)[0][2]
    g["kind"][two] = kind
    g["param"][two, 0] = 4 * n
    g["param"][np.nonzero(g["kind"] == abi.RY)[0][-1], 0] = 0
    theta = np.random.default_rng(2).uniform(-3, 3, 4 * n + 1)
    terms = observable(n, 9)
    got = plain(n, g, theta, terms, math.pi / 2)
    assert np.abs(got - oracle.parameter_shift(n, g, theta, terms)).max() < BAR


@pytest.mark.parametrize("tile_bits", [10, 11, 12])
def test_batch_sweep_matches_the_shifted_circuits(tile_bits):
    """One more instance that has no sweep (a parameter used twice) sends the whole
    batch through the shifted circuits; the others' results agree, at every width."""
    specs, thetas = [], []
    for n in (5, 8, 11, 12, 13, 14, 16):
        gates = workloads.basic_entangling_template(n, 2)
        terms = workloads.heisenberg_terms(n, *np.random.default_rng(n).uniform(-1, 1, (3, n - 1)),
                                           0.3)
        specs.append((n, gates, 4 * n, terms))
        thetas.append(np.random.default_rng(n).uniform(-np.pi, np.pi, 4 * n))
    twice = specs[0][1].copy()
    twice["param"][np.nonzero(twice["kind"] == abi.RY)[0][-1], 0] = 0
    res = []
    for extra in (False, True):
        b = BatchedParameterShift(specs + ([(5, twice, 20, specs[0][3])] if extra else []))
        call("lq_batch_set_tile_bits", b._h, tile_bits)
        e, g = b.gradients(np.concatenate(thetas + ([thetas[0]] if extra else [])))
        res.append((e[:len(specs)], g[:sum(map(len, thetas))]))
        assert b.tuning()["tile_bits"] == tile_bits
        b.close()
    assert np.abs(res[0][0] - res[1][0]).max() < 1e-12 * max(1.0, np.abs(res[1][0]).max())
    assert np.abs(res[0][1] - res[1][1]).max() < BAR


def test_non_finite_parameters_give_what_the_rule_gives():
    n = 5
    gates = workloads.basic_entangling_template(n, 1)
    terms = workloads.heisenberg_terms(n, [0.5] * 4, [0.4] * 4, [0.3] * 4, 0.2)
    theta = np.linspace(-1, 1, 2 * n)
    theta[3] = np.nan
    assert np.all(np.isnan(plain(n, gates, theta, terms, math.pi / 2)))
