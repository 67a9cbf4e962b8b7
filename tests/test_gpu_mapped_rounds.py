"""GPU: fused circuits as mapped rounds, where the planner and the kernel have edges:
one-thread-pair tiles (n = T = 5), every tile width, states of one and of two tiles,
permutations left in the map at a pass's end (with outside controls), controlled and
two-angle rotations, quarter turns, diagonals waiting across passes and across a far
SWAP, and deferred renormalisation; against the oracle at the suite's 1e-12."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import Circuit, State, abi, workloads
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu
TOL = 1e-12

SINGLE = [abi.H, abi.X, abi.Y, abi.Z, abi.S, abi.T, abi.RX, abi.RY, abi.RZ, abi.PHASE, abi.U3]
PAIR = [abi.CNOT, abi.SWAP, abi.CZ, abi.CPHASE, abi.CRX, abi.CRY, abi.CRZ, abi.RXX, abi.RYY,
        abi.RZZ]


def gates_of(n, count, seed, far=True, kinds=SINGLE + PAIR):
    r = np.random.default_rng(seed)
    g = abi.empty_gates(count)
    for k in range(count):
        kind = kinds[r.integers(len(kinds))]
        g["kind"][k] = kind
        g["angle"][k] = r.uniform(-4, 4, 3)
        if r.integers(12) == 0:
            g["angle"][k, 0] = np.pi  # no cosine: a quarter turn
        a, b = (int(x) for x in r.choice(n, 2, replace=False))
        if not far:
            b = a + 1 if a + 1 < n else a - 1
        g["q"][k, 0] = a
        if kind in PAIR:
            g["q"][k, 1] = b
        if kind in (abi.RXX, abi.RYY) and r.integers(2):
            g["flags"][k] = abi.FLAG_TEXTBOOK
    return g


def run(n, g, v, width=11):
    old = C.c_int()
    call("lq_get_fusion_width", C.byref(old))
    st = State(n)
    try:
        call("lq_set_fusion_width", width)
        st.set_vector(v)
        call("lq_apply_circuit", st.handle, n, abi.gate_ptr(g), len(g), None, 0, abi.EXEC_FUSED)
        return st.vector()
    finally:
        call("lq_set_fusion_width", old.value)
        st.close()


@pytest.mark.parametrize("width", [5, 6, 8, 10, 11, 12])
@pytest.mark.parametrize("n", [5, 6, 9, 12, 13, 15])
def test_random_circuits(n, width):
    for seed, far in ((1, True), (2, False)):
        g = gates_of(n, 90, 100 * n + 10 * width + seed, far)
        v = random_state(n, n + seed)
        assert np.abs(run(n, g, v, width) - oracle.apply_circuit(v.copy(), g)).max() < TOL


@pytest.mark.parametrize("kinds", [[abi.CNOT, abi.U3], [abi.CNOT, abi.X, abi.SWAP],
                                   [abi.RY], [abi.CPHASE, abi.H], [abi.CZ, abi.RZ]])
def test_families(kinds):
    """Permutations only (no round at all), rotations without any diagonal (the
    factored-out scale must not run away), diagonals only, and their mixes."""
    n = 14
    for far in (True, False):
        g = gates_of(n, 400, 7, far, kinds)
        v = random_state(n, 3)
        assert np.abs(run(n, g, v) - oracle.apply_circuit(v.copy(), g)).max() < TOL


def test_many_outside_controls_of_one_window():
    """More outside control bits than one pass's map holds."""
    n = 18
    g = gates_of(n, 60, 1, True, [abi.CNOT])
    for k in range(len(g)):  # targets at the low index bits, controls everywhere else
        g["q"][k] = (k * 7 % 10, n - 1 - k % 4, -1)
    v = random_state(n, 5)
    assert np.abs(run(n, g, v, 10) - oracle.apply_circuit(v.copy(), g)).max() < TOL


def test_circuits_without_a_mapped_form_keep_the_op_records():
    n = 10
    r = np.random.default_rng(1)
    m = r.normal(size=(4, 4)) + 1j * r.normal(size=(4, 4))
    q, _ = np.linalg.qr(m)
    g = gates_of(n, 40, 4)
    g[5]["kind"] = abi.TOFFOLI
    g[5]["q"][:] = (1, 5, 8)
    g[20]["kind"] = abi.MATRIX2
    g[20]["q"][:] = (3, 4, -1)
    g[20]["m"][:] = np.ascontiguousarray(q).view(np.float64).reshape(-1)
    v = random_state(n, 9)
    assert np.abs(run(n, g, v) - oracle.apply_circuit(v.copy(), g)).max() < TOL


@pytest.mark.parametrize("n", [5, 11, 13])
def test_renormalising_builders(n):
    """Divisions by the norm move to the end of the circuit past unitary gates, and
    stay before a gate that is not unitary."""
    r = np.random.default_rng(n)
    shrink = np.array([[0.5, 0.1], [0.0, 0.8]])
    for matrix in (False, True):
        c = Circuit(n)
        for k in range(60):
            name = ("h", "x", "s", "t", "rx_matrix", "ry_matrix")[r.integers(6)]
            a, b = (int(x) for x in r.choice(n, 2, replace=False))
            getattr(c, name)(*((a, 0.7) if "_" in name else (a,)))
            c.cnot(a, b)
            if matrix and k == 20:
                c.add_single_qubit_gate(shrink, a, "shrink")
        g = c.packed().copy()
        if matrix:  # the same matrix without the division after it
            g = np.concatenate([g, g[g["kind"] == abi.MATRIX1][:1]])
            g[-1]["flags"] = 0
            g[-1]["m"][:8] = np.asarray(shrink, dtype=np.complex128).view(np.float64).reshape(-1)
        v = 3.0 * random_state(n, 2)
        assert np.abs(run(n, g, v) - oracle.apply_circuit(v.copy(), g)).max() < TOL
        assert np.abs(run(n, g, np.zeros(1 << n, dtype=complex))).max() == 0.0


def test_non_finite_angles_stay_non_finite():
    g = gates_of(6, 20, 3)
    g["kind"][4], g["angle"][4] = abi.RY, np.nan
    assert np.isnan(run(6, g, random_state(6, 1))).all()
