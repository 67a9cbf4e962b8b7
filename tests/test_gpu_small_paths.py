"""GPU: the size-dependent branches of sampling, Pauli sums, damping and the network's
products, at the edges where each one starts."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import State, abi, learned
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu


def shots(st, count, seed):
    out = np.empty(count, dtype=np.uint64)
    call("lq_measure_shots", st.handle, C.c_uint64(count), C.c_uint64(seed),
         out.ctypes.data_as(C.POINTER(C.c_uint64)))
    return out


@pytest.mark.parametrize("n", [1, 9, 10, 11, 20])
def test_shots_around_one_chunk_and_one_level(n):
    v = random_state(n, 60 + n)
    st = State(n)
    st.set_vector(v)
    assert np.array_equal(shots(st, 3000, 5), oracle.sample_indices(v, 3000, 5))
    st.close()


def test_shots_with_rescanned_chunks_equal_the_stored_scan():
    """2^24 amplitudes: few shots scan their chunks again, many use the stored scan;
    shot k is the same draw in both."""
    n = 24
    st = State.plus_state(n)
    g = np.concatenate([_ry(q, 0.3 + 0.05 * q) for q in range(n)])
    call("lq_apply_circuit", st.handle, n, abi.gate_ptr(g), len(g), None, 0, abi.EXEC_FUSED)
    few, many = shots(st, 5000, 3), shots(st, (1 << 18) + 1, 3)
    assert np.array_equal(few, many[:5000])
    st.close()


def _ry(q, angle):
    g = abi.empty_gates(1)
    g["kind"], g["q"][0, 0], g["angle"][0, 0] = abi.RY, q, angle
    return g


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9, 12, 13, 18])
def test_pauli_sums_by_windows(n, c64):
    r = np.random.default_rng(n)
    rows = []
    for _ in range(5):
        width = int(r.integers(1, min(n, 4) + 1))
        lo = int(r.integers(0, n - width + 1))
        x = int(r.integers(1, 1 << width)) << lo
        for _ in range(3):
            rows.append((float(r.normal()), x, int(r.integers(0, 1 << n))))
    rows.append((0.3, (1 << n) - 1, int(r.integers(0, 1 << n))))  # too wide for any window
    rows += [(float(r.normal()), 0, int(r.integers(0, 1 << n))) for _ in range(10)]
    terms = np.zeros(len(rows), dtype=abi.TERM_DTYPE)
    for t, (c, x, z) in zip(terms, rows):
        t["coefficient"], t["xmask"], t["zmask"], t["ny"] = c, x, z, bin(x & z).count("1")
    v = random_state(n, 80 + n)
    if c64:
        v = v.astype(np.complex64).astype(np.complex128)
    st = State(n, abi.LQ_C64 if c64 else abi.LQ_C128)
    st.set_vector(v)
    for conv in (abi.Y_REFERENCE, abi.Y_TEXTBOOK):
        out = C.c_double()
        call("lq_expectation_pauli", st.handle, abi.term_ptr(terms), len(terms), conv,
             C.byref(out), None)
        want = oracle.expectation(v, terms, conv)
        scale = np.abs(terms["coefficient"]).sum()
        assert abs(out.value - want) < 1e-12 * scale
    st.close()


@pytest.mark.parametrize("n", [7, 11, 14])
def test_pauli_sums_of_many_terms(n):
    # more independent masks than one round holds, and groups longer than one stage
    r = np.random.default_rng(n)
    rows = [(float(r.normal()), int(r.integers(1, 1 << 7)), int(r.integers(0, 1 << n)))
            for _ in range(60)]
    rows += [(float(r.normal()), 5, int(r.integers(0, 1 << n))) for _ in range(300)]
    rows += [(float(r.normal()), 0, int(r.integers(0, 1 << n))) for _ in range(600)]
    terms = np.zeros(len(rows), dtype=abi.TERM_DTYPE)
    for t, (c, x, z) in zip(terms, rows):
        t["coefficient"], t["xmask"], t["zmask"], t["ny"] = c, x, z, bin(x & z).count("1")
    v = random_state(n, 90 + n)
    st = State(n, abi.LQ_C128)
    st.set_vector(v)
    out = C.c_double()
    call("lq_expectation_pauli", st.handle, abi.term_ptr(terms), len(terms), abi.Y_REFERENCE,
         C.byref(out), None)
    want = oracle.expectation(v, terms, abi.Y_REFERENCE)
    assert abs(out.value - want) < 1e-12 * np.abs(terms["coefficient"]).sum()
    st.close()


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("n", [11, 12, 21, 22])
@pytest.mark.parametrize("xs", [(0,), (1 << 2,), (0, 1 << 2), (1 << 9,), (1 << 5, 1 << 10, 0)])
def test_pauli_sums_that_are_sweeps(n, xs, c64):
    # lone groups above and below the size where a sweep takes them; Z strings alone
    r = np.random.default_rng(n)
    rows = [(float(r.normal()), x, int(r.integers(0, 1 << n))) for x in xs for _ in range(3)]
    rows += [(float(r.normal()), xs[0], int(r.integers(0, 1 << n)))
             for _ in range(0 if xs[0] else 20)]
    terms = np.zeros(len(rows), dtype=abi.TERM_DTYPE)
    for t, (c, x, z) in zip(terms, rows):
        t["coefficient"], t["xmask"], t["zmask"], t["ny"] = c, x, z, bin(x & z).count("1")
    v = random_state(n, 70 + n)
    if c64:
        v = v.astype(np.complex64).astype(np.complex128)
    st = State(n, abi.LQ_C64 if c64 else abi.LQ_C128)
    st.set_vector(v)
    out = C.c_double()
    call("lq_expectation_pauli", st.handle, abi.term_ptr(terms), len(terms), abi.Y_TEXTBOOK,
         C.byref(out), None)
    want = oracle.expectation(v, terms, abi.Y_TEXTBOOK)
    assert abs(out.value - want) < 1e-12 * np.abs(terms["coefficient"]).sum()
    st.close()


@pytest.mark.parametrize("n,qubits", [(1, [0]), (5, [2, 2, 4]), (12, None), (13, [12, 0])])
def test_amplitude_damping_target_lists(n, qubits):
    v = random_state(n, n)
    st = State(n)
    st.set_vector(v)
    arr = None if qubits is None else (C.c_int * len(qubits))(*qubits)
    call("lq_noise_amplitude_damping", st.handle, 0.07, arr, 0 if qubits is None else len(qubits))
    want = oracle.noise_amplitude_damping(v.copy(), 0.07, list(range(n)) if qubits is None else qubits)
    assert np.abs(st.vector() - want).max() < 1e-12
    st.close()


@pytest.mark.parametrize("shape,batch", [((1, 1, 1, 1), 1), ((33, 65, 2, 31), 32),
                                         ((32, 64, 1, 96), 33)])
def test_network_products_at_tile_edges(shape, batch):
    """Forward and gradient, with the bars of the network's other tests (FP32 sums of
    at most 65 terms)."""
    net = learned.WarmStartMLP(*shape, seed=4)
    r = np.random.default_rng(batch)
    x = r.normal(0, 1, (batch, shape[0])).astype(np.float32)
    t = r.uniform(-3, 3, (batch, shape[3])).astype(np.float32)
    m = np.ones((batch, shape[3]), dtype=np.float32)
    want = oracle.mlp_forward(shape, net.params(), x)
    assert np.abs(net.forward(x) - want).max() <= 1e-5 * max(1.0, np.abs(want).max())
    loss = net.loss_grad(x, t, m)
    want_loss, want_g = oracle.mlp_loss_grad(shape, net.params().astype(np.float64), x, t, m)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    assert np.abs(net.grads() - want_g).max() <= 1e-4 * np.abs(want_g).max()
    net.close()


@pytest.mark.parametrize("threads", [1, 6])
def test_handles_that_take_over_from_destroyed_ones(threads):
    # sizes below, at and above the kept ones, both types, more handles than are kept
    sizes = [(4, abi.LQ_C128), (16, abi.LQ_C128), (4, abi.LQ_C64), (17, abi.LQ_C128),
             (17, abi.LQ_C64), (4, abi.LQ_C128), (9, abi.LQ_C128)]
    wrong = []

    def work(seed):
        for turn in range(8):
            held = []
            for n, dtype in sizes:
                st = State(n, dtype)
                v = st.vector()
                if v[0] != 1.0 or np.count_nonzero(v) != 1:
                    wrong.append(("fresh", n, dtype))
                g = _ry(seed % n, 0.3 + seed + turn)
                call("lq_apply_circuit", st.handle, n, abi.gate_ptr(g), 1, None, 0,
                     abi.EXEC_FUSED)
                held.append((st, n, dtype, 0.3 + seed + turn))
                if len(held) > 3:
                    held.pop(0)[0].close()
            for st, n, dtype, angle in held:
                v = st.vector()
                w = [abs(np.cos(angle / 2)), abs(np.sin(angle / 2))]
                if not np.allclose([abs(v[0]), abs(v[1 << (n - 1 - seed % n)])], w, atol=1e-6):
                    wrong.append((n, dtype, angle))
                st.close()

    pool = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not wrong
