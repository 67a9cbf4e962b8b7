"""GPU: circuits captured into a CUDA graph on their state's stream.  A circuit that has a
mapped form is captured with its program in the launches, on its first submission too, and is
not touched by what the handle runs later; one without is captured from the program that the
same circuit left in the handle's buffer."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import Circuit, State, abi, workloads, xyz_heisenberg
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu


def submit(st, n, g):
    call("lq_apply_circuit", st.handle, n, abi.gate_ptr(g), len(g), None, 0, abi.EXEC_FUSED)


def captured(st, n, g):
    import torch
    p = C.c_void_p()
    call("lq_state_stream", st.handle, C.byref(p))
    stream, graph = torch.cuda.ExternalStream(p.value), torch.cuda.CUDAGraph()
    st.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        submit(st, n, g)
    return graph


def trotter(n):
    return xyz_heisenberg.create_circuit(n, jx=0.7, jy=0.6, jz=0.9, external_field=0.3,
                                         time_steps=2, dt=0.05).packed()


def replayed(st, graph, v):
    import torch
    st.set_vector(v)
    graph.replay()
    torch.cuda.synchronize()
    return st.vector()


@pytest.mark.parametrize("before", [False, True])  # submitted before, as op records
@pytest.mark.parametrize("n", [6, 10, 13])
def test_mapped_circuits(n, before):
    g, v = trotter(n), random_state(n, n)
    st = State(n)
    if before:
        submit(st, n, g)
    graph = captured(st, n, g)
    want = oracle.apply_circuit(v.copy(), g)
    assert np.abs(replayed(st, graph, v) - want).max() < 1e-12
    other = Circuit(n)  # (a Toffoli: records, in the handle's buffer)
    other.h(0)
    other.toffoli(0, 1, 2)
    for x in (other.packed(), workloads.brickwork_u3(n, 4, seed=1)):
        submit(st, n, x)
        assert np.abs(replayed(st, graph, v) - want).max() < 1e-12
    del graph
    st.close()


def test_a_circuit_without_mapped_form():
    n = 9
    c = Circuit(n)
    for q in range(n):
        c.ry(q, 0.3 + q)
    c.toffoli(0, 4, 8)
    g, v = c.packed(), random_state(n, 1)
    st = State(n)
    submit(st, n, g)
    graph = captured(st, n, g)
    assert np.abs(replayed(st, graph, v) - oracle.apply_circuit(v.copy(), g)).max() < 1e-12
    del graph
    st.close()


@pytest.mark.parametrize("n,before", [(12, False), (12, True), (19, False), (19, True)])
def test_damping_of_several_targets(n, before):
    """Its second vector belongs to the graph, whatever workspaces the handle or the pool
    hold or give back later."""
    import torch
    st, big = State(n), State(n + 1)
    q = (C.c_int * 2)(0, n - 1)

    def damp(s):
        call("lq_noise_amplitude_damping", s.handle, 0.2, q, 2)

    if before:
        damp(st)
    p = C.c_void_p()
    call("lq_state_stream", st.handle, C.byref(p))
    stream, graph = torch.cuda.ExternalStream(p.value), torch.cuda.CUDAGraph()
    st.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        damp(st)
    v = random_state(n, 4)
    want = oracle.noise_amplitude_damping(v.copy(), 0.2, [0, n - 1])
    for _ in range(2):
        assert np.abs(replayed(st, graph, v) - want).max() < 1e-12
        damp(big)
        damp(st)
    del graph
    big.close()
    st.close()
