"""GPU: amplitude damping around its size-dependent forms (one target in place, several
through a second vector that is kept with the handle or allocated for the call), against
the oracle at the suite's 1e-12."""
import ctypes as C

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import State
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,qubits", [(1, [0]), (2, [1]), (9, [8]), (10, [0]), (10, [4, 4]),
                                      (18, [17]), (18, [3])])
def test_amplitude_damping_of_one_target_in_place(n, qubits):
    v = 0.5 * random_state(n, n + 1)
    st = State(n)
    st.set_vector(v)
    arr = (C.c_int * len(qubits))(*qubits)
    call("lq_noise_amplitude_damping", st.handle, 0.3, arr, len(qubits))
    want = oracle.noise_amplitude_damping(v.copy(), 0.3, qubits)
    assert np.abs(st.vector() - want).max() < 1e-12
    st.close()


def test_one_target_needs_no_second_vector():
    """A 22-qubit state's workspace would be 64 MiB; the C header promises scratch for
    more than one target only."""
    import torch
    st = State.plus_state(22)
    st.synchronize()
    before = torch.cuda.mem_get_info()[0]
    call("lq_noise_amplitude_damping", st.handle, 0.1, (C.c_int * 1)(5), 1)
    st.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 32 << 20
    st.close()


def test_second_vector_of_a_large_state():
    n = 24  # 256 MiB: allocated for the call and given back
    st = State.plus_state(n)
    call("lq_noise_amplitude_damping", st.handle, 0.2, (C.c_int * 2)(0, n - 1), 2)
    # plus state: amplitudes by the two bits, (1 + sqrt g) + (1 + sqrt g) and so on
    g, k = np.sqrt(0.2), np.sqrt(0.8)
    want = np.array([2 * (1 + g), 1 + g + k, 2 * k])
    want /= np.sqrt((want[0] ** 2 + 2 * want[1] ** 2 + want[2] ** 2) / 4 * (1 << n))
    v = st.vector()
    i = np.arange(1 << n)
    ones = (i & 1) + (i >> (n - 1))
    assert np.abs(v - want[ones]).max() < 1e-12
    st.close()
