"""GPU: amplitude damping around its size-dependent forms (one target in place, several
through a second vector), against
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

