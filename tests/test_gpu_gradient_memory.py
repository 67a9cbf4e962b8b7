"""GPU: what a plain gradient of a large state leaves with its handle."""
import math

import numpy as np
import pytest

from logosq_b200 import State, abi, workloads
from logosq_b200._lib import call
from logosq_b200.optimization import RealAmplitudesAnsatz

pytestmark = pytest.mark.gpu


def test_partial_sums_of_a_large_state_are_given_back():
    import torch
    n, depth = 25, 20  # 525 runs of gates on 2^14 tiles: some 200 MB of partial sums
    ansatz = RealAmplitudesAnsatz(n, depth)
    gates = ansatz.template().packed()
    terms = workloads.heisenberg_terms(n, [0.5] * (n - 1), [0.4] * (n - 1), [0.3] * (n - 1), 0.2)
    theta = np.linspace(-2, 2, ansatz.num_parameters())
    grad = np.zeros(len(theta))

    def free():
        call("lq_state_synchronize", st.handle)
        return torch.cuda.mem_get_info()[0] >> 20

    st = State(n)
    before = free()
    call("lq_parameter_shift", st.handle, abi.gate_ptr(gates), len(gates), abi.f64_ptr(theta),
         len(theta), abi.term_ptr(terms), len(terms), abi.Y_REFERENCE, math.pi / 2,
         abi.f64_ptr(grad))
    assert np.abs(grad).max() > 0
    assert before - free() < 64
    st.close()
