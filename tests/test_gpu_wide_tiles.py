"""GPU: the record-driven rounds (circuits with Toffolis and general 4x4 matrices) at tile
bits 12, whose tiles take the kernel of 256 threads, beside 11; one, two and many tiles."""
import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import abi
from test_gpu_mapped_rounds import PAIR, SINGLE, TOL, gates_of, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [11, 12])
@pytest.mark.parametrize("n", [11, 12, 13, 17])
def test_circuits_without_a_mapped_form(n, width):
    g = gates_of(n, 120, 17 * n + width, kinds=SINGLE + PAIR)
    r = np.random.default_rng(n)
    for k in range(0, len(g), 7):
        g["kind"][k] = abi.TOFFOLI
        g["q"][k] = r.choice(n, 3, replace=False)
    for k in range(3, len(g), 11):
        q = np.linalg.qr(r.normal(size=(4, 4)) + 1j * r.normal(size=(4, 4)))[0]
        g["kind"][k] = abi.MATRIX2
        g["q"][k, :2] = r.choice(n, 2, replace=False)
        g["m"][k] = np.ascontiguousarray(q).view(np.float64).ravel()
    v = random_state(n, n)
    assert np.abs(run(n, g, v, width) - oracle.apply_circuit(v.copy(), g)).max() < TOL
