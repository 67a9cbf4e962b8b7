"""GPU: mapped rounds of gates whose factors meet: angles that are multiples of a quarter
turn (factors equal to 1, -1 and +-i, ties between sine and cosine), the same gate again and
again, and factors waiting under one mask for several rotations; against the oracle."""
import math

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import abi
from test_gpu_mapped_rounds import PAIR, SINGLE, TOL, gates_of, run

pytestmark = pytest.mark.gpu
TURNS = [0.0, math.pi / 2, -math.pi / 2, math.pi, -math.pi, 2 * math.pi, 1e-9]


@pytest.mark.parametrize("n,width", [(5, 5), (9, 11), (13, 11), (14, 12)])
@pytest.mark.parametrize("few", [1, 3, 7])
def test_angles_that_meet(n, width, few):
    for seed in range(4):
        g = gates_of(n, 120, 31 * n + seed, far=seed % 2 == 0)
        r = np.random.default_rng(seed)
        g["angle"] = np.asarray(TURNS)[r.permutation(len(TURNS))[:few]][
            r.integers(few, size=g["angle"].shape)]
        v = random_state(n, seed)
        assert np.abs(run(n, g, v, width) - oracle.apply_circuit(v.copy(), g)).max() < TOL


@pytest.mark.parametrize("width", [5, 6, 8, 11])
@pytest.mark.parametrize("n", [5, 6, 9, 10])
def test_small_states_with_few_two_angle_rotations(n, width):
    """Up to 10 qubits a circuit keeps to mapped rounds with a twelfth of its gates being
    controlled rotations, RXX or RYY: here six of 90."""
    plain = [k for k in SINGLE + PAIR if k not in (abi.CRX, abi.CRY, abi.RXX, abi.RYY)]
    for seed in range(3):
        g = gates_of(n, 90, 13 * n + seed, far=seed != 1, kinds=plain)
        r = np.random.default_rng(seed)
        for k, kind in zip(range(5, 90, 15), [abi.CRX, abi.CRY, abi.RXX, abi.RYY] * 2):
            g["kind"][k] = kind
            g["q"][k, :2] = r.choice(n, 2, replace=False)
            g["flags"][k] = abi.FLAG_TEXTBOOK * int(r.integers(2)) if kind in (
                abi.RXX, abi.RYY) else 0
        v = random_state(n, seed)
        assert np.abs(run(n, g, v, width) - oracle.apply_circuit(v.copy(), g)).max() < TOL
