"""GPU: mapped rounds of gates whose factors meet: angles that are multiples of a quarter
turn (factors equal to 1, -1 and +-i, ties between sine and cosine), the same gate again and
again, and factors waiting under one mask for several rotations; against the oracle."""
import math

import numpy as np
import pytest

import oracle
from helpers import random_state
from test_gpu_mapped_rounds import TOL, gates_of, run

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
