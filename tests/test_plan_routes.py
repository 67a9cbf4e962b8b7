"""CPU: which engine a circuit's plan is for.  lq_plan_circuit counts the rounds of the plan
that runs, lq_plan_dump those of the op-record plan; mapped rounds come to another number."""
import ctypes as C

import numpy as np
import pytest

from logosq_b200 import Circuit, abi, workloads, xyz_heisenberg
from logosq_b200._lib import call


def mapped(n, g):
    passes, rounds, alone = C.c_int(), C.c_int(), C.c_int()
    call("lq_plan_circuit", n, abi.gate_ptr(g), len(g), C.byref(passes), C.byref(rounds),
         C.byref(alone))
    buf, used, none = np.zeros(8 << 20, np.uint8), C.c_size_t(), np.zeros(1)
    call("lq_plan_dump", n, abi.gate_ptr(g), len(g), abi.f64_ptr(none), 0,
         buf.ctypes.data_as(C.c_void_p), len(buf), C.byref(used))
    return rounds.value != int(buf[:8].view(np.int32)[1])


def trotter(n):
    return xyz_heisenberg.create_circuit(n, jx=0.7, jy=0.6, jz=0.9, external_field=0.3,
                                         time_steps=3, dt=0.05).packed()


def controlled(n, every, count=120):
    r, c = np.random.default_rng(n), Circuit(n)
    for k in range(count):
        q = int(r.integers(n - 1))
        if k % every == every - 1:
            c.crx(q, q + 1, float(r.uniform(-3, 3)))
        else:
            c.u3(q, *(float(x) for x in r.uniform(-3, 3, 3)))
        if k % 3 == 0:
            c.cz(q, q + 1)
    return c.packed()


@pytest.mark.parametrize("n", [5, 8, 10, 11, 14, 19, 21])
def test_trotter_steps(n):
    assert mapped(n, trotter(n)) == (n >= 11)


@pytest.mark.parametrize("n", [5, 8, 10, 11, 19, 20])
def test_circuits_without_two_angle_rotations(n):
    assert mapped(n, workloads.brickwork_u3(n, 6, seed=3))


# of 160 gates: 6, 15, 24, 30 and 40 controlled rotations
@pytest.mark.parametrize("n,every,want", [(10, 20, True), (10, 8, False), (11, 8, True),
                                          (19, 5, True), (19, 4, False), (20, 4, True),
                                          (20, 3, False)])
def test_controlled_rotations(n, every, want):
    assert mapped(n, controlled(n, every)) == want
