"""CPU: planning a circuit that was not seen before costs host time in every call with new
angles, so the mapped rounds' planner is held to a small multiple of the op-record one."""
import ctypes as C
import time

import numpy as np
import pytest

from logosq_b200 import abi, workloads, xyz_heisenberg
from logosq_b200._lib import call


def trotter(n, steps):
    return xyz_heisenberg.create_circuit(n, jx=0.7, jy=0.6, jz=0.9, external_field=0.3,
                                         time_steps=steps, dt=0.05).packed()


def least(f, repeats=15):
    f()
    t = []
    for _ in range(repeats):
        a = time.perf_counter()
        f()
        t.append(time.perf_counter() - a)
    return min(t)


@pytest.mark.parametrize("n,make", [(12, lambda: trotter(12, 3)), (19, lambda: trotter(19, 10)),
                                    (16, lambda: workloads.brickwork_u3(16, 10, seed=1))])
def test_planning_costs_a_few_op_record_plans(n, make):
    """lq_plan_circuit plans the circuit in both forms, lq_plan_dump in one and writes it
    out: 1.5 to 2.8 times as much, on a busy machine too; Trotter steps 4.2 to 5.7 times when
    the planner copied whole gate records and used the complex library's operators."""
    g = make()
    out = [C.c_int() for _ in range(3)]
    buf, used, none = np.zeros(8 << 20, np.uint8), C.c_size_t(), np.zeros(1)
    both = least(lambda: call("lq_plan_circuit", n, abi.gate_ptr(g), len(g),
                              *(C.byref(x) for x in out)))
    records = least(lambda: call("lq_plan_dump", n, abi.gate_ptr(g), len(g), abi.f64_ptr(none), 0,
                                 buf.ctypes.data_as(C.c_void_p), len(buf), C.byref(used)))
    assert both < 3.5 * records
