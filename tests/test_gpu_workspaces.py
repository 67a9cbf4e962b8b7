"""GPU: workspaces of calls that need a second vector: few are kept however many handles
used one, none after the last handle, and one handed from a stream to another waits for its
last use."""
import ctypes as C
import subprocess
import sys
import threading

import numpy as np
import pytest

import oracle
from helpers import random_state
from logosq_b200 import State
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, torch
from logosq_b200 import State
from logosq_b200._lib import call
def free():
    return torch.cuda.mem_get_info()[0] >> 20
State(20).close()
states = [State(20) for _ in range(40)]
call("lq_state_synchronize", states[-1].handle)
before = free()
for s in states:
    call("lq_noise_amplitude_damping", s.handle, 0.1, (C.c_int * 2)(0, 1), 2)
for s in states:
    call("lq_state_synchronize", s.handle)
kept = before - free()
for s in states[1:]:
    s.close()
one = free()
states[0].close()
print(kept, free() - one)
"""


def test_few_workspaces_stay_and_none_after_the_last_handle():
    """40 states of 20 qubits: 640 MiB of second vectors when each handle kept its own."""
    out = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, check=True)
    kept, back = map(int, out.stdout.split())
    assert kept <= 256 + 64   # (and the driver's granularity)
    assert back >= 16         # a state of 16 MiB at the least, and the workspaces


def test_workspaces_in_turn_on_many_streams():
    n, count = 18, 6  # 4 MiB each: more than a handle keeps for itself
    v = [random_state(n, k) for k in range(count)]
    want = [oracle.noise_amplitude_damping(x.copy(), 0.2, [0, 7, n - 1]) for x in v]
    states = []
    for x in v:
        states.append(State(n))
        states[-1].set_vector(x)
    q = (C.c_int * 3)(0, 7, n - 1)
    failed = []

    def work(mine):
        try:
            for s in mine:  # no wait in between: the same buffers go from stream to stream
                call("lq_noise_amplitude_damping", s.handle, 0.2, q, 3)
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(states[k::3],)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for s, w in zip(states, want):
        assert np.abs(s.vector() - w).max() < 1e-12
        s.close()


def test_samples_between_dampings():
    """The pool's buffers serve calls of other sizes and kinds: the same samples as from a
    handle that never shared one."""
    n, shots = 21, 2000
    x = random_state(n, 3)
    a, b = State(n), State(19)
    a.set_vector(x)

    def sample():
        out = np.empty(shots, np.uint64)
        call("lq_measure_shots", a.handle, shots, 5, out.ctypes.data_as(C.POINTER(C.c_uint64)))
        return out

    first = sample()
    for _ in range(3):
        call("lq_noise_amplitude_damping", b.handle, 0.1, (C.c_int * 2)(0, 1), 2)
        assert np.array_equal(sample(), first)
    a.close()
    b.close()


GROWING = """
import ctypes as C, torch, numpy as np
from logosq_b200 import State
from logosq_b200._lib import call
def free():
    return torch.cuda.mem_get_info()[0] >> 20
st = State.plus_state(23)
call("lq_state_synchronize", st.handle)
before = free()
low = []
for k in range(40):
    out = np.empty(100 + 3000 * k, np.uint64)
    call("lq_measure_shots", st.handle, len(out), k, out.ctypes.data_as(C.POINTER(C.c_uint64)))
    low.append(before - free())
print(max(low), low[-1] - low[-2], low[-1])
"""


def test_workspaces_of_growing_sizes():
    """Samples of 23 qubits want 64 MiB and a little more each time: they share a buffer, and
    a call that finds only smaller ones takes their place."""
    out = subprocess.run([sys.executable, "-c", GROWING], capture_output=True, text=True,
                         check=True)
    most, last, kept = map(int, out.stdout.split())
    assert most <= 256 + 64
    assert last == 0 and kept > 0  # nothing allocated for the last call alone
