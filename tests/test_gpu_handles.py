"""GPU: what a handle's end leaves alone: graph captures on other streams, readers of
its amplitudes on other streams, and the contents of the next handle."""
import threading

import numpy as np
import pytest

from helpers import random_state
from logosq_b200 import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("held", [0, 6])  # the spare list empty, and full
def test_closing_a_handle_leaves_a_capture_on_another_thread_alone(held):
    import torch
    for st in [State(6) for _ in range(held)]:
        st.close()
    st = State(6)
    st.synchronize()
    x = torch.zeros(8, device="cuda")
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        x += 1
        t = threading.Thread(target=st.close)
        t.start()
        t.join()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8


def test_a_copy_outlives_the_handle_it_was_made_from():
    # sizes whose buffers the next handle takes over; the copy is still queued when the
    # source goes and the next handle writes |0...0>
    for n in (1, 8, 16):
        v = random_state(n, n)
        for _ in range(20):
            src = State(n)
            src.set_vector(v)
            dst = src.clone()
            src.close()
            nxt = State(n)
            assert np.array_equal(dst.vector(), v)
            w = nxt.vector()
            assert w[0] == 1.0 and np.count_nonzero(w) == 1
            nxt.close()
            dst.close()
