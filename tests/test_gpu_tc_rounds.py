"""GPU: the tensor-core pass with several tiles per SM (its groups take turns, tiles rotate
through the buffers, the last round is not full) and with as many blocks as stay in
shared memory or more.  The state is one 12-qubit vector in every tile, times a power of
two and a sign per tile, and the gates act inside the tiles: all tiles must come out
equal to the bit up to those factors, and equal to the complex128 engine on the 12-qubit
vector within test_gpu_tc.py's bar for few blocks (1e-5 of the largest amplitude)."""
import numpy as np
import pytest

from logosq_b200 import State, abi, workloads
from logosq_b200._lib import call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [0, 1, 4])  # 0: one block
@pytest.mark.parametrize("n,h", [(19, 4), (20, 12), (21, 4), (21, 10), (22, 14)])
def test_tc_pass_with_many_tiles(n, h, layers):
    v = workloads.gaussian_state(12, 7).astype(np.complex64)
    t = np.arange(1 << (n - 12))
    s = (np.where(t % 3 == 0, -1.0, 1.0) * 2.0 ** -(t % 5)).astype(np.float32)
    # index bits: 4 low ones of the tile, c2 (h - 4 of them), the tile's 8 others, c4
    full = np.empty((1 << (n - h - 8), 256, 1 << (h - 4), 16), dtype=np.complex64)
    full[...] = v.reshape(1, 256, 1, 16) * s.reshape(1 << (n - h - 8), 1, 1 << (h - 4), 1)
    g = workloads.brickwork_u3(12, max(layers, 1), seed=n)
    g = g if layers else g[:5]
    want = State.zero_state(12)
    want.set_vector(v.astype(np.complex128))
    call("lq_apply_circuit", want.handle, 12, abi.gate_ptr(g), len(g), None, 0, abi.EXEC_FUSED)
    ref = want.vector().reshape(256, 16)
    want.close()
    # qubit q of the small circuit is its index bit 11 - q; the same tile bit of the state
    big = g.copy()
    for row in big["q"]:
        for j in range(2):
            if row[j] >= 0:
                b = 11 - row[j]
                row[j] = n - 1 - (b if b < 4 else b - 4 + h)
    st = State.zero_state(n, dtype=abi.LQ_C64)
    st.set_vector(full.reshape(-1).astype(np.complex128))
    call("lq_apply_circuit_tc", st.handle, n, abi.gate_ptr(big), len(big), None, 0, None, None)
    got = st.vector().astype(np.complex64).reshape(full.shape)
    st.close()
    one = got / s.reshape(1 << (n - h - 8), 1, 1 << (h - 4), 1)
    assert (one == one[:1, :, :1, :]).all()
    assert np.abs(one[0, :, 0, :] - ref).max() < 1e-5 * np.abs(ref).max()
