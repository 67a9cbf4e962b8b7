"""GPU: the tile widths of the batched gradients' two engines."""
import numpy as np
import pytest

from logosq_b200 import workloads
from logosq_b200._lib import call
from logosq_b200.batch import heisenberg_batch

pytestmark = pytest.mark.gpu


def test_the_two_engines_choose_their_widths_independently():
    recs = workloads.heisenberg_instances(3, seed=5, n_lo=13, n_hi=14)
    theta = np.concatenate([r["theta"] for r in recs])
    ref = heisenberg_batch(recs)
    _, g11 = ref.gradients(theta)
    b = heisenberg_batch(recs)
    bad = theta.copy()
    bad[0] = np.nan
    b.gradients(bad)  # the shifted circuits tune their width
    _, g = b.gradients(theta)
    assert b.tuning()["tile_bits"] == 11  # and the sweep keeps its own
    assert np.array_equal(g, g11)
    call("lq_batch_set_tile_bits", b._h, 12)
    assert b.tuning()["tile_bits"] == 12
    call("lq_batch_set_tile_bits", b._h, 0)
    assert b.tuning()["tile_bits"] == 0
    _, g = b.gradients(theta)
    assert np.array_equal(g, g11)
    ref.close()
    b.close()
