"""The frozen schedule's numbering of the links that move: every block length, shift and direction
against the oracle's schedule, and against the plain pass where nothing is frozen."""
import numpy as np
import pytest

import oracle as orc
import qcb

pytestmark = pytest.mark.gpu

# odd and even block lengths, one block a side, blocks of two (runs of one site), a single
# movable site a run, uneven extents, four lanes a link and one
CASES = [
    ((6, 6, 6, 12), 3, (0, 1, 2, 1)),
    ((4, 4, 4, 4), 4, (3, 0, 1, 2)),
    ((4, 2, 6, 8), 2, (1, 1, 0, 1)),
    ((10, 20, 10, 10), 5, (4, 0, 3, 2)),
    ((18, 12, 18, 24), 6, (5, 2, 0, 1)),
    ((6, 2, 4, 2), 1, (0, 0, 0, 0)),
]


@pytest.mark.parametrize("dims,lcore,shift", CASES)
def test_frozen_sweep_against_oracle(ctx, dims, lcore, shift):
    """Frozen links keep their bits; the others are the oracle's to the tolerance of every FP64
    heatbath (1e-11); FP32 moves the same links."""
    u = orc.hot_philox(dims, 31)
    f = qcb.GaugeField(ctx, dims)
    f.set_links(u)
    f.heatbath_frozen(6.0, 1, 1, 17, 0, lcore, shift)
    got = f.get_links()
    ref, fails = orc.heatbath_cb_frozen(u, dims, 6.0, 1, 1, 17, 0, lcore, shift)
    assert fails == 0
    moved = np.any(ref != u, axis=(-2, -1))
    assert np.array_equal(np.any(got != u, axis=(-2, -1)), moved)
    assert np.abs(got - ref).max() < 1e-11
    for nr in (12, 18):
        s = qcb.GaugeField(ctx, dims, "fp32", nr)
        s.set_links(u)
        before = s.get_links()
        s.heatbath_frozen(6.0, 1, 1, 17, 0, lcore, shift)
        assert np.array_equal(np.any(s.get_links() != before, axis=(-2, -1)), moved)
        s.close()
    f.close()
