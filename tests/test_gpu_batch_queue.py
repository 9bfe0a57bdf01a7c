"""Batched heatbaths queued behind one another: each call's couplings, seeds and sweep counters are
its own, however far the device is behind the host."""
import numpy as np
import pytest

import qcb
from qcb import _lib

pytestmark = pytest.mark.gpu


def test_queued_heatbaths_keep_their_parameters(ctx):
    dims = [(16, 16, 16, 16), (8, 8, 8, 8)]
    single = [qcb.GaugeField(ctx, d, "fp32", 12) for d in dims]
    batched = [qcb.GaugeField(ctx, d, "fp32", 12) for d in dims]
    # the first call runs for milliseconds; the others are queued within microseconds
    calls = [(6.0, 60, 0), (5.7, 2, 60), (6.3, 1, 62), (5.85, 3, 63), (6.2, 2, 66)]
    for k, f in enumerate(single):
        for beta, n, first in calls:
            _lib.check(_lib.lib().qcb_heatbath(f.h, beta, n, 1, 11 + k, first))
    batch = qcb.Batch(ctx, batched)
    ctx.sync()
    for beta, n, first in calls:
        batch.heatbath([beta] * 2, n, 1, [11, 12], [first] * 2)
    ctx.sync()
    for f, g in zip(single, batched):
        assert np.array_equal(f.get_links(), g.get_links())
    batch.close()


def test_new_tiles_behind_a_queued_heatbath(ctx):
    dims = [(16, 16, 16, 16), (8, 8, 8, 8)]
    single = [qcb.GaugeField(ctx, d, "fp32", 12) for d in dims]
    batched = [qcb.GaugeField(ctx, d, "fp32", 12) for d in dims]
    calls = [(6.0, 60, 0), (5.7, 2, 60)]
    for k, f in enumerate(single):
        for beta, n, first in calls:
            _lib.check(_lib.lib().qcb_heatbath(f.h, beta, n, 1, 11 + k, first))
    batch = qcb.Batch(ctx, batched)
    ctx.sync()
    for beta, n, first in calls:
        batch.heatbath([beta] * 2, n, 1, [11, 12], [first] * 2)
    batch.set_tiles(hb=[64, 32])
    ctx.sync()
    for f, g in zip(single, batched):
        assert np.array_equal(f.get_links(), g.get_links())
    batch.close()
