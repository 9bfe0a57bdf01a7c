"""The batched heatbath's work items (a warp's each) on every branch of their sizing: results are
those of the single lattice, bit for bit."""
import numpy as np
import pytest

import qcb
from qcb import _lib

pytestmark = pytest.mark.gpu

CASES = {
    "one link group a level": [(2, 2, 2, 2)],
    "fewer items than blocks": [(4, 4, 4, 4), (6, 6, 4, 4), (2, 2, 2, 2)],
    "more lattices than the prefix sums in shared memory": [(2, 2, 2, 2)] * 1030 + [(4, 4, 4, 2)],
    "one lattice, a ragged last item of 64 or more": [(20, 20, 20, 22)],
    "overlapping lattices, two groups an item": [(18, 16, 16, 16), (16, 16, 16, 16), (16, 16, 14, 18), (16,) * 4],
}


@pytest.mark.parametrize("prec,nr", [("fp32", 12), ("fp64", 18)])
@pytest.mark.parametrize("name", CASES)
def test_items_of_every_size(ctx, name, prec, nr):
    dims = CASES[name]
    n = len(dims)
    fields = []
    for k, d in enumerate(dims):
        f = qcb.GaugeField(ctx, d, prec, nr)
        f.hot_start(60 + k)
        fields.append(f)
    picked = sorted({0, n // 2, n - 1})
    singles = []
    for k in picked:
        f = qcb.GaugeField(ctx, dims[k], prec, nr)
        f.hot_start(60 + k)
        _lib.check(_lib.lib().qcb_heatbath(f.h, 5.5 + 0.001 * k, 2, 1, 9 + k, k))
        singles.append(f)
    batch = qcb.Batch(ctx, fields)
    batch.heatbath([5.5 + 0.001 * k for k in range(n)], 2, 1, [9 + k for k in range(n)], list(range(n)))
    plaq = batch.plaquette()
    for k, f in zip(picked, singles):
        assert np.array_equal(f.get_links(), fields[k].get_links())
        assert abs(plaq[k] - qcb.observables.mean_plaquette_global(f)) < 1e-13
    batch.close()
