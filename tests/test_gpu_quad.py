"""The FP64 heatbath with four lanes per link (18-real, lattices of up to 14208 links a pass) at the
ends of its range, against the oracle and against the one-lane kernels, which larger lattices and
batches use."""
import numpy as np
import pytest

import oracle as orc
import qcb
from qcb import _lib
from qcb import slabs as qs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 4, 2, 6), (10, 6, 4, 2), (12, 12, 12, 16), (14, 12, 12, 16)])
@pytest.mark.parametrize("hits,beta", [(1, 6.0), (2, 0.4)])
def test_heatbath_and_plaquette(ctx, dims, hits, beta):
    """Both sides of the bound (13824 and 16128 links), partial blocks, small couplings (many
    rejected attempts), the measuring pass: the links of the one-lane kernels (a batch's) bit for
    bit.  At beta = 6 also the oracle's, to the tolerance of every FP64 heatbath; at 0.4 a link of
    2^4 amplifies the last bit of W = U A, of small norm, to 1e-8 in any of the kernels."""
    u = orc.hot_philox(dims, 19)
    f, one = qcb.GaugeField(ctx, dims), qcb.GaugeField(ctx, dims)
    f.set_links(u)
    one.set_links(u)
    hp = qcb.io.default_params()
    hp.beta, hp.N_samples, hp.N_sweeps, hp.N_hits = beta, 1, 1, hits
    p = qcb.heatbathcb.samples_plaquette(f, hp, qcb.PhiloxStream(seed=5, sweep=3))
    batch = qcb.Batch(ctx, [one])
    batch.heatbath([beta], 1, hits, [5], [3])
    ctx.sync()
    got = f.get_links()
    assert np.array_equal(got, one.get_links())
    assert abs(p - batch.plaquette()[0]) < 1e-12
    if beta == 6.0:
        ref, fails = orc.heatbath_cb(u, dims, beta, 1, hits, 5, 3)
        assert fails == 0
        assert np.abs(got - ref).max() < 1e-11
        assert abs(p - orc.plaquette(ref, dims)) < 1e-12
    batch.close()
    one.close()
    f.close()


def test_same_links_as_the_one_lane_kernels(ctx):
    """A lattice above the bound, its slabs (below it) and a batch (one lane) agree bit for bit, with
    and without frozen links."""
    dims = (12, 12, 12, 24)
    lib = _lib.lib()
    whole = qcb.GaugeField(ctx, dims)
    whole.hot_start(8)
    sl = qs.SlabLattice(ctx, dims, 2)
    sl.hot_start(8)
    _lib.check(lib.qcb_heatbath(whole.h, 6.0, 2, 2, 77, 0))
    sl.heatbath(6.0, 2, 2, 77, 0)
    assert np.array_equal(sl.get_links(), whole.get_links())
    sl.close()
    whole.close()
    small = (6, 4, 8, 4)
    a, b = qcb.GaugeField(ctx, small), qcb.GaugeField(ctx, small)
    a.hot_start(9)
    b.hot_start(9)
    _lib.check(lib.qcb_heatbath(a.h, 5.8, 3, 1, 12, 4))
    batch = qcb.Batch(ctx, [b])
    batch.heatbath([5.8], 3, 1, [12], [4])
    ctx.sync()
    assert np.array_equal(a.get_links(), b.get_links())
    batch.close()
    a.heatbath_frozen(6.0, 2, 1, 3, 0, 2, (1, 0, 1, 1))
    ref, _ = orc.heatbath_cb_frozen(b.get_links(), small, 6.0, 2, 1, 3, 0, 2, (1, 0, 1, 1))
    assert np.abs(a.get_links() - ref).max() < 1e-11
    a.close()
    b.close()
