"""The batch autotuner times only work items that a launch can have, and what it keeps are bounds that
change a launch (or the default)."""
import pytest

import qcb

pytestmark = pytest.mark.gpu


def batch_of(ctx, dims, prec, nr):
    return qcb.Batch(ctx, [qcb.GaugeField(ctx, d, prec, nr) for d in dims])


@pytest.mark.parametrize("prec,nr", [("fp64", 18), ("fp32", 12)])
def test_nothing_is_timed_where_there_is_one_size(ctx, prec, nr):
    """FP64 heatbaths have items of 32 links, and so has an FP32 batch that does not fill the chip; flows of
    fewer than 4096 blocks have blocks of 32 sites."""
    b = batch_of(ctx, [(4, 4, 4, 4), (6, 6, 6, 6), (8, 8, 8, 8)], prec, nr)
    before = ctx.launches()
    b.autotune(None)
    assert ctx.launches() == before
    assert b.tiles() == ([256] * 3, [256] * 3)
    b.close()


def test_picks_are_items_that_launches_have(ctx, tmp_path):
    """Twelve overlapping lattices: 13824 groups of 32 links a pass on 2368 warps make items of 160 links, the most."""
    dims = [(16, 16, 16, 16)] * 6 + [(16, 16, 16, 20)] * 6
    b = batch_of(ctx, dims, "fp32", 12)
    before = ctx.launches()
    b.autotune(tmp_path / "tune.json")
    assert ctx.launches() > before
    hb, flow = b.tiles()
    assert set(hb) <= {32, 64, 96, 128, 256} and set(flow) <= {32, 64, 96, 256}, (hb, flow)
    before = ctx.launches()
    b.autotune(tmp_path / "tune.json")  # from the file
    assert ctx.launches() == before and b.tiles() == (hb, flow)
    b.close()
