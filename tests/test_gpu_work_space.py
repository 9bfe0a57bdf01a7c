"""Work space of the flow and the clover: made once for a context, not again for every lattice and batch,
and plans that were made on a buffer follow when it is replaced."""
import ctypes as C

import numpy as np
import pytest
import torch

import qcb
from qcb import _lib

pytestmark = pytest.mark.gpu


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def qe(f):
    return qcb.observables.topo_q_e_clover_global(f)


def test_first_measurement_of_a_lattice_does_not_allocate(ctx):
    warm = qcb.GaugeField(ctx, (16, 16, 16, 16), "fp32", 12)
    qe(warm)  # the context's loop buffer
    f = qcb.GaugeField(ctx, (64, 64, 64, 64), "fp32", 12)  # 2.1 MB of partial sums
    before = free()
    qe(f)
    _lib.check(_lib.lib().qcb_heatbath_plaquette(f.h, 6.0, 1, 1, 3, 0, C.byref(C.c_double())))
    assert free() == before
    f.close()
    warm.close()


def test_batches_share_the_context_s_buffer_and_plan_ahead(ctx):
    fields = [qcb.GaugeField(ctx, (16, 16, 16, 32), "fp64", 18) for _ in range(2)]
    for k, f in enumerate(fields):
        f.hot_start(5 + k)
    alone = [qe(f) for f in fields]
    batches = [qcb.Batch(ctx, fields[:1]), qcb.Batch(ctx, fields[1:])]
    before = free()
    for b, ref in zip(batches, alone):
        q, e = b.topo_qe()
        assert abs(q[0] - ref[0]) < 1e-12 * max(1.0, abs(ref[0])) and abs(e[0] - ref[1]) < 1e-12 * ref[1]
        b.flow_steps(0.02, 1)
    assert before - free() < 8 << 20  # the loops of one of these lattices take 57 MB
    for b in batches:
        b.close()
    for f in fields:
        f.close()


def test_plans_follow_a_replaced_buffer():
    """A context of its own whose loop buffer is made larger under a batch's captured plan."""
    c = qcb.Context(0)
    small = [qcb.GaugeField(c, (4, 4, 4, 4), "fp64", 18), qcb.GaugeField(c, (4, 6, 8, 4), "fp64", 18)]
    ref = [qcb.GaugeField(c, f.dims, "fp64", 18) for f in small]
    for k, (f, r) in enumerate(zip(small, ref)):
        f.hot_start(5 + k)
        r.hot_start(5 + k)
    batch = qcb.Batch(c, small)
    args = dict(n_sweeps=0, n_hits=1, eps=0.02, n_groups=2, rk_per_group=1)
    _, rec, graph = batch.run([6.0, 6.0], [1, 2], [0, 0], **args)
    qe(qcb.GaugeField(c, (128, 128, 128, 4), "fp64", 12))  # two of its time slices take 1.8 GB
    _, again, graph = batch.run([6.0, 6.0], [1, 2], [0, 0], **args)
    assert graph and np.array_equal(rec, again)
    batch.flow_steps(0.02, 2)
    c.sync()
    for f, r in zip(small, ref):
        _lib.check(_lib.lib().qcb_flow_steps(r.h, 0.02, 2))
        assert np.array_equal(f.get_links(), r.get_links())
    c.close()
