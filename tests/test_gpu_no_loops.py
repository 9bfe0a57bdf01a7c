"""The flow and the clover where no plaquette-loop work space is to be had: staples and leaves are
multiplied out, and calls that needed no work space before there was one still need none."""
import numpy as np
import pytest

import oracle as orc
import qcb
from qcb import _lib
from qcb import slabs as qs

pytestmark = pytest.mark.gpu

# remainders of the 64- and 128-site blocks, extents of two
DIMS = [(2, 2, 2, 2), (2, 2, 4, 6), (4, 6, 8, 4), (6, 6, 6, 10)]


@pytest.fixture
def without():
    c = qcb.Context(0)
    c.set_loop_bytes(0)
    yield c
    c.close()


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,nr", [("fp64", 18), ("fp64", 12), ("fp32", 18), ("fp32", 12)])
def test_matches_oracle(without, dims, prec, nr):
    """Records and two steps.  Bounds of the path with loops (test_gpu_loops): its roundings are as many."""
    u = orc.hot_philox(dims, 91)
    f = qcb.GaugeField(without, dims, prec, nr)
    f.set_links(u)
    tol = 1e-12 if prec == "fp64" else 1e-5
    ref = orc.flow_measure(u, dims, 0.02, 2, 1).reshape(-1, 3)
    rec = qcb.observables.topo_charge_flowed(f, qcb.GradientFlow(0.02), 2, 1).reshape(-1, 3)
    for a, b in zip(rec, ref):
        assert abs(a[1] - b[1]) <= 10 * tol * max(1.0, abs(b[1])) and abs(a[2] - b[2]) <= tol * b[2]
    q, e = qcb.observables.topo_q_e_clover_global(f)
    assert abs(q - rec[0, 1]) < 1e-12 and abs(e - rec[0, 2]) < 1e-12 * e
    _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 2))
    assert np.abs(f.get_links() - orc.flow_steps(u, dims, 0.02, 2)).max() < 2 * tol


def test_links_off_su3(without):
    dims = (4, 6, 4, 6)
    rng = np.random.default_rng(4)
    u = orc.hot_philox(dims, 92)
    u = u + 1e-3 * (rng.standard_normal(u.shape) + 1j * rng.standard_normal(u.shape))
    f = qcb.GaugeField(without, dims, "fp64", 18)
    f.set_links(u)
    (_, qr, er), = orc.flow_measure(u, dims, 0.02, 1, 0).reshape(-1, 3)
    q, e = qcb.observables.topo_q_e_clover_global(f)
    assert abs(q - qr) <= 1e-11 * max(1.0, abs(qr)) and abs(e - er) <= 1e-12 * er
    _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 1))
    assert np.abs(f.get_links() - orc.flow_steps(u, dims, 0.02, 1)).max() < 1e-12 * np.abs(u).max()


@pytest.mark.parametrize("prec,nr,tol", [("fp64", 18, 1e-12), ("fp32", 12, 1e-5)])
def test_batch_with_lattices_that_do_not_fit(ctx, without, prec, nr, tol):
    """A limit below two time slices of the larger lattices, which stand between smaller ones."""
    dims = [(4, 4, 4, 4), (12, 12, 12, 4), (2, 2, 4, 6), (12, 12, 8, 6), (4, 4, 4, 4)]
    without.set_loop_bytes(2 * 576 * (108 * (8 if prec == "fp64" else 4) + 8) - 1)  # 12 x 12 x 8: 576 indices
    single = [qcb.GaugeField(ctx, d, prec, nr) for d in dims]
    batched = [qcb.GaugeField(without, d, prec, nr) for d in dims]
    for k, (f, g) in enumerate(zip(single, batched)):
        f.hot_start(30 + k)
        g.hot_start(30 + k)
    batch = qcb.Batch(without, batched)
    n = len(dims)
    _, rec, graph = batch.run([6.0] * n, [1] * n, [0] * n, n_sweeps=0, n_hits=1, eps=0.02, n_groups=1, rk_per_group=1)
    assert graph
    batch.flow_steps(0.02, 3)
    q, e = batch.topo_qe()
    for k, f in enumerate(single):
        ref = qcb.observables.topo_charge_flowed(f, qcb.GradientFlow(0.02), 2, 1).reshape(-1, 3)
        _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 3))
        qr, er = qcb.observables.topo_q_e_clover_global(f)
        for a, b in ((rec[k][0], ref[0]), (rec[k][1], ref[1]), ((0, q[k], e[k]), (0, qr, er))):
            assert abs(a[1] - b[1]) <= 10 * tol * max(1.0, abs(b[1])) and abs(a[2] - b[2]) <= tol * b[2], k
        assert np.abs(batched[k].get_links() - f.get_links()).max() < 3 * tol, k
        f.close()


def test_server_and_slabs(ctx, without):
    dims = (4, 4, 4, 8)
    ref = qcb.GaugeField(ctx, dims, "fp64", 18)
    f = qcb.GaugeField(without, dims, "fp64", 18)
    for g in (ref, f):
        g.hot_start(8)
    without.sync()
    srv = qcb.Server(without, "fp64", 18, hbm_budget=1 << 26, quantum_steps=2)
    srv.submit_flow(f, 0.02, 5)
    srv.drain(60)
    job, = srv.poll(10)
    sl = qs.SlabLattice(without, dims, 2, "fp64", 18)
    sl.hot_start(8)
    sl.flow_steps(0.02, 5)
    _lib.check(_lib.lib().qcb_flow_steps(ref.h, 0.02, 5))
    q, e = qcb.observables.topo_q_e_clover_global(ref)
    for a, b in ((job.q, job.e), sl.topo_qe()):
        assert abs(a - q) < 1e-11 * max(1.0, abs(q)) and abs(b - e) < 1e-12 * e
    assert job.status == 0 and np.abs(sl.get_links() - ref.get_links()).max() < 1e-12
    sl.close()
    srv.close()
    ref.close()
