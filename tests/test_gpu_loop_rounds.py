"""A small plaquette-loop buffer: lattices in rounds of time slices, alone, in a batch between lattices
that fit, and as jobs of a server.  A site's loops, its links and its share of Q and E do not depend on
the rounds; only the order of the sums of Q and E does (FP64 sums: 1e-12)."""
import numpy as np
import pytest

import qcb
from qcb import _lib

pytestmark = pytest.mark.gpu


def loop_bytes(dims, prec, slices):
    """Bytes of `slices` time slices of loops: eight reals and a trace for each plane and parity, a byte a link."""
    stride = (slices * dims[0] * dims[1] * dims[2] // 2 + 63) // 64 * 64
    return stride * (6 * 2 * 9 * (8 if prec == "fp64" else 4) + 8)


@pytest.fixture
def limited():
    """A context of its own, whose loop buffer a test may limit."""
    c = qcb.Context(0)
    yield c
    c.close()


def fields(c, dims, prec, nr):
    out = []
    for k, d in enumerate(dims):
        f = qcb.GaugeField(c, d, prec, nr)
        f.hot_start(70 + k)
        out.append(f)
    return out


def close(q, e, qr, er):
    return abs(q - qr) <= 1e-12 * max(1.0, abs(qr)) and abs(e - er) <= 1e-12 * er


def flowed(f, groups, rk):
    return qcb.observables.topo_charge_flowed(f, qcb.GradientFlow(0.02), groups, rk).reshape(-1, 3)


@pytest.mark.parametrize("prec,nr", [("fp64", 18), ("fp64", 12), ("fp32", 18), ("fp32", 12)])
@pytest.mark.parametrize("dims,slices", [((4, 6, 8, 10), 2), ((4, 6, 8, 10), 3), ((4, 6, 8, 10), 8), ((2, 2, 4, 6), 2),
                                         ((12, 4, 6, 4), 3)])
def test_rounds_of_one_lattice(ctx, limited, dims, slices, prec, nr):
    """Records before odd and even steps, and three steps in place."""
    whole, = fields(ctx, [dims], prec, nr)
    f, = fields(limited, [dims], prec, nr)
    limited.set_loop_bytes(loop_bytes(dims, prec, slices))
    assert close(*qcb.observables.topo_q_e_clover_global(f), *qcb.observables.topo_q_e_clover_global(whole))
    for a, b in zip(flowed(f, 3, 1), flowed(whole, 3, 1)):
        assert a[0] == b[0] and close(a[1], a[2], b[1], b[2])
    for g in (f, whole):
        _lib.check(_lib.lib().qcb_flow_steps(g.h, 0.02, 3))
    assert np.array_equal(f.get_links(), whole.get_links())
    whole.close()


DIMS = [(4, 4, 4, 4), (6, 4, 4, 6), (8, 8, 8, 8), (4, 4, 4, 4), (6, 6, 6, 6), (4, 6, 8, 10), (2, 2, 4, 6)]


# of the loops of 8^4, in time slices: all lattices at once, groups of whole lattices, 8^4 (and with
# three slices 4x6x8x10) in rounds between groups of the others
@pytest.mark.parametrize("slices", [40, 8, 5, 3])
@pytest.mark.parametrize("prec,nr", [("fp64", 18), ("fp32", 12)])
def test_groups_and_rounds_of_a_batch(ctx, limited, slices, prec, nr):
    single = fields(ctx, DIMS, prec, nr)
    batched = fields(limited, DIMS, prec, nr)
    limited.set_loop_bytes(loop_bytes((8, 8, 8, 8), prec, slices))
    batch = qcb.Batch(limited, batched)
    n = len(DIMS)
    _, rec, graph = batch.run([6.0] * n, [1] * n, [0] * n, n_sweeps=0, n_hits=1, eps=0.02, n_groups=2, rk_per_group=1)
    assert graph
    q, e = batch.topo_qe()
    batch.flow_steps(0.02, 3)
    q3, e3 = batch.topo_qe()
    limited.sync()
    for k, f in enumerate(single):
        ref = flowed(f, 3, 1)
        for g in range(3):
            assert close(rec[k][g][1], rec[k][g][2], ref[g][1], ref[g][2]), (k, g)
        assert close(q[k], e[k], ref[0][1], ref[0][2]), k
        _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 3))
        assert np.array_equal(batched[k].get_links(), f.get_links()), k
        assert close(q3[k], e3[k], *qcb.observables.topo_q_e_clover_global(f)), k
        f.close()


@pytest.mark.parametrize("slices", [8, 3])
def test_groups_and_rounds_of_a_server(ctx, limited, slices):
    """Flow jobs of different lengths, several ticks each."""
    single = fields(ctx, DIMS, "fp32", 12)
    jobs = fields(limited, DIMS, "fp32", 12)
    limited.sync()
    limited.set_loop_bytes(loop_bytes((8, 8, 8, 8), "fp32", slices))
    srv = qcb.Server(limited, "fp32", 12, hbm_budget=1 << 28, quantum_steps=3)
    steps = [3 + 2 * k for k in range(len(DIMS))]
    ids = {srv.submit_flow(f, 0.02, n): k for k, (f, n) in enumerate(zip(jobs, steps))}
    srv.drain(60)
    results = srv.poll(100)
    assert len(results) == len(DIMS)
    for r in results:
        k = ids[r.id]
        assert r.status == 0
        _lib.check(_lib.lib().qcb_flow_steps(single[k].h, 0.02, steps[k]))
        assert close(r.q, r.e, *qcb.observables.topo_q_e_clover_global(single[k])), k
    srv.close()
    for f in single:
        f.close()
