"""The plaquette-loop field behind the Wilson flow and the clover: shapes at the edges of its
blocks and planes against the oracle, and a lattice whose loops do not fit into the loop buffer
at once (worked through in rounds of time slices) against the same lattice cut into slabs."""
import numpy as np
import pytest

import oracle as orc
import qcb
from qcb import _lib
from qcb import slabs as qs

pytestmark = pytest.mark.gpu

# extents of two (both neighbours are one site), remainders of the 32- and 128-site blocks, one
# long direction each
DIMS = [(2, 2, 2, 2), (2, 2, 4, 6), (4, 2, 2, 10), (34, 4, 2, 2), (2, 18, 4, 6), (4, 4, 22, 4), (6, 6, 2, 26), (8, 8, 8, 4)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,nr", [("fp64", 18), ("fp64", 12), ("fp32", 18), ("fp32", 12)])
def test_flow_step_and_clover_match_oracle(ctx, dims, prec, nr):
    """One RK3 step and Q, E before and after it.  FP32 links: a loop is three products of six
    roundings each, a link's force twelve loops and transports of them (below 600 roundings of
    6e-8, times the step of 0.02), the exponential and the product a dozen more for each of three
    stages: 1e-5 covers them.  E and Q follow from loops of the same accuracy."""
    u = orc.hot_philox(dims, 4242)
    f = qcb.GaugeField(ctx, dims, prec, nr)
    f.set_links(u)
    tol = 1e-12 if prec == "fp64" else 1e-5

    def check_qe(ref):
        q, e = qcb.observables.topo_q_e_clover_global(f)
        (_, qr, er), = orc.flow_measure(ref, dims, 0.02, 1, 0).reshape(-1, 3)
        assert abs(q - qr) <= 10 * tol * max(1.0, abs(qr)), (q, qr)
        assert abs(e - er) <= tol * er, (e, er)

    check_qe(u)
    _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 1))
    ref = orc.flow_steps(u, dims, 0.02, 1)
    assert np.abs(f.get_links() - ref).max() < tol
    check_qe(ref)
    f.close()


@pytest.mark.parametrize("eps", [0.11, 0.6])
def test_large_steps_match_oracle(ctx, eps):
    """Steps at which some (0.11) and all (0.6) exponentials need every term of the series."""
    dims = (4, 6, 4, 6)
    u = orc.hot_philox(dims, 77)
    f = qcb.GaugeField(ctx, dims)
    f.set_links(u)
    _lib.check(_lib.lib().qcb_flow_steps(f.h, eps, 1))
    assert np.abs(f.get_links() - orc.flow_steps(u, dims, eps, 1)).max() < 1e-12
    f.close()


def test_rounds_of_time_slices_match_slabs(ctx):
    """64^3 x 10 in FP64 has 1.13 GB of loops: rounds of eight and two slices through the buffer,
    the slice before a round kept from the one before it.  Slabs of two slices hold theirs whole;
    the links are the same bit for bit, Q and E to the order of the sums."""
    dims = (64, 64, 64, 10)
    whole = qcb.GaugeField(ctx, dims, "fp64", 12)
    whole.hot_start(31)
    sl = qs.SlabLattice(ctx, dims, 5, "fp64", 12)
    sl.hot_start(31)
    qw, ew = qcb.observables.topo_q_e_clover_global(whole)
    q, e = sl.topo_qe()
    assert abs(q - qw) < 1e-11 * max(1.0, abs(qw)) and abs(e - ew) < 1e-12 * ew
    _lib.check(_lib.lib().qcb_flow_steps(whole.h, 0.02, 1))
    sl.flow_steps(0.02, 1)
    assert np.array_equal(sl.get_links(), whole.get_links())
    sl.close()
    whole.close()
