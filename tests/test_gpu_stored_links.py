"""The force and the clover are those of the stored links, whether or not these are exactly unitary:
18-real storage holds whatever was written to it, such as links from a single-precision file."""
import numpy as np
import pytest

import oracle as orc
import qcb
from qcb import _lib
from qcb import slabs as qs

pytestmark = pytest.mark.gpu

DIMS = [(4, 6, 8, 4), (2, 2, 4, 6), (6, 4, 4, 10)]


def off_by(u, size, seed, only=None):
    """u with links moved off SU(3) by relative noise of the given size (of all links, or of the
    fraction `only` of them)."""
    rng = np.random.default_rng(seed)
    n = rng.standard_normal(u.shape) + 1j * rng.standard_normal(u.shape)
    if only is not None:
        n = n * (rng.random(u.shape[:5]) < only)[..., None, None]
    return u + size * n


def projected(u):
    """Rows 0 and 1 orthonormalised, row 2 their conjugate cross product (FP32 flow steps end so)."""
    r0 = u[..., 0, :] / np.linalg.norm(u[..., 0, :], axis=-1, keepdims=True)
    r1 = u[..., 1, :] - (r0.conj() * u[..., 1, :]).sum(-1, keepdims=True) * r0
    r1 = r1 / np.linalg.norm(r1, axis=-1, keepdims=True)
    return np.stack([r0, r1, np.cross(r0, r1).conj()], axis=-2)


def check(ctx, u, dims, prec, tol):
    """Q, E and one RK3 step against the oracle."""
    f = qcb.GaugeField(ctx, dims, prec, 18)
    f.set_links(u)
    q, e = qcb.observables.topo_q_e_clover_global(f)
    (_, qr, er), = orc.flow_measure(u, dims, 0.02, 1, 0).reshape(-1, 3)
    assert abs(q - qr) <= 10 * tol * max(1.0, abs(qr)), (q, qr)
    assert abs(e - er) <= tol * er, (e, er)
    _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 1))
    ref = orc.flow_steps(u, dims, 0.02, 1)
    got = f.get_links()
    if prec == "fp32":
        ref = projected(ref)
    assert np.abs(got - ref).max() < tol * max(1.0, np.abs(u).max())
    f.close()


@pytest.mark.parametrize("dims", DIMS)
def test_links_of_single_precision_in_fp64(ctx, dims):
    """FP64 arithmetic on links that are unitary to 1e-7: the bounds of the FP64 path (test_gpu_loops)."""
    u = orc.hot_philox(dims, 5).astype(np.complex64).astype(np.complex128)
    check(ctx, u, dims, "fp64", 1e-12)


@pytest.mark.parametrize("size", [2e-14, 1e-12, 1e-9, 1e-4])
def test_links_off_su3_in_fp64(ctx, size):
    """On both sides of the bound up to which a link counts as unitary.  Below it the relative error of a
    transported loop is at most the bound, 1e-12; a noise of 2e-14 stays a factor of ten below."""
    dims = DIMS[0]
    check(ctx, off_by(orc.hot_philox(dims, 6), size, 1), dims, "fp64", 1e-12)


@pytest.mark.parametrize("only", [0.003, 0.2])
def test_a_few_links_off_su3(ctx, only):
    """Sites whose loops are moved along good and bad links side by side."""
    dims = (8, 6, 4, 6)
    check(ctx, off_by(orc.hot_philox(dims, 7), 1e-3, 2, only), dims, "fp64", 1e-12)


@pytest.mark.parametrize("dims", DIMS[:2])
def test_links_off_su3_in_fp32(ctx, dims):
    """FP32 links 1e-2 off SU(3), rounded to their storage; the bounds of the FP32 path (test_gpu_loops)."""
    u = off_by(orc.hot_philox(dims, 8), 1e-2, 3).astype(np.complex64).astype(np.complex128)
    check(ctx, u, dims, "fp32", 1e-5)


def test_batch_and_single_are_the_same_off_su3(ctx):
    """One lattice alone and in a batch, and the flow's record against the clover alone."""
    dims = [(4, 4, 4, 4), (4, 6, 8, 4), (2, 2, 4, 6)]
    us = [off_by(orc.hot_philox(d, 9 + k), 1e-4, k, 0.1) for k, d in enumerate(dims)]
    single = [qcb.GaugeField(ctx, d, "fp64", 18) for d in dims]
    batched = [qcb.GaugeField(ctx, d, "fp64", 18) for d in dims]
    for f, g, u in zip(single, batched, us):
        f.set_links(u)
        g.set_links(u)
    batch = qcb.Batch(ctx, batched)
    q, e = batch.topo_qe()
    for k, f in enumerate(single):
        rec = qcb.observables.topo_charge_flowed(f, qcb.GradientFlow(0.02), 1, 1).reshape(-1, 3)
        ref = orc.flow_measure(us[k], dims[k], 0.02, 1, 1).reshape(-1, 3)
        assert np.abs(rec - ref).max() < 1e-11
        assert abs(q[k] - rec[0, 1]) < 1e-12 and abs(e[k] - rec[0, 2]) < 1e-12 * e[k]
        _lib.check(_lib.lib().qcb_flow_steps(f.h, 0.02, 2))
    batch.flow_steps(0.02, 2)
    ctx.sync()
    for f, g in zip(single, batched):
        assert np.array_equal(f.get_links(), g.get_links())
    batch.close()


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec,nr,tol", [("fp64", 12, 1e-13), ("fp64", 18, 1e-13), ("fp32", 12, 1e-6), ("fp32", 18, 1e-6)])
def test_plaquette_is_that_of_the_stored_links(ctx, dims, prec, nr, tol):
    """12-real storage keeps rows 0 and 1 as they were written; the link is these and their conjugate cross
    product.  A plaquette of FP32 links is two products and a trace, below 20 roundings of 6e-8, and the
    mean of hundreds of them is closer."""
    u = off_by(orc.hot_philox(dims, 12), 1e-2, 5)
    f = qcb.GaugeField(ctx, dims, prec, nr)
    f.set_links(u)
    stored = f.get_links()
    assert np.abs(stored[..., :2, :] - u[..., :2, :]).max() < 1e-7
    ref = orc.plaquette(stored, dims)
    assert abs(qcb.observables.mean_plaquette_global(f) - ref) < tol
    batch = qcb.Batch(ctx, [f])
    assert abs(batch.plaquette()[0] - ref) < tol
    batch.close()
    f.close()


@pytest.mark.parametrize("prec,size", [("fp64", 1e-4), ("fp32", 1e-3)])
def test_rounds_and_slabs_are_the_same_off_su3(ctx, prec, size):
    """Bad links next to the edges of rounds of time slices and of slabs, where the loops' neighbours come
    from the round before or from a halo: the links are those of the whole lattice, bit for bit."""
    dims = (4, 6, 4, 12)
    u = off_by(orc.hot_philox(dims, 14), size, 6, 0.1)
    c = qcb.Context(0)
    whole, rounds = qcb.GaugeField(ctx, dims, prec, 18), qcb.GaugeField(c, dims, prec, 18)
    c.set_loop_bytes(3 * 64 * (108 * (8 if prec == "fp64" else 4) + 8))  # 48 indices a slice: three or four
    sl = qs.SlabLattice(ctx, dims, 3, prec, 18)
    for f in (whole, rounds, sl):
        f.set_links(u)
    q, e = qcb.observables.topo_q_e_clover_global(whole)
    for a, b in (qcb.observables.topo_q_e_clover_global(rounds), sl.topo_qe()):
        assert abs(a - q) <= 1e-12 * max(1.0, abs(q)) and abs(b - e) <= 1e-12 * e
    _lib.check(_lib.lib().qcb_flow_steps(whole.h, 0.02, 2))
    _lib.check(_lib.lib().qcb_flow_steps(rounds.h, 0.02, 2))
    sl.flow_steps(0.02, 2)
    assert np.array_equal(rounds.get_links(), whole.get_links())
    assert np.array_equal(sl.get_links(), whole.get_links())
    sl.close()
    c.close()
    whole.close()
