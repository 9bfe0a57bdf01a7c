"""The plaquette's reduction and the measured sweep on every branch of their grids (planes side by
side, one block column, a grid-stride loop, chunked totals), against the oracle or the plaquettes of
single planes."""
import numpy as np
import pytest

import oracle as orc
import qcb

pytestmark = pytest.mark.gpu

STORAGES = [("fp64", 18), ("fp64", 12), ("fp32", 18), ("fp32", 12)]


@pytest.mark.parametrize("prec,nr", STORAGES)
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 4, 2, 6), (6, 10, 4, 2), (12, 12, 10, 14), (18, 16, 14, 20)])
def test_plaquette_and_measured_sweep(ctx, dims, prec, nr):
    """Mean plaquette against the oracle's: FP64 1e-13; FP32 3e-7, six roundings of 6e-8 in a site's
    value and a mean over sites that does not grow them.  A measured sweep's plaquette is that of
    its links."""
    u = orc.hot_philox(dims, 23)
    f = qcb.GaugeField(ctx, dims, prec, nr)
    f.set_links(u)
    tol = 1e-13 if prec == "fp64" else 3e-7
    got = f.get_links()
    assert abs(qcb.observables.mean_plaquette_global(f) - orc.plaquette(got, dims)) < tol
    hp = qcb.io.default_params()
    hp.beta, hp.N_samples, hp.N_sweeps, hp.N_hits = 5.8, 1, 1, 1
    p = qcb.heatbathcb.samples_plaquette(f, hp, qcb.PhiloxStream(seed=8, sweep=2))
    # Re tr(U A) / 3 of FP32 links is a sum of six terms: twice the bound
    assert abs(p - qcb.observables.mean_plaquette_global(f)) < 2 * tol
    f.close()


@pytest.mark.parametrize("dims", [(36, 32, 32, 32), (32, 32, 64, 36)])
def test_grid_stride_and_chunked_totals(ctx, dims):
    """More blocks than the grid holds, more partials than one block adds up: a cold lattice has
    plaquette 1 exactly, and a measured sweep agrees with its links' plaquette."""
    f = qcb.GaugeField(ctx, dims, "fp32", 12)
    assert qcb.observables.mean_plaquette_global(f) == 1.0
    hp = qcb.io.default_params()
    hp.beta, hp.N_samples, hp.N_sweeps, hp.N_hits = 6.0, 1, 1, 1
    p = qcb.heatbathcb.samples_plaquette(f, hp, qcb.PhiloxStream(seed=8, sweep=2))
    assert abs(p - qcb.observables.mean_plaquette_global(f)) < 6e-7
    f.close()
