"""The energy density of FP32 links has hardly a systematic error: rounding to nearest averages out over the
planes of a lattice."""
import numpy as np
import pytest

import qcb
from qcb import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr", [12, 18])
def test_systematic_error_of_the_energy_density(ctx, nr):
    """Mean of (E - E64) / E64 over twelve fields of 16^4 against the same links in FP64.  A plane's |F|^2
    carries some tens of roundings of 6e-8: about 3e-7, over 4e5 planes 5e-10 a field and 1.5e-10 for
    the mean.  8e-10 is a hundredth of a rounding and that once more; a third of the trace rounded in each
    diagonal element is 1.1e-9."""
    dims = (16, 16, 16, 16)
    h, d = qcb.GaugeField(ctx, dims), qcb.GaugeField(ctx, dims)
    f = qcb.GaugeField(ctx, dims, "fp32", nr)
    rel = []
    for k in range(12):
        h.hot_start(40 + k)
        _lib.check(_lib.lib().qcb_heatbath(h.h, 6.0, 20, 1, k, 0))
        f.copy_from(h)
        d.copy_from(f)
        _, e = qcb.observables.topo_q_e_clover_global(f)
        _, ref = qcb.observables.topo_q_e_clover_global(d)
        rel.append((e - ref) / ref)
    assert abs(np.mean(rel)) < 8e-10, (np.mean(rel), np.std(rel))
    for g in (h, d, f):
        g.close()


def test_energy_density_of_links_slightly_off_unitarity(ctx):
    """FP32 18-real links with |U| a few roundings above 1, as a handful of sweeps leaves them: E is that of the
    stored links (FP64 on the same links), within the rounding noise of 25000 planes (3e-7 / 160 each
    field, ten times that), where loops moved along them as if they were unitary are off by 8e-7."""
    dims = (8, 8, 8, 8)
    h, d = qcb.GaugeField(ctx, dims), qcb.GaugeField(ctx, dims)
    f = qcb.GaugeField(ctx, dims, "fp32", 18)
    h.hot_start(3)
    _lib.check(_lib.lib().qcb_heatbath(h.h, 6.0, 20, 1, 7, 0))
    f.set_links(h.get_links() * (1 + 2e-7))
    d.copy_from(f)
    _, e = qcb.observables.topo_q_e_clover_global(f)
    _, ref = qcb.observables.topo_q_e_clover_global(d)
    assert abs(e - ref) < 2e-8 * ref, (e - ref) / ref
    for g in (h, d, f):
        g.close()
