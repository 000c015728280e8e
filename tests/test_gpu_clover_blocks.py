"""Q, E, their timeslices and the plaquette charge from blocks of six planes by 32 sites, on lattices with
partly empty blocks and timeslices (8, 96, 72, 240 and 4,536 sites a timeslice), and from one thread a site on
two-row links (the last, 72,576 sites), the three storages: against the FP64 oracle on the links as stored
(products are FP64 in every storage, and the third row of two-row links is rebuilt alike in the kernels and
in a download), and against the flow measurement's own sums.
Bound: FP64 densities of twelve products each, summed with compensation: 1e-11 of E, and of Q where it is
not small; 1e-12 between the library's own sums."""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32_12"])
@pytest.mark.parametrize("ext", [(2, 2, 2, 2), (2, 4, 6, 4), (8, 6, 2, 6), (6, 2, 10, 12), (16, 18, 14, 18)])
def test_observables(oracle, ext, prec):
    G = lt.GaugeField(ext, prec)
    G.upload(oracle.heatbath(ext, haar_links_numpy(ext, 5), 5.8, 2, 7, 0))
    W = G.download()
    want = oracle.measure(ext, W, 6.0)
    q, e = lt.CloverObservables(G)
    assert q == pytest.approx(float(np.sum(want["q_t"])), abs=1e-11)
    assert e == pytest.approx(float(np.sum(want["e_t"])), rel=1e-11)
    np.testing.assert_allclose(lt.TopChargeCloverTimeslice(G), want["q_t"], atol=1e-11)
    np.testing.assert_allclose(lt.EnergyDensityCloverTimeslice(G), want["e_t"], rtol=1e-11)
    assert lt.TopChargePlaquette(G) == pytest.approx(want["Q_plaq"], abs=1e-11)
    np.testing.assert_allclose(lt.TopChargeCloverTimeslice(G).sum(), q, atol=1e-12)
    np.testing.assert_allclose(lt.EnergyDensityCloverTimeslice(G).sum(), e, rtol=1e-12)
    F = lt.GaugeField(ext, prec)
    p, qf, ef = lt.GradientFlowKernel(G, F, lt.RK3, None, 0.01).Measure(1, 0)
    assert p[0] == pytest.approx(lt.PlaquetteSum(G), rel=1e-12)
    assert qf[0] == pytest.approx(q, abs=1e-12) and ef[0] == pytest.approx(e, rel=1e-12)
