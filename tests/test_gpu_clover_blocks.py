"""Q, E, their timeslices and the plaquette charge from blocks of six planes by 32 sites, on lattices with
partly empty blocks and timeslices (8, 96, 36 and 240 sites), the three storages: against the FP64 oracle on
the links as stored (products are FP64 in every storage), and against the flow measurement's own sums.
Bound: FP64 sums of up to 720 densities of twelve products each, 1e-11 of the sum of their absolute values."""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32_12"])
@pytest.mark.parametrize("ext", [(2, 2, 2, 2), (2, 4, 6, 4), (8, 6, 2, 6), (6, 2, 10, 12)])
def test_observables(oracle, ext, prec):
    G = lt.GaugeField(ext, prec)
    G.upload(oracle.heatbath(ext, haar_links_numpy(ext, 5), 5.8, 2, 7, 0))
    W = G.download()
    want = oracle.measure(ext, W, 6.0)
    q, e = lt.CloverObservables(G)
    # two-row links: the third row is rebuilt in FP32 on both sides, up to its rounding
    tol = 1e-6 if prec == "fp32_12" else 1e-11
    assert q == pytest.approx(float(np.sum(want["q_t"])), abs=tol)
    assert e == pytest.approx(float(np.sum(want["e_t"])), rel=tol)
    np.testing.assert_allclose(lt.TopChargeCloverTimeslice(G).sum(), q, atol=1e-12)
    np.testing.assert_allclose(lt.EnergyDensityCloverTimeslice(G).sum(), e, rtol=1e-12)
    F = lt.GaugeField(ext, prec)
    p, qf, ef = lt.GradientFlowKernel(G, F, lt.RK3, None, 0.01).Measure(1, 0)
    assert p[0] == pytest.approx(lt.PlaquetteSum(G), rel=1e-12)
    assert qf[0] == pytest.approx(q, abs=1e-12) and ef[0] == pytest.approx(e, rel=1e-12)
