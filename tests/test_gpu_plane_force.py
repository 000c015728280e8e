"""The Wilson force of all links in the three storages, as a force, as fused kicks and drifts, as the kick that
ends a trajectory and as flow stages, on lattices with partly empty blocks (V = 16, 96, 288, 720 and 6,000
sites against 32 a block) and extents of 2, against the FP64 oracle on the links as they are stored.

What runs where: the plaquette planes (k_plaq_planes, k_plane_step) serve FP64 flow stages after the
first, FP32 ones above 4,736 sites (the last lattice), and FP64 and FP32 kicks after the first drift, the last of
them without a drift; a force and what comes first take the staple, and two-row links always do.

Bounds: FP64 1e-12.  FP32: a plaquette entry is three products of unit rows, each a sum of three
complex products rounded by at most 6 eps, the conjugation two more; six of them add up to at most
6 * 5 * 6 eps = 1.1e-5 absolute, on a force whose largest entries are of order one; a step moves a
link by at most the step size times that.
"""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy, rel_err

pytestmark = pytest.mark.gpu

EXTS = [(2, 2, 2, 2), (2, 4, 6, 2), (4, 6, 2, 6), (6, 2, 10, 6), (6, 10, 10, 10)]
TOL = {"fp64": 1e-12, "fp32": 1.1e-5, "fp32_12": 1.1e-5}


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32_12"])
@pytest.mark.parametrize("ext", EXTS)
def test_force_flow_and_md(oracle, ext, prec):
    G = lt.GaugeField(ext, prec)
    G.upload(oracle.heatbath(ext, haar_links_numpy(ext, 5), 5.8, 2, 7, 0))
    W = G.download()
    want = oracle.gauge_force(ext, W, 6.0)
    assert np.abs(lt.WilsonAction(6.0).Force(G) - want).max() < TOL[prec] * max(1.0, np.abs(want).max())
    F = lt.GaugeField(ext, prec)
    lt.GradientFlowKernel(G, F, lt.RK3, None, 0.02)(2)
    assert rel_err(F.download(), oracle.flow_rk3(ext, W, 0.02, 2)) < TOL[prec]
    k = lt.HMCKernel(G, lt.WilsonAction(6.0), 0.3, integrator=lt.OMF_2)
    k.RandomMomentum(1)
    P = k.GetMomenta()
    k.Integrate(3)
    Uo, Po = oracle.omf2(ext, W, P, 6.0, 0.3, 3)[:2]
    assert rel_err(G.download(), Uo) < TOL[prec]
    assert np.abs(k.GetMomenta() - Po).max() < 10.0 * TOL[prec]


def test_given_links_of_fp32_accuracy(oracle):
    """An FP64 handle with links rounded to FP32 (unitary to 1e-7 only): the force and the clover derivative
    of the links as given, to FP64 rounding."""
    ext = (4, 6, 2, 6)
    U = oracle.heatbath(ext, haar_links_numpy(ext, 5), 5.8, 2, 7, 0).astype(np.float32).astype(np.float64)
    G = lt.GaugeField(ext)
    G.upload(U)
    assert rel_err(lt.WilsonAction(6.0).Force(G), oracle.gauge_force(ext, U, 6.0)) < 1e-12
    assert rel_err(lt.CloverDerivative(G), oracle.clover_derivative(ext, U)) < 1e-12
    assert lt.TopChargeClover(G) == pytest.approx(oracle.topcharge(ext, U), rel=1e-11, abs=1e-13)
