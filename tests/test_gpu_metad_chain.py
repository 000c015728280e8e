"""The metadynamics force with the corner sums of the clover derivative and the conjugated Lambdas of the
recursion, on lattices with partly empty blocks and extents of 2, against the FP64 oracle on the links as
stored.  FP64 1e-11 as elsewhere; FP32 1e-5 of the largest entry a stout level (each level's recursion
repeats some forty products of rounded matrices: 40 * 3 eps = 7e-6), the bound of the 16^4 comparison.
"""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32_12"])
@pytest.mark.parametrize("n_stout", [0, 1, 3])
@pytest.mark.parametrize("ext", [(2, 2, 2, 2), (2, 4, 6, 2), (6, 2, 10, 6)])
def test_force(oracle, ext, n_stout, prec):
    G = lt.GaugeField(ext, prec)
    G.upload(oracle.heatbath(ext, haar_links_numpy(ext, 5), 5.8, 2, 7, 0))
    W = G.download()
    bias = lt.MetaBiasPotential(-8, 8, 800, 0.05, 0.08, 10, 1000)
    k = lt.HMCMetaDKernel(G, bias, lt.WilsonAction(6.0), 1.0, 0.1, n_stout)
    F, q = k.CalculateTopologicalForce(dvdq=0.7)
    want, wq = oracle.metad_force(ext, W, 0.1, n_stout, 0.7)
    tol = 1e-11 if prec == "fp64" else 1e-5 * (1 + n_stout)
    assert np.abs(F - want).max() < tol * np.abs(want).max()
