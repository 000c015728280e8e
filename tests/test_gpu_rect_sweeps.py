"""Checkerboard4 sub-sweeps with rectangle actions (nine warps to 32 links): extents of 4, where the two-step
neighbours on both sides coincide, and blocks that end inside a row, in the three storages.

FP64: 1e-11 against the oracle, heatbath on the oracle's Philox streams.  FP32: the staple of 24 paths is off
by at most 32 eps a path (four products), weighted 11.5 for Luescher-Weisz, 2.2e-5; the reflections of
a rough field amplify that up to fourfold over the sixteen sub-sweeps of a sweep.
"""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import LUESCHER_WEISZ, haar_links_numpy, rel_err

pytestmark = pytest.mark.gpu

EXTS = [(4, 4, 4, 4), (4, 8, 4, 12), (8, 4, 12, 4)]


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32_12"])
@pytest.mark.parametrize("ext", EXTS)
def test_overrelaxation(oracle, ext, prec):
    G = lt.GaugeField(ext, prec)
    G.upload(oracle.heatbath(ext, haar_links_numpy(ext, 4), 6.0, 2, 3, 0))
    W = G.download()
    lt.Iterator.Checkerboard4(lt.OverrelaxationSubgroupKernel(G, lt.LuescherWeiszAction(6.0)), 1)
    want = oracle.overrelax4(ext, W, 1, LUESCHER_WEISZ)
    assert rel_err(G.download(), want) < (1e-11 if prec == "fp64" else 1e-4)


@pytest.mark.parametrize("ext", EXTS)
def test_heatbath(oracle, ext):
    U = oracle.heatbath(ext, haar_links_numpy(ext, 4), 6.0, 2, 3, 0)
    G = lt.GaugeField(ext)
    G.upload(U)
    lt.Iterator.Checkerboard4(lt.HeatbathKernel(G, lt.LuescherWeiszAction(6.0), seed=9, counter=2), 1)
    assert rel_err(G.download(), oracle.heatbath4(ext, U, 6.0, 1, 9, 2, LUESCHER_WEISZ)) < 1e-11
    assert np.isfinite(G.check_links())
