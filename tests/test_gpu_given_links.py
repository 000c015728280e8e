"""Flows, molecular dynamics and the metadynamics force start from the links as they are given: until a
projection (a flow stage, a drift, a stout level) has made them unitary to the storage's rounding, forces
are multiplied out, whatever the links' distance from SU(3).

FP64: links rounded to FP32, as a configuration file of that accuracy holds them; 1e-12 as elsewhere (a force
that takes them for unitary is off by 1e-7).  FP32: links with entries off by up to 1e-3, which nothing
refuses (check_links reports them); a force of up to 24 paths of three products, each rounded by at most
6 eps, is off by 24 * 4 * 6 eps = 3.5e-5 of its largest entry, and by 1e-5 a smearing level on top
(test_gpu_metad_chain.py).
"""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy, rel_err

pytestmark = pytest.mark.gpu
EXT = (4, 6, 2, 6)


def links(oracle, ext=EXT):
    return oracle.heatbath(ext, haar_links_numpy(ext, 5), 5.8, 2, 7, 0)


def fp32_accurate(oracle, ext=EXT):
    return links(oracle, ext).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("integrator,iid", [(lt.Euler, 0), (lt.RK2, 1), (lt.RK3, 2), (lt.RK3W7, 3)])
def test_flow_fp64(oracle, integrator, iid):
    U = fp32_accurate(oracle)
    G, F = lt.GaugeField(EXT), lt.GaugeField(EXT)
    G.upload(U)
    for _ in range(2):   # the second flow finds the handle's scratch fields in place
        lt.GradientFlowKernel(G, F, integrator, None, 0.02)(3)
        assert rel_err(F.download(), oracle.flow(EXT, U, 0.02, 3, iid)) < 1e-12
    # a resumed flow after a link has been replaced
    F.set_link(77, 2, U[0, 0, ..., 0] + 1j * U[0, 0, ..., 1])
    W = F.download()
    lt.GradientFlowKernel(G, F, integrator, None, 0.02).Resume(2)
    assert rel_err(F.download(), oracle.flow(EXT, W, 0.02, 2, iid)) < 1e-12


def test_flow_measure_fp64(oracle):
    U = fp32_accurate(oracle)
    G, F = lt.GaugeField(EXT), lt.GaugeField(EXT)
    G.upload(U)
    p, q, e = lt.GradientFlowKernel(G, F, lt.RK3, None, 0.02).Measure(3, 2)
    for k in range(3):
        W = oracle.flow_rk3(EXT, U, 0.02, 2 * (k + 1))
        assert p[k] == pytest.approx(oracle.plaquette_sum(EXT, W), rel=1e-12)
        assert e[k] == pytest.approx(oracle.energy(EXT, W), rel=1e-11)
        assert q[k] == pytest.approx(oracle.topcharge(EXT, W), rel=1e-10, abs=1e-12)


@pytest.mark.parametrize("integrator", ["Leapfrog", "OMF_2", "OMF_4_slow", "OMF_4_friction_slow"])
def test_md_fp64(oracle, integrator):
    U = fp32_accurate(oracle)
    G = lt.GaugeField(EXT)
    G.upload(U)
    integ = getattr(lt.Integrators.HMC, integrator)
    k = lt.HMCKernel(G, lt.WilsonAction(6.0), 0.3, integrator=integ)
    k.RandomMomentum(1)
    P = k.GetMomenta()
    k.Integrate(3)
    Uo, Po = oracle.md_integrate(EXT, U, P, 6.0, 0.3, 3, integ.ID)[:2]
    assert rel_err(G.download(), Uo) < 1e-12
    assert rel_err(k.GetMomenta(), Po) < 1e-12


def off_unitary(oracle, ext=EXT):
    U = links(oracle, ext)
    return U + 1e-3 * np.random.default_rng(3).uniform(-1.0, 1.0, U.shape)


def test_kick_fp32(oracle):
    """A kick alone: leapfrog with drifts that move no link's force by more than the bound."""
    G = lt.GaugeField(EXT, "fp32")
    G.upload(off_unitary(oracle))
    W = G.download()
    tau = 1e-3
    k = lt.HMCKernel(G, lt.WilsonAction(6.0), tau, integrator=lt.Leapfrog)
    k.SetMomenta(np.zeros(W.shape))
    k.Integrate(1)
    # the first half kick alone: the oracle's whole step from the same links and no momenta
    P = oracle.md_integrate(EXT, W, np.zeros(W.shape), 6.0, tau, 1, lt.Leapfrog.ID)[1]
    got = k.GetMomenta()
    assert np.abs(got - P).max() < 3.5e-5 * np.abs(P).max()


@pytest.mark.parametrize("ext", [EXT, (10, 8, 10, 8)])   # below and above the size where FP32 stages take planes
def test_flow_fp32(oracle, ext):
    G, F = lt.GaugeField(ext, "fp32"), lt.GaugeField(ext, "fp32")
    G.upload(off_unitary(oracle, ext))
    W = G.download()
    lt.GradientFlowKernel(G, F, lt.Euler, None, 0.1)(1)
    want = oracle.flow(ext, W, 0.1, 1, 0)
    step = np.abs(want - oracle.flow(ext, W, 0.0, 1, 0)).max()
    # the step itself to 3.5e-5 of its largest entry; the projected links to 8 eps
    assert np.abs(F.download() - want).max() < 3.5e-5 * step + 8 * 2.0 ** -24


@pytest.mark.parametrize("n_stout", [1, 2])
def test_metad_force_fp32(oracle, n_stout):
    G = lt.GaugeField(EXT, "fp32")
    G.upload(off_unitary(oracle))
    W = G.download()
    bias = lt.MetaBiasPotential(-8, 8, 800, 0.05, 0.08, 10, 1000)
    F, _ = lt.HMCMetaDKernel(G, bias, lt.WilsonAction(6.0), 1.0, 0.1, n_stout).CalculateTopologicalForce(dvdq=0.7)
    want, _ = oracle.metad_force(EXT, W, 0.1, n_stout, 0.7)
    assert np.abs(F - want).max() < (3.5e-5 + 1e-5 * n_stout) * np.abs(want).max()
