"""Device memory: scratch that a call can do without never costs another call the memory that it
needs, and every call gives the same results without that scratch.

Results with and without it differ by the rounding of other products: FP64 1e-12 as elsewhere; FP32 links
1e-5, forces and momenta 5e-5 of their largest entry (24 paths of four roundings of 6 eps: 3.5e-5, and 1e-5
a smearing level)."""
import ctypes as C
import gc

import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu
EXT = (10, 8, 10, 8)   # above the size where FP32 flow stages take the plaquette planes


def held(limit=0, deny=0):
    n = C.c_uint64()
    assert lt.lib().lt_memory_test(limit, deny, C.byref(n)) == 0
    return n.value


@pytest.fixture(autouse=True)
def clean():
    gc.collect()
    assert lt.lib().lt_release_memory() == 0
    yield
    held()


def _links(ext=EXT):
    G = lt.GaugeField(ext)
    G.upload(haar_links_numpy(ext, 4))
    lt.UpdateSweeps(G, 6.0, 3, 1, 1, seed=3)
    U = G.download()
    G.close()
    return U


class Run:
    """One operation on handles of its own; run() may be repeated from the same links."""

    def __init__(self, op, prec, U, ext=EXT):
        self.op, self.U = op, U
        self.G = lt.GaugeField(ext, prec)
        self.fields = [self.G]
        if op.startswith("flow"):
            self.F = lt.GaugeField(ext, prec)
            self.fields.append(self.F)

    def run(self):
        G, op = self.G, self.op
        G.upload(self.U)
        if op.startswith("flow"):
            act = {"flow": None, "flow_lw": lt.LuescherWeiszAction(6.0), "flow_zeuthen": lt.ZeuthenFlow()}[op]
            lt.GradientFlowKernel(G, self.F, lt.RK3, act, 0.02)(2)
            return {"links": self.F.download()}
        if op == "force_lw":
            return {"force": lt.LuescherWeiszAction(6.0).Force(G)}
        bias = lt.MetaBiasPotential(-8, 8, 800, 0.05, 0.08, 10, 1000)
        bias.set_grid(np.linspace(0.0, 80.0, 801))
        if op == "force_metad":
            return {"force": lt.HMCMetaDKernel(G, bias, lt.WilsonAction(6.0), 1.0, 0.1, 2).CalculateTopologicalForce(dvdq=1.0)[0]}
        if op == "metad":
            k = lt.HMCMetaDKernel(G, bias, lt.WilsonAction(6.0), 0.3, 0.1, 2, integrator=lt.OMF_2)
        else:
            act = lt.LuescherWeiszAction(6.0) if op == "hmc_lw" else lt.WilsonAction(6.0)
            k = lt.HMCKernel(G, act, 0.3, integrator=lt.OMF_2)
        k.RandomMomentum(1)
        k.Integrate(2)
        return {"links": G.download(), "momenta": k.GetMomenta()}

    def close(self):
        for f in self.fields:
            f.close()


def same(a, b, prec):
    for k in a:
        tol = 1e-12 if prec == "fp64" else 1e-5 if k == "links" else 5e-5
        assert np.abs(a[k] - b[k]).max() < tol * max(np.abs(b[k]).max(), 1.0 if k == "links" else 0.0), k


OPS = ["flow", "flow_lw", "flow_zeuthen", "hmc", "hmc_lw", "metad", "force_lw", "force_metad"]
# two-row links: the Wilson force has no scratch beside the second link field
CASES = [(op, p) for p in ("fp64", "fp32", "fp32_12") for op in OPS if not (p == "fp32_12" and op == "flow")]


@pytest.mark.parametrize("op,prec", CASES)
def test_without_scratch_and_at_its_limit(op, prec):
    U = _links()
    base = held()
    r = Run(op, prec, U)
    want = r.run()
    with_scratch = held() - base
    r.close()
    assert lt.lib().lt_release_memory() == 0

    held(deny=1)
    r = Run(op, prec, U)
    same(r.run(), want, prec)
    need = held() - base
    assert need < with_scratch
    r.close()
    assert lt.lib().lt_release_memory() == 0

    # no more memory than a run without scratch takes, a little of it, and nearly all of it
    for more in (0, (with_scratch - need) // 3, with_scratch - need - 1):
        held(limit=base + need + more)
        r = Run(op, prec, U)
        for _ in range(2):
            same(r.run(), want, prec)
        assert held(limit=base + need + more) <= base + need + more
        r.close()


@pytest.mark.parametrize("op,prec", [("flow", "fp64"), ("hmc_lw", "fp32"), ("metad", "fp32_12")])
def test_two_handles(op, prec):
    """The idle scratch of one handle gives way to what another needs, and comes back when there is memory."""
    U = _links()
    base = held()
    held(deny=1)
    r = Run(op, prec, U)
    want = r.run()
    need = held() - base
    r.close()
    assert lt.lib().lt_release_memory() == 0
    held(limit=base + 2 * need)
    A, B = Run(op, prec, U), Run(op, prec, U)
    for r in (A, B, A, B):
        same(r.run(), want, prec)
    B.close()
    same(A.run(), want, prec)
    A.close()


def test_release_memory():
    U = _links()
    keep = lt.GaugeField((4, 4, 4, 4))   # the store is emptied with the last handle
    base = held()
    r = Run("flow", "fp64", U)
    want = r.run()
    before = held()
    planes = 6 * int(np.prod(EXT)) * 64
    assert lt.lib().lt_release_memory() == 0
    assert held() == before - planes
    same(r.run(), want, "fp64")
    assert held() == before
    r.close()
    assert held() == before   # in the store
    assert lt.lib().lt_release_memory() == 0
    assert held() == base
    keep.close()


def test_captured_call_keeps_its_scratch():
    """A graph holds the addresses of the scratch: after a captured call it stays with the handle."""
    import torch
    G = lt.GaugeField(EXT)
    G.upload(_links())
    k = lt.HMCKernel(G, lt.WilsonAction(6.0), 0.1, integrator=lt.OMF_2)
    k.RandomMomentum(1)
    s = C.c_void_p()
    assert lt.lib().lt_get_stream(G.handle, C.byref(s)) == 0
    omf2 = lambda: lt.lib().lt_omf2(G.handle, 6.0, 0.1, 1, None, None)  # noqa: E731
    assert lt.lib().lt_release_memory() == 0   # the store of _links' handle
    assert omf2() == 0
    G.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(s.value)):
        graph.capture_begin(capture_error_mode="thread_local")
        assert omf2() == 0
        graph.capture_end()
    before = held()
    assert lt.lib().lt_release_memory() == 0
    assert held() == before
    assert omf2() == 0   # the same scratch serves later calls
    G.synchronize()
    assert lt.lib().lt_release_memory() == 0
    assert held() == before
    del graph
    G.close()


def test_threads_at_the_limit():
    """Calls of several threads with memory for what they need, and scratch for some of them."""
    import threading
    U = _links()
    base = held()
    held(deny=1)
    r = Run("metad", "fp32", U)
    want = r.run()
    need = held() - base
    r.close()
    assert lt.lib().lt_release_memory() == 0
    held(limit=base + 3 * need + need // 2)
    bad = []

    def work():
        try:
            for _ in range(3):
                r = Run("metad", "fp32", U)
                same(r.run(), want, "fp32")
                r.close()
        except Exception as e:   # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_store_keeps_the_newest():
    """A store that is full gives up its oldest buffers: fields of a size used now stay after fields of a size
    that is not asked for again have filled it."""
    small, big = (8, 8, 8, 8), (16, 8, 8, 8)
    keep = lt.GaugeField((4, 4, 4, 4))
    nb = 8 * 72 * int(np.prod(small))
    held(limit=8 * 5 * nb)   # the store keeps an eighth: two big fields' links, or five small ones'
    old = [lt.GaugeField(big) for _ in range(3)]
    for f in old:
        f.close()
    lt.GaugeField(small).close()
    before = held(limit=8 * 5 * nb)
    f = lt.GaugeField(small)   # from the store
    assert held(limit=8 * 5 * nb) == before
    f.close()
    keep.close()


def test_ensemble_from_the_store():
    """An ensemble's buffers and the link copies of its tuning come from the store: a destroyed handle's buffers
    serve them, or give way to them."""
    keep = [lt.GaugeField((8, 8, 8, 8)) for _ in range(2)]
    lt.GaugeField((12, 8, 8, 8)).close()
    before = held()
    E = lt.Ensemble(keep, [6.0, 6.0], seed=1)
    assert held() > before
    lt.GaugeField((8, 8, 8, 8)).close()
    full = held()
    held(limit=full)   # the tuning copies 4.7 MB of links: the 2.4 and 3.5 MB of the store
    E.autotune()
    assert held() <= full
    E.sweeps(1)
    del E
    for f in keep:
        f.close()
