"""The store of device buffers behind the handles: buffers serve the next handle of the same size, results
do not depend on what a buffer held, threads may create and destroy at once, and the memory goes back to
the device with the last handle."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu
EXT = (8, 6, 4, 10)


def bundle(U, prec):
    G = lt.GaugeField(EXT, prec)
    G.upload(U)
    return [d["Plaquette"] for d in lt.Observables(G, 6.0, 2, 2, 0.02)], G.download()


def test_reuse_and_threads():
    U = haar_links_numpy(EXT, 1)
    keep = lt.GaugeField(EXT)   # a live handle: destroyed handles' buffers stay in the store
    want = {p: bundle(U, p) for p in ("fp64", "fp32_12")}
    bad = []

    def work(prec):
        for _ in range(5):
            p, links = bundle(U, prec)
            if p != want[prec][0] or not np.array_equal(links, want[prec][1]):
                bad.append(prec)

    threads = [threading.Thread(target=work, args=(p,)) for p in ("fp64", "fp32_12", "fp64", "fp32_12")]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    keep.close()


def test_given_back_with_the_last_handle():
    """In a process of its own: a field of 110 MB stays in the store while another handle lives and goes
    back to the device with the last one."""
    code = """
import torch, lettuce_b200 as lt
free = lambda: torch.cuda.mem_get_info()[0] >> 20
small = lt.GaugeField((4, 4, 4, 4))
start = free()
big = lt.GaugeField((24, 24, 24, 14))
assert free() < start - 100
big.close()
assert free() < start - 100
small.close()
assert free() > start - 16
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
