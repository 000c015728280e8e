"""The split sub-sweeps of small lattices (six warps to 32 links) against the batched kernels, which give
one thread to a link: the same products and sums in the same order, so the same bits.  Lattices with partly
empty blocks (8, 240 links a sub-sweep), one block per SM and several, and the first size past the rule."""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("ext", [(2, 2, 2, 2), (4, 6, 2, 10), (8, 8, 8, 8), (12, 12, 12, 12), (14, 12, 14, 14)])
def test_same_bits_as_one_thread_a_link(ext, prec):
    U = haar_links_numpy(ext, 6)
    A, B = lt.GaugeField(ext, prec), lt.GaugeField(ext, prec)
    A.upload(U)
    B.upload(U)
    lt.UpdateSweeps(A, 6.0, 2, 1, 2, seed=5)
    lt.Ensemble([B], [6.0], seed=5).sweeps(2, 1, 2)
    assert np.array_equal(A.download(), B.download())
