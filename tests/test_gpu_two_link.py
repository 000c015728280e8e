"""The rectangle force from the two-link fields (k_two_links, k_rect_outer) against the staples
multiplied out path by path (lt_staples), at the edges of its range: extents of 2 and 4, where
the two-step shifts wrap onto the site or meet each other, blocks with a remainder, the three storages.

Bound: a path of up to five links is four products of unit rows, each entry rounded by at most
6 eps (a sum of three complex products), plus the stored two-link product, 32 eps in all; the paths'
weights add up to 6 c_plaq + 18 |c_rect|; the product with U^dag multiplies by at most 3 and both
sides are rounded.
"""
import numpy as np
import pytest

import lettuce_b200 as lt
from ltref import haar_links_numpy

pytestmark = pytest.mark.gpu

EPS = {"fp64": 2.0 ** -53, "fp32": 2.0 ** -24, "fp32_12": 2.0 ** -24}


def algebra(m):
    m = 0.5 * (m - np.conj(np.swapaxes(m, -1, -2)))
    return m - np.trace(m, axis1=-2, axis2=-1)[..., None, None] / 3.0 * np.eye(3)


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp32_12"])
@pytest.mark.parametrize("ext", [(2, 2, 2, 2), (2, 4, 6, 2), (4, 4, 4, 4), (6, 2, 10, 6)])
@pytest.mark.parametrize("act", [lt.LuescherWeiszAction, lt.DBW2Action])
def test_force_matches_direct_paths(prec, ext, act):
    action = act(6.0)
    G = lt.GaugeField(ext, prec)
    G.upload(haar_links_numpy(ext, 3))
    cplx = lambda a: a[..., 0] + 1j * a[..., 1]  # noqa: E731
    U, S = cplx(G.download()), cplx(action.Staple(G))
    want = algebra(S @ np.conj(np.swapaxes(U, -1, -2)))
    got = cplx(action.Force(G))
    weight = 6.0 * action.c_plaq + 18.0 * abs(action.c_rect)
    assert np.abs(got - want).max() < 2.0 * 3.0 * 32.0 * EPS[prec] * weight
