"""The exact direct sum of the demag potential at the edges of its launch: node counts at, below
and above a block of 64, fewer sources than one share of the split, one and several blocks, one
and two charge sets, both Gauss rules."""
import numpy as np
import pytest

import feellgood_gb300 as fg
from oracle import fgo
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 2, 6), (1, 1, 15), (1, 2, 10), (5, 4, 4)])
@pytest.mark.parametrize("one_point", [False, True])
@pytest.mark.parametrize("first_order", [False, True])
def test_direct_sum_edges(shape, one_point, first_order):
    m = cases.cuboid(*shape)
    u = cases.perturbed_state(m["xyz"], seed=11, sigma=0.3)
    v = cases.tangent_field(u, seed=12)
    H = np.array([1e4, -2e4, 5e3])
    o = fgo.Oracle(m, cases.oracle_regions(), one_gauss_point=one_point)
    o.set_state(u, v)
    c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_DIRECT, one_gauss_point=int(one_point),
                   first_order=int(first_order))
    c.set_state(u, v)
    c.compute_all(H)
    s = c.get_state(0)
    # both sides add at most 4,000 FP64 terms: rounding below 4e3 * 2^-53 = 4e-13 of the summed
    # magnitudes, which cancel by less than an order of magnitude for m and by about one for v
    po, pv = o.demag(0), o.demag(1)
    assert np.linalg.norm(s["phi"] - po) < 4e-12 * np.linalg.norm(po)
    assert np.linalg.norm(c.demag(0) - po) < 4e-12 * np.linalg.norm(po)
    if not first_order:
        assert np.linalg.norm(s["phiv"] - pv) < 1e-11 * np.linalg.norm(pv)
