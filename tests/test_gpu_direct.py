"""The exact direct sum of the demag potential at the edges of its launches: as a matrix over the
nodes (one and several blocks of rows, node counts at, below and above their multiples, one and
several shares of the columns, one and two fields, both Gauss rules) and, where the matrix would be
too large, as the sum over Gauss points."""
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


def test_direct_sum_over_gauss_points_where_the_matrix_does_not_fit():
    """45,000 nodes (a matrix of 48 GB): the potentials of a few nodes against their sums."""
    m = cases.cuboid(74, 74, 7)
    u = cases.perturbed_state(m["xyz"], seed=13, sigma=0.3)
    v = cases.tangent_field(u, seed=14)
    c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_DIRECT)
    c.set_state(u, v)
    c.compute_all(np.zeros(3))
    s = c.get_state(0)
    o = fgo.Oracle(m, cases.oracle_regions())
    o.set_state(u, v)
    pick = np.linspace(0, len(m["xyz"]) - 1, 12).astype(int)
    for which, got in ((0, s["phi"]), (1, s["phiv"])):
        pts, q, corr = o.charges(which)
        ref = np.array([((q / np.linalg.norm(pts - m["xyz"][i], axis=1)).sum() + corr[i]) / (4 * np.pi) for i in pick])
        # 1.4 million FP64 terms on either side, summed in shares of thousands
        assert np.linalg.norm(got[pick] - ref) < 1e-11 * np.linalg.norm(ref) * (1 if which == 0 else 10)


def test_demag_blocks_of_the_direct_sum():
    """The matrix and the sum over Gauss points by choice, and what a context reports."""
    m = cases.cuboid(5, 4, 4)
    u = cases.perturbed_state(m["xyz"], seed=15, sigma=0.3)
    v = cases.tangent_field(u, seed=16)
    o = fgo.Oracle(m, cases.oracle_regions())
    o.set_state(u, v)
    n = len(m["xyz"])
    for blocks, form in ((0, 3), (1, 1), (2, 3), (3, 3)):
        c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_DIRECT, demag_blocks=blocks)
        assert c.demag_info() == (form, 24 * n * n if form == 3 else 0)
        c.set_state(u, v)
        c.compute_all(np.zeros(3))
        s = c.get_state(0)
        # as test_direct_sum_edges
        assert np.linalg.norm(s["phi"] - o.demag(0)) < 4e-12 * np.linalg.norm(o.demag(0))
        assert np.linalg.norm(s["phiv"] - o.demag(1)) < 1e-11 * np.linalg.norm(o.demag(1))
    for blocks in (-1, 4):
        with pytest.raises(fg.FgError):
            fg.Context(m, cases.regions(), demag_blocks=blocks)


def test_launches_are_counted():
    """fg_counters: the kernels that each call launches (8 nodes: the matrix in one share)."""
    m = cases.cuboid(1, 1, 1)
    u = cases.perturbed_state(m["xyz"], seed=17)
    c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_DIRECT)

    def count(call):
        n = c.counters()[0]
        call()
        return c.counters()[0] - n

    assert count(lambda: c.set_state(u)) == 1                    # the copy to CURRENT
    assert count(lambda: c.energy(np.zeros(3))) == 1
    assert count(lambda: c.compute_all(np.zeros(3))) == 3        # demag, energies, evolution
    assert count(lambda: c.demag(0)) == 1


def test_a_matrix_that_does_not_fit_is_an_error_where_it_is_asked_for():
    """117,000 nodes: a matrix of 328 GB. Creation fails with its own status, and works without it."""
    m = fg.cuboid(16, 16, 400, 40.0, 40.0, 1000.0, 1e-9, cases.MS)
    with pytest.raises(fg.FgError) as e:
        fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_DIRECT, demag_blocks=3)
    assert e.value.status == 6 and "does not fit" in str(e.value)  # FG_ENOMEM
    assert fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_DIRECT).demag_info() == (1, 0)
