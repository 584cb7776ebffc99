"""The FP64 path's FMM (digit-product translations on the tensor cores, double-single near field
and P2M) against the same tree on the FP64 pipe, at the edges of its launches: a single tile and
tiles that end inside a level or an octant, one level (no M2M or L2L), deep flat and long trees,
leaves with few and many nodes, one and two charge sets, uneven forests."""
import numpy as np
import pytest

import feellgood_gb300 as fg
from oracle import fgo
from tests import cases

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# (1, 1, 1): 8 nodes; (3, 3, 3) at depth 2: one octant per leaf; (8, 8, 8) at depth 3: 64 leaves of
# each octant, not a multiple of a 48-cell tile; plates and bars at depths whose leaves are partly
# empty; a shallow tree with hundreds of nodes per leaf
@pytest.mark.parametrize("shape,leaf", [((1, 1, 1), -2), ((3, 3, 3), -2), ((8, 8, 8), -3), ((30, 26, 1), -5),
                                        ((2, 3, 60), -6), ((15, 14, 13), -2), ((11, 7, 5), -4)])
def test_fp64_fmm_edges(shape, leaf):
    m = cases.cuboid(*shape)
    u = cases.perturbed_state(m["xyz"], seed=21, sigma=0.3)
    v = cases.tangent_field(u, seed=22)
    H = np.zeros(3)
    pot = []
    for native in (0, 1):
        c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=leaf, fmm_native_fp64=native)
        c.set_state(u, v)
        c.compute_all(H)
        s = c.get_state(0)
        pot.append((s["phi"], s["phiv"], c.demag(0), c.demag(1)))
    # digits carry 2^-46 of the largest coefficient, double-single sums about 2^-46 of the summed
    # magnitudes, which cancel by up to two orders of magnitude for a random tangent field
    for k in range(4):
        assert _rel(pot[0][k], pot[1][k]) < (2e-13 if k % 2 == 0 else 1e-12)
    # two sets in one evaluation follow the arithmetic of one
    assert _rel(pot[0][0], pot[0][2]) < 1e-14 and _rel(pot[0][1], pot[0][3]) < 1e-14


# the FP64 tree of the FP32 + refinement path: one level; tiles of 32 cells that are full, ragged or
# one cell; near-field tasks of 1 to 8 targets; 64 leaves of each octant; few blocks of P2M
@pytest.mark.parametrize("shape,leaf", [((1, 1, 1), -2), ((3, 3, 3), -2), ((8, 8, 8), -3), ((30, 26, 1), -5),
                                        ((2, 3, 60), -6), ((15, 14, 13), -2), ((11, 7, 5), -4)])
@pytest.mark.parametrize("overlap", [0, 1])
def test_refinement_fp64_tree_edges(shape, leaf, overlap):
    m = cases.cuboid(*shape)
    u = cases.perturbed_state(m["xyz"], seed=23, sigma=0.3)
    v = cases.tangent_field(u, seed=24)
    pot = []
    for o in (dict(precision=fg.FG_PREC_FP32_REFINE, fmm_overlap=overlap), dict(fmm_native_fp64=1)):
        c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=leaf, **o)
        c.set_state(u, v)
        c.compute_all(np.zeros(3))
        s = c.get_state(0)
        pot.append((s["phi"], s["phiv"]))
    # 1/r to 1e-13 and sums to 2^-44 of the summed magnitudes, which cancel by up to one order of
    # magnitude for the magnetisation and two for a random tangent field
    assert _rel(pot[0][0], pot[1][0]) < 1e-12 and _rel(pot[0][1], pot[1][1]) < 1e-11


def test_fp64_forest_matches_single_trees():
    meshes = [cases.cuboid(*s) for s in ((9, 9, 9), (4, 6, 5), (12, 3, 2), (2, 2, 2))]
    us = [cases.perturbed_state(m["xyz"], seed=30 + k, sigma=0.3) for k, m in enumerate(meshes)]
    b = fg.Context(meshes, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=-3)
    b.set_state(np.concatenate(us))
    pb = b.demag(0)
    for k, m in enumerate(meshes):
        c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=-3)
        c.set_state(us[k])
        assert _rel(pb[b.node_offsets[k]:b.node_offsets[k + 1]], c.demag(0)) < 1e-13


# uneven leaves: the tasks of the large samples' leaves are cut down to a single pair of targets
@pytest.mark.parametrize("shapes,leaf", [([(12, 12, 12), (2, 2, 2)], -2), ([(16, 3, 2), (1, 1, 1), (5, 5, 5)], -3)])
def test_refinement_forest_of_uneven_leaves(shapes, leaf):
    meshes = [cases.cuboid(*s) for s in shapes]
    us = [cases.perturbed_state(m["xyz"], seed=50 + k, sigma=0.3) for k, m in enumerate(meshes)]
    phi = {}
    for p in (fg.FG_PREC_FP32_REFINE, fg.FG_PREC_FP64):
        c = fg.Context(meshes, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=leaf, precision=p)
        c.set_state(np.concatenate(us))
        phi[p] = c.demag(0)
        o = c.node_offsets
    # FP32 products and sums of some thousand terms that cancel by one to two orders of magnitude
    for k in range(len(meshes)):
        a, b = (x[o[k]:o[k + 1]] for x in (phi[fg.FG_PREC_FP32_REFINE], phi[fg.FG_PREC_FP64]))
        assert _rel(a, b) < 2e-5


def test_not_a_number_propagates():
    """A magnetisation that is not a number reaches every potential that depends on it."""
    m = cases.cuboid(6, 6, 6)
    u = cases.perturbed_state(m["xyz"], seed=40)
    u[5] = np.nan
    c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=-3)
    c.set_state(u)
    assert np.isnan(c.demag(0)).all()


# a coarse mesh at a large depth: interior nodes with no Gauss point in the leaves around them, whose
# near field is zero
@pytest.mark.parametrize("shape,leaf", [((2, 2, 2), -6), ((4, 3, 2), -7)])
@pytest.mark.parametrize("first_order", [0, 1])
def test_fp64_fmm_targets_without_near_sources(shape, leaf, first_order):
    m = cases.cuboid(*shape)
    u = cases.perturbed_state(m["xyz"], seed=25, sigma=0.3)
    v = cases.tangent_field(u, seed=26)
    pot = []
    for native in (0, 1):
        c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=leaf, fmm_native_fp64=native,
                       first_order=first_order)
        c.set_state(u, v)
        c.compute_all(np.zeros(3))
        s = c.get_state(0)
        pot.append((s["phi"], s["phiv"], c.demag(0), c.demag(1)))
    # as test_fp64_fmm_edges
    for k in (0, 2, 3) if first_order else range(4):
        assert _rel(pot[0][k], pot[1][k]) < (2e-13 if k % 2 == 0 else 1e-12)


# every form of the near field and P2M, and those that a tree cannot have. At depth 2 a leaf of
# (15, 14, 13) has more than 6,144 elements around it: no blocks. Of a bar of 520 cells it has 5,500, but
# 1,048 of its own (five Gauss points), more than the 1,024 of a P2M block, or 653 (one) on 525 nodes,
# whose columns take two tiles, as those of 506 cells do with five
@pytest.mark.parametrize("shape,leaf,one_point,auto", [
    ((3, 3, 3), -2, 0, 3), ((3, 3, 3), -2, 1, 3), ((11, 7, 5), -3, 0, 3), ((11, 7, 5), -3, 1, 3),
    ((15, 14, 13), -2, 0, 1), ((15, 14, 13), -2, 1, 1), ((1, 1, 520), -2, 0, 2), ((1, 1, 520), -2, 1, 3),
    ((1, 1, 506), -2, 0, 3)])
def test_demag_blocks_forms(shape, leaf, one_point, auto):
    m = cases.cuboid(*shape)
    u = cases.perturbed_state(m["xyz"], seed=27, sigma=0.3)
    v = cases.tangent_field(u, seed=28)

    def potentials(**o):
        c = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=leaf, one_gauss_point=one_point, **o)
        c.set_state(u, v)
        c.compute_all(np.zeros(3))
        s = c.get_state(0)
        return c.demag_info(), (s["phi"], s["phiv"], c.demag(0), c.demag(1))

    (form, _), ref = potentials(fmm_native_fp64=1)
    assert form == 0
    (form, n0), default = potentials()
    assert form == auto and (n0 > 0) == (form > 1)
    for blocks in (1, 2, 3):
        if blocks > auto:
            with pytest.raises(fg.FgError) as e:
                potentials(demag_blocks=blocks)
            assert "too many elements" in str(e.value)
            continue
        (form, n), pot = potentials(demag_blocks=blocks)
        assert form == blocks and (n > 0) == (blocks > 1)
        if blocks == 1 and shape[2] > 500:
            continue  # the sums hold coordinates to 2^-45 of a leaf's width, here 130 cells
        for k in range(4):  # as test_fp64_fmm_edges
            assert _rel(pot[k], ref[k]) < (2e-13 if k % 2 == 0 else 1e-12)
            if blocks == auto:
                assert np.array_equal(pot[k], default[k])


@pytest.mark.parametrize("o", [dict(), dict(first_order=1), dict(precision=fg.FG_PREC_FP32_REFINE),
                               dict(fmm_native_fp64=1)])
def test_the_depth_search_leaves_the_tree_of_its_depth(o):
    """A tree kept from the search over depths gives the bits of one made for that depth alone, whichever
    of the candidates it was, and its stage times do not count the trials."""
    for shape in ((6, 5, 4), (14, 13, 12), (40, 36, 1)):
        m = cases.cuboid(*shape)
        u = cases.perturbed_state(m["xyz"], seed=29, sigma=0.3)
        v = cases.tangent_field(u, seed=30)
        a = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, profile=1, **o)
        assert np.all(np.array(a.fmm_timings()) == 0)
        b = fg.Context(m, cases.regions(), demag=fg.FG_DEMAG_FMM, fmm_leaf=-a.counters()[1], **o)
        for c in (a, b):
            c.set_state(u, v)
            c.compute_all(np.zeros(3))
        sa, sb = a.get_state(0), b.get_state(0)
        assert np.array_equal(sa["phi"], sb["phi"]) and np.array_equal(sa["phiv"], sb["phiv"])
        assert np.array_equal(a.demag(0), b.demag(0)) and np.array_equal(a.demag(1), b.demag(1))


# layers of two magnetisations, with charged triangles between them, beside or around one that is not
# magnetic: nodes, elements and regions that the blocks have to leave out
@pytest.mark.parametrize("Ms", [(cases.MS, 3e5, 0.0), (0.0, cases.MS, 0.0, 3e5)])
@pytest.mark.parametrize("one_point", [0, 1])
def test_blocks_of_several_regions(Ms, one_point):
    m = cases.layered_cuboid(7, 6, 9, Ms)
    reg = [cases.regions()[0]] + [dict(cases.regions()[1], Ms=x) for x in Ms]
    u = cases.perturbed_state(m["xyz"], seed=31, sigma=0.3)
    v = cases.tangent_field(u, seed=32)
    mag = np.unique(m["tets"][np.array((0.0,) + Ms)[m["tet_reg"]] > 0])
    o = fgo.Oracle(m, [fgo.make_region()] + [fgo.make_region(A=cases.AE, Ms=x, alpha=0.5) for x in Ms],
                   one_gauss_point=bool(one_point))
    o.set_state(u, v)
    exact = [o.demag(0)[mag], o.demag(1)[mag]]

    def potentials(**k):
        c = fg.Context(m, reg, one_gauss_point=one_point, **k)
        c.set_state(u, v)
        c.compute_all(np.zeros(3))
        s = c.get_state(0)
        return [s["phi"][mag], s["phiv"][mag]]

    # FP64 sums of at most 15,000 terms on either side (15,000 x 2^-53 = 2e-12 of the summed
    # magnitudes, an order of magnitude more for the cancelling sums of v)
    for blocks in (1, 3):
        p = potentials(demag=fg.FG_DEMAG_DIRECT, demag_blocks=blocks)
        assert _rel(p[0], exact[0]) < 1e-11 and _rel(p[1], exact[1]) < 3e-11
    ref = potentials(demag=fg.FG_DEMAG_FMM, fmm_leaf=-3, fmm_native_fp64=1)
    assert _rel(ref[0], exact[0]) < 1e-4 and _rel(ref[1], exact[1]) < 1e-3  # the expansions' truncation
    for blocks in (1, 2, 3):
        p = potentials(demag=fg.FG_DEMAG_FMM, fmm_leaf=-3, demag_blocks=blocks)
        assert _rel(p[0], ref[0]) < 2e-13 and _rel(p[1], ref[1]) < 1e-12  # as test_fp64_fmm_edges
