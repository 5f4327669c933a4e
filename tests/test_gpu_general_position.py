"""Pairs in general position through sbc_clip_pair (rings straight from the
hits) and pairs that are not: rings as the oracle's in both modes, and the
diagnostics as if the arrays had been built."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[False, True], ids=["intersection", "union"])
def mode(request):
    c = sbclip.Clipper(0, union=request.param)
    yield c, request.param
    c.close()


def zigzag(n, height, x0, x1):
    """A ring whose n teeth cross the x axis inside [x0, x1]."""
    x = np.linspace(x0, x1, 2 * n + 1) + np.linspace(0.0, 0.01, 2 * n + 1)
    y = np.where(np.arange(2 * n + 1) % 2 == 0, -height, height) * np.linspace(1.0, 1.3, 2 * n + 1)
    return np.concatenate([np.stack([x, y], 1), [[x1 + 3.0, 5 * height], [x0 - 2.0, 5.1 * height]]])[::-1].copy()


def pairs():
    spear = np.array([[-400.0, -0.31], [900.0, 0.11], [880.0, 0.9]])
    yield gen.star(24, 1), gen.star(18, 2, centre=(0.2, 0.1))
    yield gen.star(3, 3), gen.star(3, 4, centre=(0.1, 0.0))
    # crossings per edge on either side of 4, 32 and 128 (a lane, a warp, a
    # block), and more than the block takes
    for teeth in (2, 5, 16, 17, 63, 64, 65, 700, 2500):
        yield spear, zigzag(teeth, 1.7, -100.0, 120.0)
        yield zigzag(teeth, 1.7, -100.0, 120.0), spear
    # around 4,096 crossings (one block's pointer doubling, or the grid's)
    yield gen.star(1400, 5, R=100.0), gen.star(1300, 6, centre=(30.0, 10.0), R=100.0)
    yield gen.star(1700, 7, R=100.0), gen.star(1500, 8, centre=(20.0, 10.0), R=100.0)
    # nothing crosses: inside, around, apart; a vertex in line with its neighbours
    yield gen.star(300, 9, R=100.0), gen.star(200, 10, R=3.0)
    yield gen.star(300, 9, R=3.0), gen.star(200, 10, R=100.0)
    yield gen.star(300, 9, R=3.0), gen.star(200, 10, centre=(50.0, 0.0), R=3.0)
    yield np.array([[0.0, 0.1], [1.0, 0.1], [2.0, 0.1], [1.1, 3.0]]), gen.star(40, 11, centre=(1.0, 0.3), R=60.0)
    yield np.array([[0.0, 0.1], [1.0, 0.1], [2.0, 0.1], [1.1, 3.0]]), gen.star(40, 12, centre=(1.0, 1.3), R=0.7)
    # a vertex on an edge, overlapping edges
    yield np.array([[0.0, 0.0], [4.0, 0.0], [4.0, 4.0], [0.0, 4.0]]), np.array([[1.0, 4.0], [3.0, 4.0], [2.0, 9.0]])
    yield np.array([[0.0, 0.0], [4.0, 0.0], [4.0, 4.0], [0.0, 4.0]]), np.array([[2.0, 4.0], [7.0, 2.0], [2.0, -3.0]])


@pytest.mark.parametrize("i", range(len(list(pairs()))))
def test_rings(mode, i):
    cl, union = mode
    b, c = list(pairs())[i]
    for x, y in ((b, c), (b, c[::-1].copy())):
        try:
            ref = oracle_py.clip(x, [y], union=union)
        except oracle_py.OracleError:
            with pytest.raises(sbclip.SbcError):
                cl.clip_pair(x, y)
            continue
        assert rings_equal(cl.clip_pair(x, y), oracle_py.rings_of(ref["overlays"][0])), i


def test_diagnostics_after_the_rings(clipper):
    """The arrays of rows A9-A14 are the oracle's when asked for after the
    call, in any order, and asking leaves the result as it was."""
    b, c = gen.star(400, 21, R=10.0), gen.star(350, 22, centre=(2.0, 1.0), R=10.0)
    off, xy = clipper.clip_pair_flat(b, c, copy=False)
    before = (off.copy(), xy.copy())
    o = oracle_py.clip(b, [c])["overlays"][0]
    assert clipper.stats()["unique"] == len(o["uniq_b"])
    assert clipper.stats()["slots_b"] == len(o["merged_balpha"])
    assert clipper.stats()["slots_c"] == len(o["merged_calpha"])
    for name in ("label_b", "merged_cnb", "uniq_b", "isect_ab", "uniq_c", "merged_balpha"):
        assert np.array_equal(clipper.debug_array(name), o[name]), name
    assert np.array_equal(clipper.debug_array("isect_xy").reshape(-1), np.asarray(o["isect_xy"]).reshape(-1))
    assert np.array_equal(off, before[0]) and np.array_equal(xy, before[1])


def test_every_overlay_of_a_tree(clipper):
    b = gen.star(900, 31, R=50.0)
    ovs = [gen.star(n, 40 + n, centre=(x, 3.0), R=30.0) for n, x in ((20, 0.0), (300, 30.0), (5, -40.0), (90, 200.0))]
    ref = oracle_py.clip(b, ovs)["overlays"]
    for got, r in zip(clipper.clip(b, ovs), ref):
        assert rings_equal(got, oracle_py.rings_of(r))


@pytest.mark.parametrize("n", [1, 30, 64, 65, 66, 90])
def test_zero_border_keys(clipper, n):
    """n vertices within a border key of the least x value: their keys are
    zero, and the reference's never-written border slot comes after them.  Up
    to 64 the ranks follow it, above that the stages that build the arrays."""
    t = np.arange(n + 1)
    left = np.stack([-1.0 + 1e-12 * t, 1.0 - 2.0 * t / (n + 1)], 1)
    b = np.concatenate([left, [[-0.999, -1.01], [1.0, 0.0], [0.3, 1.1]]])
    c = gen.star(40, 90 + n, centre=(-0.9, 0.02), R=0.5)
    o = oracle_py.clip(b, [c])
    assert rings_equal(clipper.clip_pair(b, c), oracle_py.rings_of(o["overlays"][0]))
    assert np.array_equal(clipper.debug_array("elementary"), o["tree"]["ea"])
    st = clipper.stats()
    assert st["cover_entries"] == o["stats"]["cover_total"]
    assert st["leaf_end_entries"] == o["stats"]["leaf_end_total"]
    assert np.array_equal(clipper.debug_array("uniq_b"), o["overlays"][0]["uniq_b"])


def test_more_hits_than_the_first_guess(clipper):
    """Spiky stars whose edge groups and hits overflow the direct search's
    first buffers on a new context."""
    cl = sbclip.Clipper(0)
    try:
        b, c = gen.star(9000, 3, R=1000.0), gen.star(7000, 4, centre=(150.0, 90.0), R=1000.0)
        ref = oracle_py.rings_of(oracle_py.clip(b, [c])["overlays"][0])
        for _ in range(2):
            assert rings_equal(cl.clip_pair(b, c), ref)
    finally:
        cl.close()


@pytest.mark.parametrize("union", [False, True], ids=["intersection", "union"])
@pytest.mark.parametrize("n", [12, 300, 3000])
def test_result_vertices_in_line(n, union):
    """Vertices in line with their neighbours, which the clean-up removes: one
    on an edge, on every edge, two and three in a row, the first vertex, a ring
    that is a sliver; with crossings, without any, one tree over several
    overlays.  Rings as the oracle's."""
    from test_gpu_wide_pairs import with_points
    cl = sbclip.Clipper(0, union=union)
    try:
        b = gen.star(n, 1210 + n, R=50.0)
        pairs = []
        for k, (edges, where) in enumerate((((1,), (0.4,)), (range(n), (0.5,)), ((2, 7), (0.3, 0.8)),
                                            ((0, n - 1), (0.2, 0.5, 0.9)))):
            c = gen.star(n + 3 - k, 1300 + n + k, centre=(4.1 + k, -2.3), R=45.0)
            pairs += [(with_points(b, edges, where), c), (b, with_points(c, edges, where)),
                      (np.roll(with_points(b, edges, where), 2, axis=0), with_points(c, edges, where)),
                      (with_points(b, edges, where), c + [400.0, 0.0]),
                      (with_points(b, edges, where), (c - [4.1 + k, -2.3]) * 0.01 + [0.3, 0.2])]
        v, w = b[3], b[4]
        t = (w - v) / np.hypot(*(w - v))
        inward = np.array([-t[1], t[0]])
        tip = (v + w) / 2 + 2e-6 * inward
        pairs.append((b, np.array([tip, tip - inward * 30.0 + 0.1 * t, tip - inward * 29.0 - 0.2 * t])))
        for x, c in pairs:
            try:
                ref = oracle_py.rings_of(oracle_py.clip(x, [c], union=union)["overlays"][0])
            except oracle_py.OracleError:
                continue
            assert rings_equal(cl.clip_pair(x, c), ref)
        if not union:
            ovs = [c for _, c in pairs[:4]]
            got = cl.clip(pairs[0][0], ovs)
            for g, o in zip(got, oracle_py.clip(pairs[0][0], ovs)["overlays"]):
                assert rings_equal(g, oracle_py.rings_of(o))
    finally:
        cl.close()
