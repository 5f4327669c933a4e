"""The pair pipeline's candidate search without the grid: every pair of edges
whose float boxes meet is found once, on either side of its groups of 32 edges
and of its queues of 32 pairs, for polygons whose groups lie apart and for ones
whose groups span much of the box; only edges that reach the other group's box
are tested."""
import numpy as np
import pytest

import oracle_py
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu


def float_boxes(p):
    """The edges' boxes, rounded outwards to float."""
    q = np.roll(p, -1, axis=0)
    lo, hi = np.minimum(p, q), np.maximum(p, q)
    flo, fhi = lo.astype(np.float32), hi.astype(np.float32)
    flo = np.where(flo > lo, np.nextafter(flo, np.float32(-np.inf)), flo)
    fhi = np.where(fhi < hi, np.nextafter(fhi, np.float32(np.inf)), fhi)
    return flo, fhi


def meeting(b, c):
    (bl, bh), (cl, ch) = float_boxes(b), float_boxes(c)
    return int(((bl[:, None] <= ch) & (bh[:, None] >= cl)).all(2).sum())


def spokes(n, shift, R=100.0):
    """Every second vertex near the centre: an edge group's box is a wedge's."""
    t = 2 * np.pi * (np.arange(n) + 0.37) / n
    r = np.where(np.arange(n) % 2, R, 0.05 * R)
    return np.stack([r * np.cos(t), r * np.sin(t)], 1) + shift


def check(clipper, b, c):
    ref = oracle_py.clip(b, [c])["overlays"][0]
    assert rings_equal(clipper.clip_pair(b, c), oracle_py.rings_of(ref))
    st = clipper.stats()
    assert st["grid_pairs"] == meeting(b, c)
    assert st["raw_hits"] == len(ref["raw_b"]) and st["unique"] == len(ref["uniq_b"])
    return st


@pytest.mark.parametrize("nb", [3, 31, 32, 33, 65])
@pytest.mark.parametrize("nc", [3, 32, 33, 64, 1025])
def test_every_pair_once(clipper, nb, nc):
    b = gen.star(nb, 10 + nb, R=100.0)
    check(clipper, b, gen.star(nc, 20 + nc, centre=(9.0, 4.0), R=100.0))
    check(clipper, b, gen.star(nc, 30 + nc, centre=(9.0, 4.0), R=8.0))
    check(clipper, gen.star(nc, 40 + nc, R=100.0), b + [300.0, 1.0])


@pytest.mark.parametrize("n", [64, 200, 900])
def test_wide_groups(clipper, n):
    check(clipper, spokes(n, [0.0, 0.0]), gen.star(n + 1, 5, centre=(45.0, 38.0), R=9.0))
    check(clipper, gen.star(n + 1, 6, centre=(45.0, 38.0), R=9.0), spokes(n, [0.0, 0.0]))
    check(clipper, spokes(n, [0.0, 0.0]), spokes(n, [0.31, 0.17], R=60.0))


def test_edges_out_of_reach_are_not_tested(clipper):
    """About 6,600 group pairs meet, of which 6.8 million edge pairs could be tested."""
    b, c = gen.star(10_000, 1, R=1000.0), gen.star(8_000, 2, centre=(250.0, 100.0), R=1000.0)
    clipper.clip_pair(b, c)
    assert clipper.stats()["work_units"] < 2_500_000
