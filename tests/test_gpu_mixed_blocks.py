"""Small pairs of every sort side by side, four to a block of the
general-position kernel: its warps leave at different steps, or have no pair at
all.  Every pair as the oracle has it, in every mixture."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu

SQ = np.array([[0.0, 0.1], [4.0, 0.0], [4.1, 4.0], [0.2, 4.2]])


def zigzag(n, a):
    """n long teeth side by side, turned by a."""
    y = np.linspace(-5.0, 5.0, n) + 0.01 * np.sin(np.arange(n))
    p = np.stack([np.where(np.arange(n) % 2, 9.0, -9.0) + 0.1 * np.cos(np.arange(n)), y], 1)
    p = np.concatenate([p, [[12.0, 7.1], [13.0, -8.0]]])
    return p @ np.array([[np.cos(a), np.sin(a)], [-np.sin(a), np.cos(a)]])


def sorts():
    star = lambda n, s, **k: gen.star(n, s, R=10.0, **k)
    flat = np.insert(star(20, 9), 4, (star(20, 9)[3] + star(20, 9)[4]) / 2, axis=0)
    touch = star(20, 3, centre=(2.0, 1.0))
    touch[5] = (star(24, 1)[2] + star(24, 1)[3]) / 2
    return [
        (star(24, 1), star(18, 2, centre=(2.0, 1.0))),          # crossings
        (zigzag(20, 0.1), zigzag(21, 1.5)),                     # more than the first pass has room for
        (star(24, 1), star(18, 2, centre=(90.0, 1.0))),         # none
        (star(24, 1), 0.01 * star(18, 2)),                      # one inside the other
        (star(24, 1), touch),                                   # a vertex on an edge
        (SQ, np.array([[4.0, 0.0], [7.0, 1.3], [5.0, 3.7]])),   # a shared vertex (and x value)
        (np.round(SQ), SQ + [1.7, 2.3]),                        # a shared x value
        (SQ, np.array([[1.0, 0.075], [3.0, 0.025], [3.3, 2.0], [1.2, 2.1]])),  # edges that overlap
        (flat, star(18, 2, centre=(2.0, 1.0))),                 # a vertex in line
        (SQ[:2], SQ),                                           # too few vertices
        (star(200, 6), star(90, 7, centre=(2.0, 1.0))),         # wide
    ]


@pytest.mark.parametrize("union", [False, True], ids=["intersection", "union"])
@pytest.mark.parametrize("seed", range(4))
def test_every_mixture(union, seed):
    pairs, ref = sorts(), []
    for b, c in pairs:
        try:
            ref.append(oracle_py.rings_of(oracle_py.clip(b, [c], union=union)["overlays"][0]))
        except oracle_py.OracleError:
            ref.append(None)
    assert sum(r is None for r in ref) <= 3
    rng = np.random.default_rng(seed)
    pick = rng.integers(0, len(pairs), 601 + seed)  # the last block is not full
    pick[:44] = np.repeat(np.arange(11), 4)         # blocks of one sort
    cl = sbclip.Clipper(0, union=union)
    try:
        rings, status = cl.clip_batch([pairs[i][0] for i in pick], [pairs[i][1] for i in pick])
    finally:
        cl.close()
    for i, got, st in zip(pick, rings, status):
        assert (st == 0) == (ref[i] is not None)
        assert ref[i] is None or rings_equal(got, ref[i]), i
