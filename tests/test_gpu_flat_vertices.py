"""Result vertices whose |area3| is below the clean-up's epsilon in one order of
their neighbours and not in the other (foster/polyclip.h:767-787 takes the
ring's): a vertex close to one end of a long edge, at coordinates where the
rounding of an area is of the epsilon's size.  Rings as the oracle's."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu


def with_point(poly, edge, t):
    w = poly[(edge + 1) % len(poly)]
    return np.insert(poly, edge + 1, poly[edge] + t * (w - poly[edge]), axis=0)


def pairs(R, t, seeds):
    for s in seeds:
        x = with_point(gen.star(12, s, R=R), s % 12, t)
        yield x, gen.star(9, 1000 + s, centre=(0.25 * R, 0.1 * R), R=R)


@pytest.fixture(scope="module", params=[False, True], ids=["intersection", "union"])
def mode(request):
    c = sbclip.Clipper(0, union=request.param)
    yield c, request.param
    c.close()


def check(cl, union, b, c):
    try:
        ref = oracle_py.rings_of(oracle_py.clip(b, [c], union=union)["overlays"][0])
    except oracle_py.OracleError:
        with pytest.raises(sbclip.SbcError):
            cl.clip_pair(b, c)
        return 0
    assert rings_equal(cl.clip_pair(b, c), ref)
    return sum(len(r) for r in ref)


@pytest.mark.parametrize("R,t", [(1e4, 1e-3), (1e5, 1e-3), (1e5, 1 - 1e-3), (1e5, 1e-4), (1e6, 1e-2), (1e6, 0.5)])
def test_near_an_end_of_its_edge(mode, R, t):
    cl, union = mode
    for b, c in pairs(R, t, (47, 82, 97, 337, 395) + tuple(range(60))):
        check(cl, union, b, c)
        check(cl, union, c, b)
        check(cl, union, b[::-1].copy(), c)


def test_without_crossings(mode):
    """The whole polygon is the result."""
    cl, union = mode
    for b, _ in pairs(1e5, 1e-3, range(40)):
        far = gen.star(9, 5, centre=(9e5, 0.0), R=1e5) if union else gen.star(9, 5, R=9e5)
        check(cl, union, b, far)
        check(cl, union, far, b)


def test_large_pairs_of_a_batch(mode):
    """The pairs above the batch's split, which the pair pipeline clips."""
    cl, union = mode
    cases = list(pairs(1e5, 1e-3, (47, 82, 97, 337, 395)))
    split = cl.batch_shape()["split"]
    cl.set_batch_shape(split=3)
    try:
        rings, status = cl.clip_batch([b for b, _ in cases], [c for _, c in cases])
        assert cl.batch_info()["large_pairs"] == len(cases)
    finally:
        cl.set_batch_shape(split=split)
    for (b, c), got, st in zip(cases, rings, status):
        ref = oracle_py.rings_of(oracle_py.clip(b, [c], union=union)["overlays"][0])
        assert st == 0 and rings_equal(got, ref)
