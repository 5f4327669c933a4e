"""Pairs whose rows A9-A18 run on a block instead of a warp: rings equal to the
oracle's, bit for bit, for plain crossings (the block's own labelling and
tracing) and for touching and overlapping edges (its first warp's serial
steps), in both modes and on either side of the size rule."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu


def comb(teeth, y0, y1, x0, up, flat):
    """A comb along x: a bar and `teeth` slanted teeth with flat tips at y1
    (or at flat[i] of the way).  No vertical edge."""
    s = 1.0 if up else -1.0
    v = []
    for i in range(teeth):
        tip = y0 + (y1 - y0) * flat[i % len(flat)]
        v += [(x0 + i, y0), (x0 + i + 0.13, tip), (x0 + i + 0.57, tip), (x0 + i + 0.71, y0)]
    bar = [(x0 + teeth + 0.31, y0 - s * 1.0), (x0 - 0.83, y0 - s * 1.0)]
    p = np.array(v + bar)
    return p if not up else p[::-1].copy()


def want(base, ov, union):
    return oracle_py.rings_of(oracle_py.clip(base, [ov], union=union)["overlays"][0])


@pytest.fixture(scope="module", params=[False, True], ids=["intersection", "union"])
def mode(request):
    c = sbclip.Clipper(0, union=request.param)
    yield c, request.param
    c.close()


def test_plain_crossings(mode):
    """Records on both sides of the block's line (512) and up to 20,000, an
    overlay that starts inside the base and one that starts outside, one of
    either orientation, a whole base inside an overlay."""
    cl, union = mode
    base = gen.star(2500, 71, R=100.0)
    ovs = [gen.star(n, 900 + n, centre=(x, 7.0), R=r)
           for n, x, r in ((3, 0.0, 90.0), (64, 20.0, 40.0), (127, 30.0, 60.0), (300, 10.0, 80.0),
                           (301, -35.0, 95.0), (1200, 25.0, 100.0), (2400, 3.0, 100.0),
                           (700, 0.0, 30.0), (40, 0.0, 1000.0), (50, 900.0, 20.0))]
    ovs.append(ovs[5][::-1].copy())
    rings, status = cl.clip_pairwise(base, ovs)
    assert (status == 0).all()
    for got, o in zip(rings, ovs):
        assert rings_equal(got, want(base, o, union))
    assert cl.pairwise_info()["big_pairs"] == 0


def test_overlaps_and_touches(mode):
    """Flat tips of the two combs meet along edges (delayed crossings and
    bounces): the block leaves these pairs' serial steps to one warp."""
    cl, union = mode
    base = comb(420, 0.0, 1.0, 0.0, True, [1.0, 0.7, 1.0, 1.0])
    ovs = [comb(n, 2.0, 1.0, x, False, f)
           for n, x, f in ((400, 0.2937, [1.0, 1.4]), (300, 40.4143, [1.0, 1.3, 1.0]),
                           (410, 3.6189, [1.5, 1.2, 1.45]), (8, 5.2711, [1.0]))]
    rings, status = cl.clip_pairwise(base, ovs)
    for got, o, st in zip(rings, ovs, status):
        try:
            ref = want(base, o, union)
        except oracle_py.OracleError:
            assert st != 0
            continue
        assert st == 0 and rings_equal(got, ref)
