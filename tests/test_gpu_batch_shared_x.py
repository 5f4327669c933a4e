"""The batch engine's front on a warp where vertices share an x value, or only
its rounding to float: at the sizes where a lane takes another vertex more and
where the endpoint sort leaves shared memory.  Rings and statuses as the
oracle's, area to 1e-12 of the rings' absolute terms."""
import numpy as np
import pytest

import area_grad
import oracle_py
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu

KINDS = {
    "apart": lambda b, c: None,
    "one float": lambda b, c: b.__setitem__((-1, 0), b[0, 0] * (1 + 1e-13)),
    "one value": lambda b, c: b.__setitem__((-1, 0), b[0, 0]),
    "one value in both polygons": lambda b, c: c.__setitem__((1, 0), b[1, 0]),
    "three of one float, two of one value": lambda b, c: (b.__setitem__((-1, 0), b[0, 0]),
                                                          c.__setitem__((2, 0), b[0, 0] * (1 - 1e-13))),
    "zeros of either sign": lambda b, c: (b.__setitem__((0, 0), 0.0), c.__setitem__((0, 0), -0.0)),
    "a grid": lambda b, c: (b.__setitem__(slice(None), np.round(b * 4) / 4), c.__setitem__(slice(None), np.round(c * 4) / 4)),
}


@pytest.mark.parametrize("E", [7, 31, 32, 33, 64, 65, 96, 97, 128, 129, 200, 255, 256])
def test_front_on_a_warp(clipper, E):
    bases, ovs, ref = [], [], []
    for i, kind in enumerate(KINDS.values()):
        nb = max(4, E // 3 + i % 2) if E > 7 else 4
        # (the largest sizes stay below the block's line with a small polygon)
        nb = min(nb, 4096 // E) if E > 128 else nb
        b = gen.star(nb, 100 + E + i, R=20.0)
        c = gen.star(E - nb, 300 + E + i, centre=(3.1, 1.7), R=20.0)
        kind(b, c)
        try:
            r = oracle_py.rings_of(oracle_py.clip(b, [c])["overlays"][0])
        except oracle_py.OracleError:
            r = None
        bases.append(b), ovs.append(c), ref.append(r)
    rings, status = clipper.clip_batch(bases, ovs)
    area, st2 = clipper.area_forward(bases, ovs)
    assert sum(r is not None for r in ref) >= 5
    for p, r in enumerate(ref):
        assert (status[p] == 0) == (st2[p] == 0) == (r is not None), list(KINDS)[p]
        if r is not None:
            assert rings_equal(rings[p], r), list(KINDS)[p]
            scale = sum(float(np.abs(x).max() ** 2) * len(x) for x in r) + 1e-300
            assert abs(area[p] - area_grad.shoelace(r)) <= 1e-12 * scale
