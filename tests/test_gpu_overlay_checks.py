"""The one-base-many-overlays engine's conditions on an overlay, found by one
thread of its preparation wherever the vertex stands: an x value that is not
finite (refused), a vertical edge, an x value of the base (the pair pipeline)."""
import numpy as np
import pytest

import oracle_py
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu

ALL_ONES = np.array([0x7FFFFFFFFFFFFFFF], dtype=np.uint64).view(np.float64)[0]  # sorts after every value


@pytest.mark.parametrize("n", [3, 40, 257, 1000])
def test_one_vertex_decides(clipper, n):
    base = gen.star(300, 3, R=100.0)
    ovs, kinds = [], []
    for i in range(60):
        o = gen.star(n, 100 + i, centre=(5.0 + i, 3.0), R=20.0)
        v, kind = (i * 37) % n, i % 6
        if kind == 1:
            o[v, 0] = np.nan
        elif kind == 2:
            o[v, 0] = -np.inf
        elif kind == 3:
            o[v, 0] = o[(v + 1) % n, 0]
        elif kind == 4:
            o[v, 0] = base[i, 0]
        elif kind == 5:
            o[v, 0] = ALL_ONES
        ovs.append(o)
        kinds.append(kind)
    for _ in range(3):
        rings, status = clipper.clip_pairwise(base, ovs)
        for o, kind, got, st in zip(ovs, kinds, rings, status):
            if kind in (1, 2, 5):
                assert st == 1 and got == []
                continue
            try:
                ref = oracle_py.rings_of(oracle_py.clip(base, [o])["overlays"][0])
            except oracle_py.OracleError:
                assert st != 0
                continue
            assert st == 0 and rings_equal(got, ref)
