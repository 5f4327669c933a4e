"""Pairs that the shortcuts of the pair pipeline do not fit: two vertices with
one x value (the tree from the endpoint sort, at once), a hit that is no proper
crossing (the records, at once).  Rings as the oracle's, and no stage runs only
to be thrown away."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu


def kernels(cl, base, ovs):
    ref = oracle_py.clip(base, ovs)["overlays"]
    for _ in range(2):  # the first call grows buffers
        sbclip.profile_begin()
        got = cl.clip(base, ovs)
        prof = sbclip.profile_end()
        for g, r in zip(got, ref):
            assert rings_equal(g, oracle_py.rings_of(r))
    return {k: n for k, (_, n) in prof.items()}


def shared_x(p):
    p = p.copy()
    p[len(p) // 2, 0] = p[1, 0]
    return p


@pytest.mark.parametrize("n", [12, 300, 5000])
def test_shared_x(clipper, n):
    b, c = gen.star(n, 3, R=100.0), gen.star(n - 2, 4, centre=(20.0, 9.0), R=100.0)
    plain = kernels(clipper, b, [c])
    assert clipper.stats()["vertex_sort"] == 2 and plain["k_gp_hits"] == 1
    k = kernels(clipper, shared_x(b), [c])
    assert clipper.stats()["vertex_sort"] == 0
    # the endpoints are sorted once, the vertices' order is not expanded again,
    # and the group pairs of the search are listed once
    assert k["k_ele_keys"] == 1 and "k_ele_expand" not in k and k["k_direct_groups"] == 1
    assert k["k_gp_hits"] == 1


@pytest.mark.parametrize("n", [12, 300, 5000])
def test_improper_hit(clipper, n):
    b, c = gen.star(n, 3, R=100.0), gen.star(n - 2, 4, centre=(20.0, 9.0), R=100.0)
    for i, e in ((n // 3, n // 4), (n // 2, n // 5)):
        c[i] = (b[e] + b[e + 1]) / 2
    for base in (b, shared_x(b)):
        k = kernels(clipper, base, [c])
        assert "k_gp_hits" not in k and clipper.stats()["unique"] % 2 == 0


def test_overlays_of_one_tree(clipper):
    """Overlays with and without improper hits, with and without a shared x
    value in the tree."""
    b = gen.star(400, 31, R=50.0)
    ovs = [gen.star(n, 40 + n, centre=(x, 3.0), R=30.0) for n, x in ((20, 0.0), (300, 30.0), (90, 10.0))]
    ovs[1][7], ovs[1][90] = (b[17] + b[18]) / 2, (b[117] + b[118]) / 2
    for base in (b, shared_x(b)):
        for order in ((0, 1, 2), (1, 0, 2)):
            k = kernels(clipper, base, [ovs[i] for i in order])
            assert k["k_gp_hits"] == 2
            assert k.get("k_ele_keys", 0) == (0 if base is b else 1) and "k_ele_expand" not in k


def test_grid_search():
    """Above the direct search's size, against the tree from the endpoint sort."""
    b, c = gen.jagged_star(170_000, 5, R=1000.0), gen.jagged_star(150_000, 6, R=1000.0, centre=(250.0, 100.0), rotation=0.3)
    ref, cl = sbclip.Clipper(0, endpoint_sort=True), sbclip.Clipper(0)
    try:
        for base in (b, shared_x(b)):
            for _ in range(2):
                assert rings_equal(cl.clip_pair(base, c), ref.clip_pair(base, c))
                assert cl.stats()["vertex_sort"] == (2 if base is b else 0)
                assert cl.stats()["raw_hits"] == ref.stats()["raw_hits"]
    finally:
        ref.close()
        cl.close()
