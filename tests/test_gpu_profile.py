"""Per-kernel profiling times each launch alone: while it is on, no two launches
of a call share the GPU, also where a call runs kernels side by side."""
import numpy as np
import pytest

import sbclip
import sbclip_gen as gen

pytestmark = pytest.mark.gpu


def alone(call):
    call()  # buffers and streams
    sbclip.profile_begin()
    call()
    prof = sbclip.profile_end()
    tl = sorted(sbclip.profile_timeline(), key=lambda x: x[1])
    assert len(tl) == sum(n for _, n in prof.values())
    for (a, s, d, _), (b, t, _, _) in zip(tl, tl[1:]):
        assert t >= s + d - 2e-3, (a, b)  # (event times are in steps of half a microsecond)
    return prof


def test_wide_and_small_pairs(clipper):
    pairs = gen.small_pairs(500, seed=9, lo=4, hi=64) + gen.small_pairs(40, seed=10, lo=300, hi=700)
    bases, ovs = [p[0] for p in pairs], [p[1] for p in pairs]
    prof = alone(lambda: clipper.area_backward(bases, ovs, np.ones(len(bases))))
    assert {"k_batch_clean", "k_batch_clean_wide", "k_batch_backward", "k_batch_backward_wide"} <= set(prof)


def test_overlays_of_every_size():
    base = gen.star(4000, 3, R=100.0)
    ovs = [gen.star(n, 50 + i, centre=(10.0 + i, 3.0), R=90.0) for i, n in enumerate((8, 40, 90, 400, 500, 1500, 3000, 3100))]
    ovs += [gen.star(9, 80 + i, centre=(50.0 + i, 3.0), R=4.0) for i in range(4)]
    touch = [o.copy() for o in ovs]
    for i, o in enumerate(touch):
        o[1] = (base[10 * i] + base[10 * i + 1]) / 2
    cl = sbclip.Clipper(0)
    try:
        cl.set_pairwise_workers(1)
        cl.set_pairwise_split(20000)
        prof = alone(lambda: cl.clip_pairwise(base, ovs + touch))
        assert cl.pairwise_info()["big_pairs"] > 0
        assert {"k_pw_clean", "k_pw_clean_wide", "k_pw_clean_huge", "k_pw_pairs", "k_pw_pairs_wide"} <= set(prof)
    finally:
        cl.close()
