"""Two crossings at one FP64 point: a needle of the base whose sides cross one
overlay edge a few millionths below the tip, at coordinates of some 10^5.  The
gradient of such a ring vertex goes to the edges of the first record that has
its coordinates, as the provenance by coordinates has it."""
import numpy as np
import pytest

import area_grad
import oracle_py
import sbclip
from conftest import rings_equal

pytestmark = pytest.mark.gpu


def needle_pair(seed):
    """Base edges 31 and 32 are the needle's sides; edges 0 to 30 cross the
    overlay many times, edges 33 on lie apart from it."""
    rng = np.random.default_rng(seed)
    k, m, t = np.arange(31), np.arange(13), np.arange(30)
    teeth = np.stack([3.0 * k + rng.uniform(0, 1, 31), np.where(k % 2 == 0, -60.0, 70.0) + rng.uniform(0, 3, 31)], 1)
    d = rng.uniform(1e-6, 4e-6)
    tip = np.array([120.0 + rng.uniform(0, 1), 50.0 + d])
    foot = tip + [rng.uniform(-3, 3), -110.0]
    apart = np.stack([200.0 + 10 * np.cos(-2.0 + 0.1 * t), -150.0 + 10 * np.sin(-2.0 + 0.1 * t)], 1)
    base = np.concatenate([teeth, [foot, tip, foot + [1e-4, 0.3]], apart, [[20.0, -300.0]]])
    low = np.stack([-15.0 + 11.0 * m, np.where(m % 2 == 0, -40.0, 30.0) + rng.uniform(0, 2, 13)], 1)
    over = np.concatenate([[[150.0, 50.0], [100.0, 50.0], [-20.0, 51.0]], low, [[145.0, -42.0]]])
    off = np.array([4e5, 3e5]) + rng.uniform(0, 10, 2)
    return base + off, over + off


SEEDS = (10, 35, 45, 63, 112, 118, 123, 136)


def pairs():
    for s in SEEDS:
        b, c = needle_pair(s)
        for shift in (0, 5, -32):  # the sides in two groups of 32 edges, in one, and at the ring's ends
            yield np.roll(b, shift, axis=0), c


def check(got, p, b, c, o, ga):
    _, rb, rc = area_grad.gradient_of_rings(b, c, oracle_py.rings_of(o), o["uniq_b"], o["uniq_c"], o["uniq_t"],
                                            o["isect_xy"])
    top = ga * max(np.abs(rb).max(), np.abs(rc).max())
    # FP64 on both sides from the same rings; edges that cross do so at 0.1 rad
    # and more, so the chain rule loses a digit, and some hundred terms add up
    assert np.abs(got[0] - ga * rb).max() <= 1e-11 * top, p
    assert np.abs(got[1] - ga * rc).max() <= 1e-11 * top, p


def test_gradient_of_the_pair_pipeline(clipper):
    """The pairs above the batch's split."""
    cases = list(pairs())
    ref = [oracle_py.clip(b, [c])["overlays"][0] for b, c in cases]
    for o in ref:
        xy = np.asarray(o["isect_xy"]).reshape(-1, 2)
        assert len(np.unique(xy, axis=0)) == len(xy) - 1
    ga = np.linspace(0.5, 2.0, len(cases))
    keep = clipper.batch_shape()["split"]
    clipper.set_batch_shape(split=3)
    try:
        for _ in range(5):
            rings, status = clipper.clip_batch([b for b, _ in cases], [c for _, c in cases])
            gb, gc = clipper.area_backward([b for b, _ in cases], [c for _, c in cases], ga)
            assert clipper.batch_info()["large_pairs"] == len(cases)
            for p, ((b, c), o) in enumerate(zip(cases, ref)):
                assert status[p] == 0 and rings_equal(rings[p], oracle_py.rings_of(o))
                check((gb[p], gc[p]), p, b, c, o, ga[p])
    finally:
        clipper.set_batch_shape(split=keep)


def test_gradient_of_the_batch_engine(clipper):
    cases = list(pairs())
    ref = [oracle_py.clip(b, [c])["overlays"][0] for b, c in cases]
    ga = np.linspace(0.5, 2.0, len(cases))
    gb, gc = clipper.area_backward([b for b, _ in cases], [c for _, c in cases], ga)
    for p, ((b, c), o) in enumerate(zip(cases, ref)):
        check((gb[p], gc[p]), p, b, c, o, ga[p])
