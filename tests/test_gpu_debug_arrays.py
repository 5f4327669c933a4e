"""sbc_debug_array after a call with several overlays: the arrays are the last
overlay's, whichever route each overlay took (in general position: rings
straight from the hits; otherwise from the arrays), and a call that fails or is
refused leaves nothing of an earlier overlay to be read as its own."""
import numpy as np
import pytest

import oracle_py
import sbclip
import sbclip_gen as gen
from conftest import rings_equal

pytestmark = pytest.mark.gpu

NAMES = ("uniq_b", "uniq_c", "uniq_t", "isect_xy", "isect_ab", "isect_ac", "merged_bxy", "merged_cxy", "merged_balpha",
         "merged_calpha", "merged_bnb", "merged_cnb", "label_b", "label_c")

BASE = gen.star(300, 21, R=10.0)


def clean(n, seed):
    return gen.star(n, seed, centre=(2.0, 1.0), R=9.0)


def touching(n, seed):
    """A vertex on a base edge: not in general position."""
    c = clean(n, seed)
    c[n // 2] = (BASE[17] + BASE[18]) / 2
    return c


def apart(n, seed):
    return gen.star(n, seed, centre=(50.0, 3.0), R=2.0)


def check(cl, base, ovs):
    ref = oracle_py.clip(base, ovs)["overlays"]
    for got, r in zip(cl.clip(base, ovs), ref):
        assert rings_equal(got, oracle_py.rings_of(r))
    for name in NAMES:
        got, want = cl.debug_array(name), np.asarray(ref[-1][name])
        assert np.array_equal(got.reshape(-1), want.reshape(-1)), name


# small overlays before large ones make the second overlay's buffers grow
@pytest.mark.parametrize("kinds", [(clean, touching), (touching, clean), (clean, clean), (touching, touching),
                                   (clean, apart), (apart, touching), (clean, touching, clean), (touching, clean, touching)])
@pytest.mark.parametrize("sizes", [(20, 400, 60), (400, 20, 200)])
def test_last_overlay(kinds, sizes):
    cl = sbclip.Clipper(0)
    try:
        check(cl, BASE, [k(n, 40 + i) for i, (k, n) in enumerate(zip(kinds, sizes))])
    finally:
        cl.close()


def test_after_a_failure():
    """An overlay in general position, then one that the reference leaves
    undefined: the call fails, no records are left, and the context goes on."""
    sq = np.array([[0.0, 0.0], [4.0, 0.0], [4.0, 4.0], [0.0, 4.0]])
    good, bad = gen.star(30, 5, centre=(1.0, 2.0), R=3.0), np.array([[2.0, -1.0], [7.0, -1.0], [7.0, 4.0], [2.0, 4.0]])
    cl = sbclip.Clipper(0)
    try:
        with pytest.raises(oracle_py.OracleError):
            oracle_py.clip(sq, [good, bad])
        with pytest.raises(sbclip.SbcError):
            cl.clip(sq, [good, bad])
        for name in NAMES:
            cl.debug_array(name)
        check(cl, sq, [good])
    finally:
        cl.close()


def test_after_a_refused_call():
    torch = pytest.importorskip("torch")
    cl = sbclip.Clipper(0)
    try:
        check(cl, BASE, [clean(50, 3)])
        with pytest.raises(sbclip.SbcError):
            cl.clip(BASE[:2], [clean(50, 3)])
        tb, tc = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (BASE, clean(50, 3)))
        with pytest.raises(sbclip.SbcError):
            cl.clip_pair_device(tb.data_ptr(), 2, tc.data_ptr(), 50)
        ref = oracle_py.clip(BASE, [clean(50, 3)])["overlays"][0]
        for name in NAMES:
            assert np.array_equal(cl.debug_array(name).reshape(-1), np.asarray(ref[name]).reshape(-1)), name
    finally:
        cl.close()
