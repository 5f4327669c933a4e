"""The batch autotuner times a setting only where it changes a launch: the
thread back end's block size where pairs of the batch were left to the lists."""
import numpy as np
import pytest

import sbclip
import sbclip_gen as gen

pytestmark = pytest.mark.gpu


def settings(pairs):
    """How many settings one tuning timed (twice each, forward and backward)."""
    torch = pytest.importorskip("torch")
    cl = sbclip.Clipper(0)
    try:
        bxy, boff = sbclip.pack_polygons([b for b, _ in pairs])
        cxy, coff = sbclip.pack_polygons([c for _, c in pairs])
        t = [torch.from_numpy(x).cuda() for x in (bxy, boff, cxy, coff, np.ones(len(pairs)))]
        g = [torch.zeros_like(t[0]), torch.zeros_like(t[2]), torch.zeros_like(t[4])]
        batch = (len(pairs), *(x.data_ptr() for x in t[:4]))
        grads = (t[4].data_ptr(), g[0].data_ptr(), g[1].data_ptr())
        # a block size that is not among those tried: each knob tries three
        cl.set_batch_shape(front=96, cand=96, back=96, backward=96)

        def launches(f):
            n0 = sbclip.kernel_launches()
            f()
            return sbclip.kernel_launches() - n0
        forward = launches(lambda: cl.area_forward_device(*batch, g[2].data_ptr()))
        backward = launches(lambda: cl.area_backward_device(*batch, *grads))
        tuned = launches(lambda: cl.autotune_batch_device(*batch, *grads))
        n = (tuned - forward) / (2 * (forward + backward))
        assert n == int(n)
        return int(n), cl.batch_shape()["back"]
    finally:
        cl.close()


def test_back_end_only_where_it_runs():
    pairs = gen.small_pairs(300, seed=77)
    assert settings(pairs) == (1 + 3 * 3, 96)
    b, c = pairs[0][0], pairs[0][1].copy()
    c[1] = (b[0] + b[1]) / 2
    assert settings(pairs + [(b, c)])[0] == 1 + 3 * 4
