"""The strip level blur in batches, either rounding: every half of a batch (each runs as one
launch) has more images than the strips' work list holds (64) and at least 6 Mpx, or a few
large images; each image's features equal a single call's, whose blur runs tiles."""
import numpy as np
import pytest

import psift
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("n,w,h", [(140, 170, 160), (10, 640, 480)])
def test_strips_of_a_batch_equal_tiles_of_single_calls(n, w, h, fused):
    imgs = [synth.blob_image(w + (i % 3), h + (i % 2), 30, 1.5, 8.0, seed=700 + i) for i in range(n)]
    # octave 0 is twice the image's size
    assert (n // 2) * 4 * w * h >= 6_000_000 and 4 * (w + 2) * (h + 1) < 6_000_000
    sift = psift.Sift.new(psift.SiftConfig().with_octaves(2))
    ctx = psift.Context(0)
    if fused:
        ctx.set_blur_rounding(ctx.BLUR_FUSED)
    got = sift.detect_and_compute_batch_u8(imgs, ctx=ctx)
    for im, g in zip(imgs, got):
        one = sift.detect_and_compute_u8(im, ctx=ctx)
        assert len(g) == len(one)
        for k in ("x", "y", "scale", "response", "orientation", "descriptors"):
            np.testing.assert_array_equal(getattr(g, k), getattr(one, k), err_msg=k)
    ctx.close()
