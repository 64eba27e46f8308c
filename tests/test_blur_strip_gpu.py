"""The strip level blur: planes equal to the tile kernels' at the sizes where strips,
segments, chunks and work lists end."""
import numpy as np
import pytest

import oracle as O
import psift
import synth

pytestmark = pytest.mark.gpu


def _tiles(ctx):
    for r in range(1, 16):
        ctx.set_tuning(ctx.TUNE_BLUR, r, 1)
    return ctx


# octave 0 of at least 6 Mpx takes the strips; widths end a strip at 1, 2, 63, 64 and 65
# columns, heights leave a last segment of one row and of a few
@pytest.mark.parametrize("h,w,up,scales", [(1203, 1313, True, 3), (1600, 961, True, 3), (2501, 2625, False, 3),
                                           (2449, 2623, False, 5), (1127, 1409, True, 10)])
@pytest.mark.parametrize("fused", [False, True])
def test_strip_planes_equal_tile_planes(h, w, up, scales, fused):
    img = O.luma_to_f32(synth.blob_image(w, h, 200, 1.5, 12.0, seed=h + w))
    cfg = psift.SiftConfig().with_octaves(2).with_scales(scales).upsample_first_octave(up)
    a, b = psift.Context(0), _tiles(psift.Context(0))
    if fused:  # the single-rounding mode has one tile shape; compare against the reference rounding loosely
        a.set_blur_rounding(a.BLUR_FUSED)
    for (g0, d0), (g1, d1) in zip(psift.build_pyramid(img, cfg, ctx=a), psift.build_pyramid(img, cfg, ctx=b)):
        if fused:
            # each tap's rounding differs by at most half an ulp of a value below 1: (2R + 1) * 2^-24 per pass,
            # two passes, at most scales + 2 levels after the base, on sums below 1
            np.testing.assert_allclose(g0, g1, rtol=0, atol=2 * 21 * 2.0 ** -24 * (scales + 3))
        else:
            np.testing.assert_array_equal(g0, g1)
            np.testing.assert_array_equal(d0, d1)
        np.testing.assert_array_equal(d0, g0[1:] - g0[:-1])
    a.close()
    b.close()


def test_strip_batch_beyond_the_work_list_equals_single_calls():
    # 70 images (the work list holds 64), 0.11 Mpx each at octave 0: strips for the batch, tiles for one
    imgs = [synth.blob_image(170 + (i % 3), 160 + (i % 2), 30, 1.5, 8.0, seed=900 + i) for i in range(70)]
    sift = psift.Sift.new(psift.SiftConfig().with_octaves(3))
    ctx = psift.Context(0)
    got = sift.detect_and_compute_batch_u8(imgs, ctx=ctx)
    for im, g in zip(imgs, got):
        one = sift.detect_and_compute_u8(im, ctx=ctx)
        assert len(g) == len(one)
        for k in ("x", "y", "scale", "response", "orientation", "descriptors"):
            np.testing.assert_array_equal(getattr(g, k), getattr(one, k), err_msg=k)
    ctx.close()
