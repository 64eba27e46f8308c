"""The extrema pass, which forms the DoG values from Gaussian planes: keypoints equal to the
CPU restatement's at the widths where spans, warps per row and mask words end."""
import numpy as np
import pytest

import oracle as O
import psift
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(64, 127), (65, 129), (40, 386), (33, 769), (3, 200), (200, 3)])
@pytest.mark.parametrize("scales", [3, 4, 8, 9])
def test_extrema_at_span_edges(h, w, scales):
    rng = np.random.default_rng(h * 1000 + w + scales)
    img = rng.random((h, w), dtype=np.float32)
    ref = O.detect_keypoints(img, 2, scales, 0.004, False)
    cfg = psift.SiftConfig().with_octaves(2).with_scales(scales).with_contrast_threshold(0.004)
    got = psift.Sift.new(cfg.upsample_first_octave(False)).detect_keypoints(img)
    assert len(got) == len(ref)
    for f in ("x", "y", "response", "octave", "layer"):
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)


# rows (octave, slice, row) around one turn of the row scan (16,384) and around its 16 rows per thread
@pytest.mark.parametrize("h,octaves", [(2730, 1), (2731, 1), (2732, 1), (3100, 4), (131, 1), (133, 3)])
def test_keypoint_order_of_tall_images(h, octaves):
    f = O.luma_to_f32(synth.blob_image(41, h, 400, 1.5, 5.0, seed=h))
    ctx = psift.Context(0)
    got = psift.Sift.new(psift.SiftConfig().with_octaves(octaves)).detect_and_compute(f, ctx=ctx)
    meta, _ = O.detect_and_compute(f, octaves, 3, 0.015, True, 0, 4096)
    assert len(got) == meta.shape[0]
    np.testing.assert_array_equal(got.x, meta[:, 0])
    np.testing.assert_array_equal(got.y, meta[:, 1])
    ctx.close()
