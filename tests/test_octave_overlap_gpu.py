"""An octave's last levels and extrema beside the next octave (small launches): the same
features as with every stage on one stream (stage timing)."""
import numpy as np
import pytest

import psift
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("octaves", [1, 2, 4])
@pytest.mark.parametrize("scales", [3, 5])
@pytest.mark.parametrize("w,h", [(160, 131), (517, 300)])
def test_features_equal_one_stream(octaves, scales, w, h):
    sift = psift.Sift.new(psift.SiftConfig().with_octaves(octaves).with_scales(scales))
    imgs = [synth.blob_image(w, h, 90, 1.5, 10.0, seed=40 + i) for i in range(2)]
    one, ctx = psift.Context(0), psift.Context(0)
    one.enable_stage_timing(True)
    for k in range(4):  # launched, captured and replayed, with changing images
        a = sift.detect_and_compute_u8(imgs[k % 2], ctx=one)
        b = sift.detect_and_compute_u8(imgs[k % 2], ctx=ctx)
        assert len(a) == len(b)
        for name in ("x", "y", "scale", "response", "orientation", "descriptors"):
            np.testing.assert_array_equal(getattr(a, name), getattr(b, name), err_msg=name)
    assert ctx.graph_replays == 3 and one.graph_replays == 0
    one.close()
    ctx.close()
