"""The extrema pass, which forms the DoG values from Gaussian planes: keypoints equal to the
CPU restatement's at the widths where spans, warps per row and mask words end."""
import numpy as np
import pytest

import oracle as O
import psift

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
