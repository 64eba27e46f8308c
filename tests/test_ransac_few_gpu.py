"""RANSAC of match sets up to and just above the size that gets the small CTAs (32 matches, by
the largest set of a launch): equal to the CPU oracle, alone and beside larger sets."""
import numpy as np
import pytest

import oracle as O
import psift
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 2, 3, 4, 5, 6, 12, 31, 32, 33, 40])
@pytest.mark.parametrize("outliers", [0.0, 0.5])
def test_few_matches(n, outliers):
    h = synth.perspective_h(1920, 1080, 8, 1.05, 4e-5, -6e-5)
    m = synth.putative_matches(n, outliers, h, 1920, 1080, 300 + n)[0] if n else np.zeros(0, psift.MATCH_DTYPE)
    more = synth.putative_matches(50, 0.3, h, 1920, 1080, 9)[0]
    for homography, (mask, ref) in ((True, O.homography_ransac(m, 3.0, None)),
                                    (False, O.similarity_ransac(m, 3.0, O.DEFAULT_SIMILARITY_RANSAC_SEED))):
        alone = psift.ransac_batch([m], homography=homography)[0]
        beside = psift.ransac_batch([more, m], homography=homography)[1]
        for got_mask, model, iters in (alone, beside):
            np.testing.assert_array_equal(np.asarray(got_mask, bool), mask)
            assert (model is None) == (ref is None) and iters == alone[2]
            if model is not None:
                k = 9 if homography else 5  # rotation_deg: atan2f may differ by an ulp
                np.testing.assert_array_equal(np.ravel(model)[:k], np.ravel(ref)[:k])
