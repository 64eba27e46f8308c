"""RANSAC CTAs of 256 threads around the end of their staged coordinates (4480 matches): the
results of a launch of more than three sets per SM equal those of one set by itself (512
threads, 9024 staged)."""
import numpy as np
import pytest

import psift
import synth

pytestmark = pytest.mark.gpu

SIZES = (4479, 4480, 4481, 4543, 4545, 5000)


@pytest.mark.parametrize("homography", [True, False])
@pytest.mark.parametrize("guided", [False, True])
def test_sets_around_the_staged_part(homography, guided):
    ctx = psift.Context(0)
    sets, weights = [], []
    for k, n in enumerate(SIZES):
        h = synth.perspective_h(1920, 1080, -15 + 6 * k, 0.9 + 0.05 * k, 1e-4, -5e-5)
        rec, feats, _ = synth.putative_matches(n, 0.2 + 0.1 * k, h, 1920, 1080, 6000 + k)
        sets.append(rec)
        weights.append(1.0 / np.maximum(feats[:, 0], 0.05))
    run = lambda m, w: psift.ransac_batch(m, homography=homography, weights=w if guided else None, ctx=ctx)  # noqa: E731
    one = [run([m], [w])[0] for m, w in zip(sets, weights)]
    for i, (mask, model, iters) in enumerate(run(sets * 80, weights * 80)):  # 480 sets
        m1, h1, it1 = one[i % len(sets)]
        np.testing.assert_array_equal(mask, m1)
        assert iters == it1 and (model is None) == (h1 is None)
        if model is not None:
            np.testing.assert_array_equal(model, h1)
    ctx.close()
