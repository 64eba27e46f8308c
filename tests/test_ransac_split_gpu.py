"""RANSAC CTAs of 512 and 256 threads (chosen by the number of sets of a launch): a
set's result does not depend on the launch it is part of."""
import numpy as np
import pytest

import psift
import synth

pytestmark = pytest.mark.gpu


def _set(k):
    u = synth.SplitMix64(77 + k).uniform(4)
    h = synth.perspective_h(1920, 1080, -20 + 40 * u[0], 0.8 + 0.4 * u[1], 1e-4 * u[2], -1e-4 * u[3])
    n = (0, 1, 2, 3, 4, 5, 127, 128, 129, 513)[k] if k < 10 else 200 + 53 * (k % 7)
    rec, feats, _ = synth.putative_matches(n, 0.2 + 0.06 * (k % 9), h, 1920, 1080, 4000 + k)
    return rec, 1.0 / np.maximum(feats[:, 0], 0.05) if n else np.zeros(0, np.float32)


@pytest.mark.parametrize("homography", [True, False])
@pytest.mark.parametrize("guided", [False, True])
def test_result_does_not_depend_on_the_number_of_sets(homography, guided):
    ctx = psift.Context(0)
    sets = [_set(k) for k in range(24)]
    run = lambda reps: psift.ransac_batch([m for m, _ in sets] * reps, homography=homography,  # noqa: E731
                                          weights=[w for _, w in sets] * reps if guided else None, ctx=ctx)
    one = run(1)  # 24 sets: 512 threads each
    for reps in (10, 20):  # 240: 512 threads; 480: 256 threads
        many = run(reps)
        for i, (mask, model, iters) in enumerate(many):
            m1, h1, it1 = one[i % 24]
            np.testing.assert_array_equal(mask, m1)
            assert iters == it1 and (model is None) == (h1 is None)
            if model is not None:
                np.testing.assert_array_equal(model, h1)
    ctx.close()
