"""Fundamental-matrix CTAs of 512 and 256 threads (chosen by the number of sets of a launch):
a set's result does not depend on the launch it is part of."""
import numpy as np
import pytest

import psift
import synth

pytestmark = pytest.mark.gpu


def test_result_does_not_depend_on_the_number_of_sets():
    ctx = psift.Context(0)
    sizes = [0, 6, 7, 8, 9, 31, 32, 33, 255, 512, 513, 700]
    sets = [synth.epipolar_matches(n, 0.05 * (k % 8), 300 + k)[0] if n else np.zeros(0, psift.MATCH_DTYPE)
            for k, n in enumerate(sizes)]
    one = psift.fundamental_batch(sets, ctx=ctx)          # 12 sets: 512 threads each
    many = psift.fundamental_batch(sets * 13, ctx=ctx)    # 156 sets: 256 threads
    for i, (mask, f, iters) in enumerate(many):
        m1, f1, it1 = one[i % len(sets)]
        np.testing.assert_array_equal(mask, m1)
        assert iters == it1 and (f is None) == (f1 is None)
        if f is not None:
            np.testing.assert_array_equal(f, f1)
    ctx.close()


@pytest.mark.parametrize("sets", [1, 36, 49, 74, 75, 148])
def test_result_does_not_depend_on_the_ctas_of_a_set(sets):
    """Clusters of three, two and one CTA (fewer as the launch holds more sets) against the
    CTAs of 256 threads of a launch of more sets than SMs."""
    ctx = psift.Context(0)
    sizes = [7, 8, 9, 33, 200, 700, 1025]
    base = [synth.epipolar_matches(n, 0.1 * (k % 8), 900 + k)[0] for k, n in enumerate(sizes)]
    base.reverse()
    opt = psift.FundamentalRansacOptions(max_iters=700)
    many = psift.fundamental_batch((base * 23)[:156], opt, ctx)
    for i, (mask, f, iters) in enumerate(psift.fundamental_batch((base * 23)[:sets], opt, ctx)):
        m1, f1, it1 = many[i % len(base)]
        np.testing.assert_array_equal(mask, m1)
        assert iters == it1 and (f is None) == (f1 is None)
        if f is not None:
            np.testing.assert_array_equal(f, f1)
    ctx.close()
