"""How many threads a match set gets in launches of more sets than SMs: sets run beside one
another as long as the SMs hold them, and results do not depend on it."""
import numpy as np
import pytest

import psift
import synth

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _sets(sizes, outliers):
    out = []
    for k, n in enumerate(sizes):
        h = synth.perspective_h(1920, 1080, -10 + 3 * k, 0.9 + 0.02 * k, 5e-5, -5e-5)
        out.append(synth.putative_matches(n, outliers, h, 1920, 1080, 800 + k)[0])
    return out


@pytest.mark.parametrize("homography,per_sm,most", [(False, 2, 1.7), (False, 3, 1.7), (True, 2, 1.5)])
def test_sets_run_side_by_side(homography, per_sm, most):
    sms = _sms()
    base = _sets([100] * 5, 0.1)
    ctx = psift.Context(0)
    ctx.enable_stage_timing(True)
    ms = []
    for n in (sms, per_sm * sms):
        best = 1e9
        for _ in range(5):
            ctx.stage_times(reset=True)
            psift.ransac_batch([base[i % 5] for i in range(n)], homography=homography, ctx=ctx)
            best = min(best, ctx.stage_times(reset=True)["ransac"][0])
        ms.append(best)
    ctx.close()
    assert ms[1] < most * ms[0], ms


@pytest.mark.parametrize("homography", [False, True])
@pytest.mark.parametrize("sizes", [(4, 5, 6, 12, 20, 31, 32), (2239, 2240, 2241, 2303, 2305, 200, 300, 33, 700)])
def test_results_do_not_depend_on_the_sets_of_a_launch(homography, sizes):
    # 128 threads stage 2240 matches; alone, a set gets 256 (up to 32 matches) or 512
    sms = _sms()
    base = _sets(sizes, 0.4)
    ctx = psift.Context(0)
    one = [psift.ransac_batch([m], homography=homography, ctx=ctx)[0] for m in base]
    for n in (2 * sms, 2 * sms + 1, 3 * sms + 1):
        for i, (mask, model, iters) in enumerate(psift.ransac_batch([base[i % len(base)] for i in range(n)],
                                                                    homography=homography, ctx=ctx)):
            m1, h1, it1 = one[i % len(base)]
            np.testing.assert_array_equal(mask, m1)
            assert iters == it1 and (model is None) == (h1 is None)
            if model is not None:
                np.testing.assert_array_equal(model, h1)
    ctx.close()
