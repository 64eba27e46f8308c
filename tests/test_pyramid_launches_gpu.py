"""The pyramid entry forms all DoG slices of an octave in one launch and hands them over in one
copy."""
import numpy as np
import pytest

import oracle as O
import psift
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scales", [3, 5])
@pytest.mark.parametrize("w,h", [(8, 8), (33, 47), (321, 200)])
def test_one_launch_per_octave_for_the_slices(w, h, scales):
    img = O.luma_to_f32(synth.blob_image(w, h, max(3, w * h // 500), 1.5, 6.0, seed=w))
    ctx = psift.Context(0)
    before = ctx.launch_count
    got = psift.build_pyramid(img, psift.SiftConfig().with_octaves(3).with_scales(scales), ctx=ctx)
    launches = ctx.launch_count - before
    assert launches == 1 + len(got) * (scales + 2) + len(got)  # base, levels, slices
    ref = O.Pyramid(img, 3, scales, True)
    assert len(got) == ref.num_octaves
    for o, (g, d) in enumerate(got):
        for s in range(scales + 2):
            np.testing.assert_array_equal(d[s], ref.plane(o, "d", s))
            np.testing.assert_array_equal(d[s], g[s + 1] - g[s])
    ctx.close()
