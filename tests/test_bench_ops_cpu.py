"""bench.py's FP32 operation count of the pyramid: a level runs strips from 6 Mpx a launch and
64 x 64 tiles below, so it depends on the images of a launch."""
import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_small_octaves_of_a_launch_count_as_tiles(bench):
    ops = {n: bench.pyramid_fp32_ops_per_image(1080, 1920, n) for n in (1, 2, 8, 64)}
    # 3840 x 2160 and 1920 x 1080 take strips at 8 images (66 and 17 Mpx), 960 x 540 and 480 x 270
    # (4.1 and 1.0 Mpx) tiles; at 64 images (8.3 Mpx) all are strips, at 1 and 2 only the first
    assert ops[1] == ops[2] > ops[8] > ops[64]
    radii = bench.level_radii()
    tiles = sum(2 * (2 * r + 1) * ((64 + 2 * r) / 64 + 1) for r in radii)
    strips = 0.0
    for r in radii:
        rows = 2 * (64 // (2 * r) * (2 * r))
        strips += (1 + rows / (rows - 2 * r)) * (3 * r + 1)
    assert ops[8][0] - ops[64][0] == pytest.approx((960 * 540 + 480 * 270) * (tiles - strips), rel=1e-12)
